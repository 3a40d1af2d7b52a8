"""The row engine's sparse form (few active axons: the hits are added from an inverted index) against the oracle,
bit-exact through the learned engine's chunks, on quiet brains with every kind of slot the index can hold:
segments 0 and >= 31, variants of other propagation lengths, axons owned by two somas, invalid targets and an axon with
more entries than the index sorts."""
import numpy as np
import pytest

import oracle
from axicor_gb300 import _native as N
from axicor_gb300 import learned as L
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W
from axicor_gb300.formats import StateView, state_blob_size

pytestmark = pytest.mark.gpu


def quiet_brain(odd: bool, seed: int):
    w = W.homeostatic(W.small(dims=(25, 23, 11), slots=70, inputs=96, p=0.05, seed=seed))
    lay, state, heads = S.generate_brain(w.spec())
    sv = StateView(state, lay.padded_n)
    rng = np.random.default_rng(seed)
    if odd:
        w.lut[1]["signal_propagation_length"] = 7        # the excitatory neurons' length is not the LUT maximum
        w.lut[1]["inertia_curve"] = np.array([128, 100, 80, 60] + [40] * 12, np.uint8)
        live = sv.targets != 0
        r = rng.random(live.shape)
        t = sv.targets
        t[live & (r < 0.02)] &= 0x00FFFFFF                                             # segment 0
        far = live & (r > 0.96)
        t[far] = (t[far] & 0x00FFFFFF) | (rng.integers(29, 60, size=far.sum()).astype(np.uint32) << 24)
        hub = live & (r > 0.5) & (r < 0.52)
        t[hub] = (t[hub] & np.uint32(0xFF000000)) | 5                                  # axon 4: thousands of entries
        bad = live & (r > 0.9) & (r < 0.9005)
        t[bad] = (t[bad] & np.uint32(0xFF000000)) | np.uint32(lay.total_axons + 9)     # out of range
        share = np.nonzero(rng.random(lay.num_neurons) < 0.02)[0]
        sv.soma_to_axon[share] = rng.integers(0, lay.num_neurons, size=share.size).astype(np.uint32)
    return w, lay, state, heads


def applicable(state, heads, lay, reach):
    """The rule of the form on the oracle's state: twice the active axons below the neurons the next tick evaluates."""
    active = int(np.any(heads.reshape(-1, 8) < reach, axis=1).sum())
    return 2 * active < int((StateView(state, lay.padded_n).timers[:lay.num_neurons] == 0).sum())


@pytest.mark.parametrize("policy", [0, 1, -1])
@pytest.mark.parametrize("odd", [False, True])
def test_sparse_chunks(gpu, odd, policy):
    lib = N.lib()
    w, lay, h_state, h_heads = quiet_brain(odd, 17)
    S.upload_lut(w.lut)
    vr, vc = (S.VramState(lay.padded_n, lay.total_axons) for _ in range(2))
    for v in (vr, vc):
        v.upload_state(h_state)
        v.upload_axon_heads(h_heads)
    words = (w.num_inputs + 31) // 32
    chunk, chunks, quiet = 20, 22, 0
    bits = S.input_bitmask(w.seed, 0, chunk * chunks, w.num_inputs, w.rate_q32)
    d_bits = S.device_array(bits)
    eng = L.LearnedEngine(vr, lay.padded_n, lay.total_axons, lay.virtual_offset, w.num_inputs, d_bits, words,
                          chunk * chunks, w.v_seg, 3)
    col = S.ShardEngine(vc)
    io_c = S.IoDeviceBuffers(words, 0, 0, chunk)
    try:
        eng.set_policy(L.Policy(policy=policy))
        for b in range(chunks):
            bm = bits[b * chunk * words:(b + 1) * chunk * words]
            eng.run(b * chunk, chunk, chunk)
            lib.gpu_device_synchronize()
            prev = lib.axc_batch_engine_mode(0)
            col.step_day_phase_batch(chunk, io_c, bm, None, None, lay.virtual_offset, w.num_inputs, None, w.v_seg, 3,
                                     b * chunk)
            col.synchronize()
            lib.axc_batch_engine_mode(prev)
            oracle.run_ticks(h_state, h_heads, w.lut, lay.padded_n, lay.total_axons, w.v_seg, b * chunk, chunk, bm,
                             words, lay.virtual_offset, w.num_inputs, dopamine=3)
            assert np.array_equal(vr.download_heads(), h_heads), f"chunk {b}: heads differ"
            assert np.array_equal(vr.download_state(), h_state), f"chunk {b}: state differs"
            quiet += applicable(h_state, h_heads, lay, 67 if odd else 31)
        assert quiet >= 6, f"the brain must be quiet enough for the form ({quiet} chunk ends)"
        cr, cc = vr.counters(), vc.counters()
        assert np.array_equal(cr[:6], cc[:6]), f"counters {cr} against the columnar kernels' {cc}"
        assert vr.error_flags() == (N.ERR_TARGET_RANGE if odd else 0)
    finally:
        eng.close()
        lib.gpu_free(d_bits)
        vr.free()
        vc.free()


@pytest.mark.parametrize("n", [4, 68, 100, 132, 1000])
def test_lit_sum_odd_counts(gpu, n):
    """Neuron counts that are no multiple of 16, each layout decided by the device: the lit-sum form
    of a frozen ring against the oracle."""
    state = np.zeros(state_blob_size(n), np.uint8)
    sv = StateView(state, n)
    rng = np.random.default_rng(n)
    A = (n + 63) // 32 * 32
    for s in range(24):
        sv.targets[s] = ((1 + s % 9) << 24) | (1 + (np.arange(n) + s + 1) % n)
    sv.weights[:24] = rng.integers(2100, 2900, size=(24, n))
    movable = rng.random((24, n)) < 0.03
    sv.weights[:24][movable] = 300
    sv.soma_to_axon[:] = np.arange(n, dtype=np.uint32)
    sv.voltage[:] = rng.integers(0, 1999, size=n)
    heads = np.full(A * 8, 0x80000000, np.uint32)
    heads.reshape(A, 8)[:n, :5] = np.arange(0, 10, 2, dtype=np.uint32)
    w = W.small()
    S.upload_lut(w.lut)
    vram = S.VramState(n, A)
    lib = N.lib()
    try:
        vram.upload_state(state)
        vram.upload_axon_heads(heads)
        eng = S.ShardEngine(vram)
        io = S.IoDeviceBuffers(1, 0, 0, 8)
        for b in range(12):
            eng.step_day_phase_batch(8, io, None, None, None, 0, 0, None, 1, 0, 8 * b)
            eng.synchronize()
            oracle.run_ticks(state, heads, w.lut, n, A, 1, 8 * b, 8, None, 0, 0, 0)
            assert np.array_equal(vram.download_heads(), heads), f"batch {b}: heads differ"
            assert np.array_equal(vram.download_state(), state), f"batch {b}: state differs"
        assert int(vram.counters()[6]) > 16, vram.counters()
    finally:
        vram.free()


@pytest.mark.parametrize("n", [68, 100, 1000])
def test_sparse_odd_counts(gpu, n):
    """The sparse form off its 128-neuron tiles and 16-byte loads: neurons that only their heartbeat fires."""
    state = np.zeros(state_blob_size(n), np.uint8)
    sv = StateView(state, n)
    rng = np.random.default_rng(n)
    A = (n + 63) // 32 * 32
    for s in range(30):
        sv.targets[s] = ((1 + s % 9) << 24) | (1 + (np.arange(n) * 7 + s + 1) % n)
    sv.weights[:30] = rng.integers(-900, 900, size=(30, n))
    sv.soma_to_axon[:] = np.arange(n, dtype=np.uint32)
    heads = np.full(A * 8, 0x80000000, np.uint32)
    w = W.small()
    w.lut[0]["threshold"] = 1 << 20
    w.lut[0]["spontaneous_firing_period_ticks"] = 211
    w.lut[0]["inertia_curve"] = np.array([128, 100, 80, 60] + [40] * 12, np.uint8)
    S.upload_lut(w.lut)
    lib = N.lib()
    vram = S.VramState(n, A)
    try:
        vram.upload_state(state)
        vram.upload_axon_heads(heads)
        eng = L.LearnedEngine(vram, n, A, 0, 0, None, 0, 0, w.v_seg, 0)
        eng.set_policy(L.Policy(policy=0))
        quiet = 0
        for b in range(12):
            eng.run(20 * b, 20, 20)
            lib.gpu_device_synchronize()
            oracle.run_ticks(state, heads, w.lut, n, A, 1, 20 * b, 20, None, 0, 0, 0)
            assert np.array_equal(vram.download_heads(), heads), f"chunk {b}: heads differ"
            assert np.array_equal(vram.download_state(), state), f"chunk {b}: state differs"
            quiet += 2 * int(np.any(heads.reshape(-1, 8) < 13, axis=1).sum()) < n
        assert quiet >= 8, quiet
        eng.close()
    finally:
        S.upload_lut(W.default_lut())
        vram.free()
