"""Every form of a tick and both ways to run it (the kernel chain, one launch), bit-exact against the oracle, with the
device's own count of what ran.

Brains of up to 4,096 neurons or axons run a batch in one launch (3,072: a per-tick call; a batch that has the GPU to
itself: 640 an SM), so the chain's kernels are reached here by larger ones, and by the shards of a zone.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from axicor_gb300 import _native as N
from axicor_gb300 import learned as L
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W
from axicor_gb300.formats import StateView, state_blob_size
from helpers import Twin
from test_row_engine_gpu import stress_brain
from test_sparse_form_gpu import quiet_brain

pytestmark = pytest.mark.gpu

DENSE, LIT_SUM, SPARSE, SCATTER, LIT_ROWS, CHECKED, ONE_LAUNCH, LAYOUTS = range(8)
CURVE = np.array([128, 110, 90, 70, 60, 50, 40, 30, 20, 16, 12, 8, 6, 4, 2, 1], np.uint8)


def stress(case):
    w = W.small(dims=(32, 16, 8), slots=96, inputs=64, p=0.1)
    dopamine = 0
    if case == "mixed_lengths":
        w.lut[0]["signal_propagation_length"], w.lut[1]["signal_propagation_length"] = 6, 3
    elif case == "dopamine_inertia":
        for v in (0, 1):
            w.lut[v]["inertia_curve"] = CURVE
            w.lut[v]["d1_affinity"], w.lut[v]["d2_affinity"] = 80, 120
        w.w_max, dopamine = 6000, 150
    elif case == "long_tail_cooling":
        w.lut[0]["signal_propagation_length"] = w.lut[1]["signal_propagation_length"] = 40
    lay, state, heads = stress_brain(w)
    sv = StateView(state, lay.padded_n)
    sv.targets[3, 7] = (sv.targets[3, 7] & np.uint32(0xFF000000)) | np.uint32(lay.total_axons + 9)   # out of range
    return w, lay, state, heads, dopamine


@pytest.mark.parametrize("case, cap", [("default", None), ("mixed_lengths", None), ("dopamine_inertia", None),
                                       ("long_tail_cooling", None), ("dopamine_inertia", 0), ("dopamine_inertia", 7)])
def test_chain_per_tick(gpu, case, cap):
    """Segments 0 and >= 31, axons of two somas, several lengths, cooling, an invalid target, a fix-up list that
    overflows: through the chain's write-through and readout."""
    w, lay, state, heads, dopamine = stress(case)
    lib = N.lib()
    prev = lib.axc_row_engine_fix_capacity(cap) if cap is not None else None
    tw = Twin(w, state=state, heads=heads, lay=lay)
    try:
        spikes = 0
        for k in range(24):
            g, o, _ = tw.step_both(dopamine=dopamine)
            assert np.array_equal(g, o), f"raster differs at tick {k}"
            tw.compare(f"tick {k}")
            spikes += int(o.sum())
        assert spikes > 0 and tw.vram.counters()[4] > 0
        assert tw.vram.error_flags() == N.ERR_TARGET_RANGE
        forms = tw.vram.forms()
        assert forms[ONE_LAUNCH] == 0 and forms[:6].sum() == 24, forms
    finally:
        if cap is not None:
            lib.axc_row_engine_fix_capacity(prev)
        tw.close()
        S.upload_lut(W.default_lut())


@pytest.mark.parametrize("case, cap", [("default", None), ("mixed_lengths", None), ("dopamine_inertia", None),
                                       ("long_tail_cooling", None), ("dopamine_inertia", 7)])
def test_chain_in_a_batch(gpu, case, cap):
    """The same in batches, as two shards of a zone."""
    w, lay, state, heads, dopamine = stress(case)
    lib = N.lib()
    prev = lib.axc_row_engine_fix_capacity(cap) if cap is not None else None
    n, A, T, words = lay.padded_n, lay.total_axons, 12, (w.num_inputs + 31) // 32
    S.upload_lut(w.lut)
    vrams = [S.VramState(n, A) for _ in range(2)]
    ids = np.arange(n, dtype=np.uint32)
    d_ids = S.device_array(ids)
    ios = [S.IoDeviceBuffers(words, 0, n, T) for _ in vrams]
    outs = [np.zeros(T * n, np.uint8) for _ in vrams]
    eng = S.ShardEngine(vrams[0])
    try:
        for v in vrams:
            v.upload_state(state)
            v.upload_axon_heads(heads)
        for b in range(3):
            bm = S.input_bitmask(w.seed, T * b, T, w.num_inputs, w.rate_q32)
            shards = (N.AxcZoneShard * 2)()
            for z, v, io, out in zip(shards, vrams, ios, outs):
                z.vram, z.padded_n, z.total_axons, z.io = v.ptrs, n, A, io.as_struct()
                z.h_input_bitmask, z.virtual_offset, z.num_virtual_axons = N.ptr(bm), lay.virtual_offset, w.num_inputs
                z.mapped_soma_ids_device, z.v_seg, z.dopamine, z.h_output_history = d_ids, 1, dopamine, N.ptr(out)
            N.check(lib.axc_step_zone_batch(shards, 2, None, 0, T, T * b, eng.stream), "axc_step_zone_batch")
            ref = np.zeros(T * n, np.uint8)
            oracle.run_ticks(state, heads, w.lut, n, A, 1, T * b, T, bm, words, lay.virtual_offset, w.num_inputs,
                             mapped_soma_ids=ids, outputs=ref, dopamine=dopamine)
            for v, out in zip(vrams, outs):
                assert np.array_equal(out, ref), f"batch {b}: raster differs"
                assert np.array_equal(v.download_heads(), heads), f"batch {b}: heads differ"
                assert np.array_equal(v.download_state(), state), f"batch {b}: state differs"
        for v in vrams:
            forms = v.forms()
            assert forms[ONE_LAUNCH] == 0 and forms[:6].sum() == 3 * T, forms
            assert v.error_flags() == N.ERR_TARGET_RANGE
    finally:
        if cap is not None:
            lib.axc_row_engine_fix_capacity(prev)
        lib.gpu_free(d_ids)
        for v in vrams:
            v.free()
        S.upload_lut(W.default_lut())


def test_chain_bitmap_wait_gives_up(gpu):
    """The update pass's wait for the staged bitmap running out in the chain's kernels: flagged, results exact."""
    w, lay, state, heads, _ = stress("default")
    lib = N.lib()
    tw = Twin(w, state=state, heads=heads, lay=lay)
    prev = lib.axc_row_engine_wait_limit(0)
    try:
        for k in range(8):
            g, o, _ = tw.step_both()
            assert np.array_equal(g, o), f"raster differs at tick {k}"
            tw.compare(f"tick {k}")
        assert tw.vram.error_flags() & N.ERR_WAIT_LIMIT
        assert tw.vram.forms()[ONE_LAUNCH] == 0
    finally:
        lib.axc_row_engine_wait_limit(prev)
        tw.close()


class Ring:
    """n neurons on the first of A axons, `slots` slots a row, in step with the oracle; every weight moves."""

    def __init__(self, n, A, slots, segs=9):
        self.n, self.A = n, A
        self.lut = W.small().lut
        for v in (0, 1):
            self.lut[v]["inertia_curve"] = CURVE
        rng = np.random.default_rng(n)
        self.state = np.zeros(state_blob_size(n), np.uint8)
        sv = StateView(self.state, n)
        for s in range(slots):
            sv.targets[s] = ((1 + s % segs) << 24) | (1 + (np.arange(n) + 3 * s + 1) % n)
        sv.weights[:slots] = rng.integers(2100, 2900, size=(slots, n)) * rng.choice([1, 1, 1, -1], size=(slots, n))
        sv.soma_to_axon[:] = np.arange(n, dtype=np.uint32)
        sv.voltage[:] = rng.integers(0, 1999, size=n)
        self.heads = np.full(A * 8, 0x80000000, np.uint32)
        self.heads.reshape(A, 8)[:, :5] = np.arange(0, 10, 2, dtype=np.uint32)
        S.upload_lut(self.lut)
        self.vram = S.VramState(n, A)
        self.vram.upload_state(self.state)
        self.vram.upload_axon_heads(self.heads)
        self.eng, self.io, self.tick = S.ShardEngine(self.vram), S.IoDeviceBuffers(0, 0, 0, 10), 0

    def run(self, per_tick, ticks=10):
        """`ticks` ticks; the forms that they ran."""
        self.vram.forms(reset=True)
        for t0 in range(0, ticks, 10):
            t = min(10, ticks - t0)
            self.eng.step_day_phase_batch(t, self.io, None, None, None, 0, 0, None, 1, 5, self.tick,
                                          use_graph=not per_tick)
            oracle.run_ticks(self.state, self.heads, self.lut, self.n, self.A, 1, self.tick, t, None, 0, 0, 0,
                             dopamine=5)
            self.tick += t
        self.eng.synchronize()
        assert np.array_equal(self.vram.download_heads(), self.heads), f"heads differ at tick {self.tick}"
        assert np.array_equal(self.vram.download_state(), self.state), f"state differs at tick {self.tick}"
        assert self.vram.error_flags() == 0
        return self.vram.forms()

    def darken(self, axons):
        """The first axons' heads are gone: dark until their somas have fired three times."""
        self.heads.reshape(self.A, 8)[:axons] = 0x80000000
        self.vram.upload_axon_heads(self.heads)

    def close(self):
        self.vram.free()
        S.upload_lut(W.default_lut())


@pytest.mark.parametrize("per_tick", [False, True])
@pytest.mark.parametrize("chain", [False, True])
@pytest.mark.parametrize("slots", [66, 96, 128])   # the second half of a lit row: positions 64 and up
def test_lit_rows_and_a_dark_axon(gpu, slots, chain, per_tick):
    """Rows of movable slots on always-lit axons (read and moved two at a time), then one axon dark."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    A = (3072 if per_tick else 640 * sms) if not chain else 640 * sms + 32
    r = Ring(600, A, slots)
    try:
        for _ in range(8):
            forms = r.run(per_tick, 64 if per_tick else 10)   # a per-tick layout is decided every 64 calls
        ticks = 64 if per_tick else 10
        assert forms[LIT_ROWS] == ticks and forms[ONE_LAUNCH] == (0 if chain else ticks), forms
        r.darken(1)
        forms = r.run(per_tick)
        assert forms[:6].sum() == 10 and forms[LIT_ROWS] < 10, forms
        if A > 90_000:   # one dark axon among many
            assert forms[CHECKED] > 0, forms
    finally:
        r.close()


@pytest.mark.parametrize("tiles", [1, 2, 4])
def test_layout_tiles(gpu, tiles):
    """Layouts whose blocks take one, two or four tiles of 32 neurons, the last of them ragged; slots on both sides of
    the segments that every axon counts as using."""
    wave = 4 * torch.cuda.get_device_properties(0).multi_processor_count
    n = 32 * (tiles - 1) * wave + 32 * 5 + 4
    r = Ring(n, (n + 63) // 32 * 32, 48, segs=23)
    try:
        layouts = 0
        for _ in range(7):
            forms = r.run(False)
            layouts += int(forms[LAYOUTS])
        assert layouts >= 2 and forms[LIT_ROWS] > 0, (layouts, forms)
    finally:
        r.close()


def test_later_layouts_keep_the_used_segments(gpu):
    """Forced, first and later layouts of the same targets, a new write (other targets), and the same again."""
    r = Ring(600, 704, 40, segs=23)
    try:
        for shift in (0, 5):
            sv = StateView(r.state, r.n)
            sv.targets[:40] = np.roll(sv.targets[:40], shift, axis=1)
            sv.targets[3] = ((24 + shift % 4) << 24) | (sv.targets[3] & np.uint32(0xFFFFFF))
            r.vram.upload_state(r.state)
            layouts = sum(int(r.run(False)[LAYOUTS]) for _ in range(60))
            assert layouts >= 4, layouts
    finally:
        r.close()


@pytest.mark.parametrize("per_tick", [False, True])
def test_many_dark_axons_take_the_dense_pass(gpu, per_tick):
    """Checking rows slot by slot pays while few have a slot on a dark axon."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r = Ring(600, 640 * sms + 32, 96)
    try:
        for _ in range(8):
            r.run(per_tick, 64 if per_tick else 10)
        r.darken(300)
        forms = r.run(per_tick, 3)
        assert forms[DENSE] > 0 and forms[CHECKED] == 0, forms
        r.run(per_tick, 20)
    finally:
        r.close()


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("gated", [False, True])
def test_learned_quiet_ticks_run_sparse(gpu, gated, odd):
    """The learned engine's quiet ticks do run from the inverted index of the rows; also in the gate, whose plain
    graphs have the form's kernels unless the brain has been busy for 256 ticks."""
    w, lay, state, heads = quiet_brain(odd, 17)
    S.upload_lut(w.lut)
    vram = S.VramState(lay.padded_n, lay.total_axons)
    vram.upload_state(state)
    vram.upload_axon_heads(heads)
    words, T = (w.num_inputs + 31) // 32, 440
    bits = S.input_bitmask(w.seed, 0, T, w.num_inputs, w.rate_q32)
    d_bits = S.device_array(bits)
    eng = L.LearnedEngine(vram, lay.padded_n, lay.total_axons, lay.virtual_offset, w.num_inputs, d_bits, words, T,
                          w.v_seg, 3)
    try:
        # every tick planned sparse: scattered until the rows have an index; or none, whatever the prediction
        eng.set_policy(L.Policy(policy=-1, ratio=1e30) if gated else L.Policy(policy=1))
        for t in range(0, T, 20):
            eng.run(t, 20, 20)
            N.lib().gpu_device_synchronize()
        oracle.run_ticks(state, heads, w.lut, lay.padded_n, lay.total_axons, w.v_seg, 0, T, bits, words,
                         lay.virtual_offset, w.num_inputs, dopamine=3)
        assert np.array_equal(vram.download_heads(), heads)
        assert np.array_equal(vram.download_state(), state)
        forms = vram.forms()
        if not (gated and odd):   # whose longer tails keep too many axons active for the exact counts
            assert forms[SPARSE] > 100, forms
        assert not gated or eng.stats()["gated_ticks"] > 200
    finally:
        eng.close()
        N.lib().gpu_free(d_bits)
        vram.free()
        S.upload_lut(W.default_lut())


def test_gate_through_a_busy_phase(gpu):
    """Quiet, then saturated for longer than the gate's graphs keep the sparse form's kernels, then quiet again."""
    w, lay, state, heads = quiet_brain(False, 23)
    busy = w.lut.copy()
    for v in (0, 1):
        busy[v]["homeostasis_penalty"], busy[v]["homeostasis_decay"] = 0, 16000
    n, A = lay.padded_n, lay.total_axons
    S.upload_lut(w.lut)
    vram = S.VramState(n, A)
    vram.upload_state(state)
    vram.upload_axon_heads(heads)
    words, T = (w.num_inputs + 31) // 32, 1000
    bits = S.input_bitmask(w.seed, 0, T, w.num_inputs, w.rate_q32)
    d_bits = S.device_array(bits)
    eng = L.LearnedEngine(vram, n, A, lay.virtual_offset, w.num_inputs, d_bits, words, T, w.v_seg, 3)
    try:
        eng.set_policy(L.Policy(policy=-1, ratio=1e30))
        for lut, t0, t1 in ((w.lut, 0, 260), (busy, 260, 620), (w.lut, 620, T)):
            S.upload_lut(lut)
            vram.forms(reset=True)
            for t in range(t0, t1, 20):
                eng.run(t, 20, 20)
                N.lib().gpu_device_synchronize()
            oracle.run_ticks(state, heads, lut, n, A, w.v_seg, t0, t1 - t0, bits[t0 * words:], words,
                             lay.virtual_offset, w.num_inputs, dopamine=3)
            assert np.array_equal(vram.download_heads(), heads), f"heads differ at tick {t1}"
            assert np.array_equal(vram.download_state(), state), f"state differs at tick {t1}"
            sparse = int(vram.forms()[SPARSE])
            assert sparse > 0 if lut is w.lut else sparse < 20, (t1, sparse)
    finally:
        eng.close()
        N.lib().gpu_free(d_bits)
        vram.free()
        S.upload_lut(W.default_lut())


def test_profiled_ticks_run_as_a_batch_does(gpu):
    """axc_profile_ticks times the rows that a batch would run on: lit rows, not a layout of its own."""
    r = Ring(600, 1024, 66)
    ms, counts = (C.c_float * 5)(), (C.c_uint64 * 7)()
    try:
        for _ in range(8):
            forms = r.run(False)
        assert forms[LIT_ROWS] == 10, forms
        r.vram.forms(reset=True)
        err = N.lib().axc_profile_ticks(C.byref(r.vram.ptrs), r.n, r.A, 1, r.tick, 10, None, 0, 0, 0, 5, 1,
                                        r.eng.stream, ms, counts)
        assert err == 0 and ms[2] > 0
        forms = r.vram.forms()
        assert forms[LIT_ROWS] == 10 and forms[ONE_LAUNCH] == 0, forms
        oracle.run_ticks(r.state, r.heads, r.lut, r.n, r.A, 1, r.tick, 10, None, 0, 0, 0, dopamine=5)
        r.tick += 10
        assert r.run(False)[LIT_ROWS] == 10
    finally:
        r.close()


@pytest.mark.parametrize("slots", [21, 23, 60])   # write-back by a thread a neuron (two), in tiles
def test_write_back_of_split_rows(gpu, slots):
    """Movable slots on lit axons laid before one on a dark axon, in every second row: each weight back in its slot."""
    r = Ring(608, 704, slots)
    try:
        sv = StateView(r.state, r.n)
        sv.targets[7, ::2] = (2 << 24) | 700   # an axon that no soma owns
        r.vram.upload_state(r.state)
        for _ in range(8):
            forms = r.run(False)
        assert forms[LIT_ROWS] > 0, forms
    finally:
        r.close()
