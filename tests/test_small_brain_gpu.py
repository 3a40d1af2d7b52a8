"""Small brains, whose ticks run in one launch (one cluster of blocks, or one block on every SM), against the oracle,
bit-exact, at the edges of their sizes: batches and per-tick calls with input, network spikes and readout, on rows whose
ticks take the dense, the lit-sum and the lit-row forms."""
import ctypes as C

import numpy as np
import pytest

import oracle
from axicor_gb300 import _native as N
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W
from axicor_gb300.formats import StateView, state_blob_size

pytestmark = pytest.mark.gpu

CLUSTER = 4096   # neurons or axons up to which a cluster runs a batch (3,072: a per-tick call); a grid: 640 an SM


def brain(n, A, kind):
    """A ring of n neurons on the first of A axons; the last 32 axons take the input."""
    rng = np.random.default_rng(n)
    state = np.zeros(state_blob_size(n), np.uint8)
    sv = StateView(state, n)
    for s in range(28):
        sv.targets[s] = ((1 + s % 9) << 24) | (1 + (np.arange(n) + 3 * s + 1) % n)
    sv.targets[28] = (3 << 24) | (A - 31 + np.arange(n) % 32)
    sv.weights[:29] = rng.integers(2100, 2900, size=(29, n))
    sv.weights[:29][rng.random((29, n)) < (0.5 if kind == "plastic" else 0.03)] = 300
    sv.soma_to_axon[:] = np.arange(n, dtype=np.uint32)
    sv.voltage[:] = rng.integers(0, 1999, size=n)
    heads = np.full(A * 8, 0x80000000, np.uint32)
    if kind != "dense":
        heads.reshape(A, 8)[:, :5] = np.arange(0, 10, 2, dtype=np.uint32)
    return state, heads


@pytest.mark.parametrize("kind", ["dense", "lit", "plastic"])
@pytest.mark.parametrize("n, A", [(4, 64), (1028, 1088), (1000, 3072), (1000, CLUSTER), (CLUSTER, CLUSTER + 32),
                                  (600, 640 * 152), (600, 640 * 152 + 32)])
def test_small_brain(gpu, n, A, kind):
    state, heads = brain(n, A, kind)
    lut = W.small().lut
    if kind == "plastic":
        lut[0]["d1_affinity"] = 64
    S.upload_lut(lut)
    lib = N.lib()
    vram = S.VramState(n, A)
    rng = np.random.default_rng(A)
    T, cap = 10, 24
    ids = np.concatenate([rng.integers(0, n, size=70), [0xFFFFFFFF]]).astype(np.uint32)
    d_ids, d_bm, d_in, d_out = S.device_array(ids), lib.gpu_malloc(4), lib.gpu_malloc(4 * cap), lib.gpu_malloc(ids.size)
    io = S.IoDeviceBuffers(1, cap, ids.size, T)
    try:
        vram.upload_state(state)
        vram.upload_axon_heads(heads)
        eng = S.ShardEngine(vram)
        tick = 0
        for b in range(14):
            bm = (rng.integers(0, 1 << 32, size=T, dtype=np.uint64) & rng.integers(0, 1 << 32, size=T, dtype=np.uint64)
                  ).astype(np.uint32)
            counts = rng.integers(0, cap + 1, size=T).astype(np.uint32)
            counts[rng.random(T) < 0.3] = 0
            spikes = rng.integers(0, A + 2, size=(T, cap)).astype(np.uint32)
            got, want = np.zeros((T, ids.size), np.uint8), np.zeros((T, ids.size), np.uint8)
            for t in range(T):
                oracle.step(state, heads, lut, n, A, 1, tick + t, bm[t:t + 1], A - 32, 32,
                            incoming=spikes[t, :counts[t]], mapped_soma_ids=ids, outputs=want[t], dopamine=b - 7)
            if b % 7 != 3:
                eng.step_day_phase_batch(T, io, bm, spikes.reshape(-1), counts, A - 32, 32, d_ids, 1, b - 7, tick,
                                         got.reshape(-1))
                eng.synchronize()
            else:
                for t in range(T):
                    assert lib.gpu_memcpy_host_to_device(d_bm, N.ptr(bm[t:t + 1]), 4)
                    assert lib.gpu_memcpy_host_to_device(d_in, N.ptr(spikes[t]), 4 * cap)
                    assert lib.cu_step_day_phase(C.byref(vram.ptrs), n, A, 1, tick + t, d_bm, A - 32, 32, d_in,
                                                 int(counts[t]), d_ids, d_out, ids.size, b - 7, None) == 0
                    assert lib.gpu_memcpy_device_to_host(N.ptr(got[t]), d_out, ids.size)
            tick += T
            assert np.array_equal(got, want), f"readout differs, ticks to {tick}"
            assert np.array_equal(vram.download_heads(), heads), f"heads differ at tick {tick}"
            assert np.array_equal(vram.download_state(), state), f"state differs at tick {tick}"
        assert vram.error_flags() == 0
        assert int(vram.counters()[3]) > 0
    finally:
        S.upload_lut(W.default_lut())
        for p in (d_ids, d_bm, d_in, d_out):
            lib.gpu_free(p)
        vram.free()
