"""The barriers of the one launch that runs a small brain's batch running out of tries.

axc_row_engine_barrier_limit(0) makes every block give up at its first barrier and return: no block waits, nothing
hangs.  The batch raises AXC_ERR_WAIT_LIMIT; the pushes that it had counted must not reach a later batch or call on
a state that was uploaded anew.
"""
import numpy as np
import pytest

import oracle
from axicor_gb300 import _native as N
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [True, False])   # a batch or per-tick calls after the batch that gave up
def test_batch_after_a_barrier_gave_up(gpu, use_graph):
    lib = N.lib()
    w = W.small(dims=(20, 20, 16), slots=40, inputs=64, p=0.1)   # 6,400 neurons: a resident grid of blocks
    lay, state, heads = S.generate_brain(w.spec())
    n, A, T, cap = lay.padded_n, lay.total_axons, 6, 40
    S.upload_lut(w.lut)
    vram = S.VramState(n, A)
    eng = S.ShardEngine(vram)
    words = (w.num_inputs + 31) // 32
    io = S.IoDeviceBuffers(words, cap, 0, T)
    rng = np.random.default_rng(1)
    bm = S.input_bitmask(w.seed, 0, T, w.num_inputs, w.rate_q32)
    spikes = rng.integers(0, A, size=T * cap).astype(np.uint32)
    counts = np.full(T, cap, np.uint32)

    def batch(graph):
        eng.step_day_phase_batch(T, io, bm, spikes, counts, lay.virtual_offset, w.num_inputs, None, 1, 0, 0,
                                 use_graph=graph)
        eng.synchronize()

    prev = lib.axc_row_engine_barrier_limit(0)
    try:
        vram.upload_state(state)
        vram.upload_axon_heads(heads)
        batch(True)
        assert vram.error_flags(clear=True) & N.ERR_WAIT_LIMIT, "the barrier that gave up must say so"
        lib.axc_row_engine_barrier_limit(prev)
        vram.upload_state(state)
        vram.upload_axon_heads(heads)
        batch(use_graph)
        assert vram.error_flags() == 0
        for t in range(T):
            oracle.step(state, heads, w.lut, n, A, 1, t, bm[t * words:(t + 1) * words], lay.virtual_offset,
                        w.num_inputs, incoming=spikes[t * cap:(t + 1) * cap])
        assert np.array_equal(vram.download_heads(), heads)
        assert np.array_equal(vram.download_state(), state)
    finally:
        lib.axc_row_engine_barrier_limit(prev)
        vram.free()
