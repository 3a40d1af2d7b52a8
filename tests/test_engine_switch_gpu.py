"""A shard stepped by the row engine and by the columnar kernels in turn, bit-exact against the oracle.

The columnar kernels (axc_batch_engine_mode(0), axc_tick_engine_mode(0)) move the weights of the .state blob
(physics.cu:281-373), so a row copy that the batch path or the per-tick entry point kept is out of date after
them.
"""
import numpy as np
import pytest

from axicor_gb300 import _native as N
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W
from test_batch_rows_reuse_gpu import BatchTwin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", ["b1" + 8 * " b0 b1", "b1" + 8 * " t0 b1", "t1 t0 t1", "t1 b0 t1"])
def test_columnar_steps_between_row_steps(gpu, steps):
    """b: batches of 10 ticks, t: 10 per-tick calls; 1: the row engine, 0: the columnar kernels."""
    lib = N.lib()
    w = W.small(dims=(16, 16, 8), slots=96, inputs=64, p=0.2)
    for v in (0, 1):
        w.lut[v]["inertia_curve"] = np.array([128, 110, 90, 70, 60, 50, 40, 30, 20, 16, 12, 8, 6, 4, 2, 1], np.uint8)
    t = BatchTwin(w, frozen=False)
    modes = lib.axc_batch_engine_mode(1), lib.axc_tick_engine_mode(1)
    try:
        for step in steps.split():
            lib.axc_batch_engine_mode(int(step[1]))
            lib.axc_tick_engine_mode(int(step[1]))
            before = t.h_state.copy()
            t.batch(10) if step[0] == "b" else t.per_tick(10)
            weights = [S.StateView(x, t.N).weights for x in (before, t.h_state)]
            assert np.count_nonzero(weights[0] != weights[1]) > 100, f"{step} must move weights"
        assert t.vram.error_flags() == 0
    finally:
        lib.axc_batch_engine_mode(modes[0])
        lib.axc_tick_engine_mode(modes[1])
        S.upload_lut(W.default_lut())
        t.close()
