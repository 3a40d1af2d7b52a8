"""A shard stepped by the row engine and by the columnar kernels in turn, bit-exact against the oracle.

The columnar kernels (axc_batch_engine_mode(0), axc_tick_engine_mode(0)) move the weights of the .state blob
(physics.cu:281-373), so a row copy that the batch path or the per-tick entry point kept is out of date after
them.
"""
import numpy as np
import pytest

import oracle
from axicor_gb300 import _native as N
from axicor_gb300 import population as Pop
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W
from axicor_gb300.formats import StateView
from test_batch_rows_reuse_gpu import BatchTwin, mostly_frozen

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
            weights = [StateView(x, t.N).weights for x in (before, t.h_state)]
            assert np.count_nonzero(weights[0] != weights[1]) > 100, f"{step} must move weights"
        assert t.vram.error_flags() == 0
    finally:
        lib.axc_batch_engine_mode(modes[0])
        lib.axc_tick_engine_mode(modes[1])
        S.upload_lut(W.default_lut())
        t.close()


def population(steps):
    """Two mostly frozen brains (their batches keep a layout of lit sums) stepped alone and as a population."""
    brains = [Pop.Brain(W.small(dims=(16, 16, 8), slots=80, inputs=64, p=0.1, seed=s), 400) for s in (1, 2)]
    pop = None
    try:
        tick = 0
        for b in brains:
            mostly_frozen(b.w, b.state0, b.lay.padded_n)
            sv = StateView(b.state0, b.lay.padded_n)   # the others freeze at every tick, each in its turn
            move = (sv.targets != 0) & (np.abs(sv.weights) < 2048)
            size = np.random.default_rng(b.w.seed).integers(50, 2048, size=int(move.sum()))
            sv.weights[move] = np.sign(sv.weights[move]) * size
            b.reset()
        S.upload_lut(brains[0].w.lut)
        engines = [S.ShardEngine(b.vram) for b in brains]
        ios = [S.IoDeviceBuffers(b.words, 0, 0, 20) for b in brains]
        for step in steps.split():
            ticks = {"alone": 20, "create": 0, "tune": 12, "run": 8}[step]
            if step == "alone":
                for b, e, io in zip(brains, engines, ios):   # (Brain.run_alone uploads the LUT, which lays the rows out anew)
                    e.step_day_phase_batch(ticks, io, b.bitmask[tick * b.words:], None, None, b.lay.virtual_offset,
                                           b.w.num_inputs, None, 1, 0, tick)
            elif step == "create":
                pop = Pop.Population(brains)
            elif step == "tune":
                pop.tune(tick, 1)
            else:
                pop.run(tick, ticks, 4)
            tick += ticks
            N.lib().gpu_device_synchronize()
        assert all(b.vram.forms()[[1, 4]].sum() > 0 for b in brains)
        for b in brains:
            state, heads = b.state0.copy(), b.heads0.copy()
            oracle.run_ticks(state, heads, b.w.lut, b.lay.padded_n, b.lay.total_axons, 1, 0, tick, b.bitmask, b.words,
                             b.lay.virtual_offset, b.w.num_inputs)
            assert np.array_equal(b.vram.download_heads(), heads)
            assert np.array_equal(b.vram.download_state(), state)
    finally:
        if pop:
            pop.close()
        for b in brains:
            b.free()
        S.upload_lut(W.default_lut())


def test_a_brains_own_batches_between_population_runs(gpu):
    """A brain's first own batch replaces the row buffers that the population made (a batch keeps a list of deferred
    slots beside them): the population takes the new ones."""
    population("create run" + 4 * " alone" + " run tune alone alone run")


@pytest.mark.parametrize("batches", [3, 4, 5, 6, 7, 8])   # between two layouts of the batch path, or not
def test_batches_around_a_population_tuning(gpu, batches):
    """The tuner's trial ticks move weights and use the rows' buffers."""
    population("alone create" + batches * " alone" + " tune alone run alone")


def test_another_state_allocation_behind_the_same_heads(gpu):
    """A captured batch holds its state's addresses; the shard is known by its heads."""
    w = W.small(dims=(16, 16, 8), slots=40, inputs=64, p=0.2)
    t = BatchTwin(w, frozen=False)
    other = S.VramState(t.N, t.A)
    first = N.ShardVramPtrs.from_buffer_copy(t.vram.ptrs)
    try:
        t.batch(10)
        other.upload_state(t.h_state)
        before = t.vram.download_state()
        for f, _ in N.ShardVramPtrs._fields_[:-1]:
            setattr(t.vram.ptrs, f, getattr(other.ptrs, f))
        t.batch(10)
        t.batch(10)
        for f, _ in N.ShardVramPtrs._fields_:
            setattr(t.vram.ptrs, f, getattr(first, f))
        assert np.array_equal(t.vram.download_state(), before), "the first allocation is left as it was"
    finally:
        t.vram.free()
        other.free()
