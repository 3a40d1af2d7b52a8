"""A shard stepped by the row engine and by the columnar kernels in turn, bit-exact against the oracle.

The columnar kernels (axc_batch_engine_mode(0), axc_tick_engine_mode(0)) move the weights of the .state blob
(physics.cu:281-373), so a row copy that the batch path or the per-tick entry point kept is out of date after
them.
"""
import ctypes as C

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


@pytest.mark.parametrize("zone", [False, True])
def test_a_batch_that_returned_an_error(gpu, zone):
    """The layout that a batch was to make is made by the next one when the batch failed before its ticks: here it is
    refused because its stream is being captured and it is to wait for its readout."""
    lib, cu = N.lib(), C.CDLL("libcuda.so.1")
    w = W.small(dims=(16, 16, 8), slots=40, inputs=64, p=0.2)
    t = BatchTwin(w, frozen=False)
    io, out = S.IoDeviceBuffers(t.words, 0, 32, 10), np.zeros(320, np.uint8)
    d_ids = S.device_array(np.arange(32, dtype=np.uint32))
    bm = S.input_bitmask(w.seed, 0, 10, w.num_inputs, w.rate_q32)
    stream, graph = C.c_void_p(), C.c_void_p()
    args = (t.N, t.A, io.as_struct(), N.ptr(bm), t.lay.virtual_offset, w.num_inputs)
    try:
        t.batch(10)
        rng = np.random.default_rng(3)   # other targets: the rows are out of date
        sv = StateView(t.h_state, t.N)
        sv.targets[:40] = sv.targets[:40][:, rng.permutation(t.N)]
        t.vram.upload_state(t.h_state)
        lib.gpu_device_synchronize()
        assert cu.cuStreamCreate(C.byref(stream), 1) == 0
        assert cu.cuStreamBeginCapture_v2(stream, 2) == 0
        if zone:
            z = N.AxcZoneShard()
            z.vram, z.padded_n, z.total_axons, z.io, z.h_input_bitmask, z.virtual_offset, z.num_virtual_axons = (
                t.vram.ptrs, *args)
            z.mapped_soma_ids_device, z.v_seg, z.h_output_history = d_ids, 1, N.ptr(out)
            err = lib.axc_step_zone_batch(C.byref(z), 1, None, 0, 10, t.tick, stream)
        else:
            err = lib.axc_step_day_phase_batch(C.byref(t.vram.ptrs), t.N, t.A, 10, C.byref(args[2]), N.ptr(bm), None,
                                               None, t.lay.virtual_offset, w.num_inputs, d_ids, 1, 0, t.tick,
                                               N.ptr(out), stream)
        assert err != 0
        cu.cuStreamEndCapture(stream, C.byref(graph))   # (an error: the capture is void)
        assert np.array_equal(t.vram.download_state(), t.h_state), "nothing ran"
        try:
            t.batch(10)
        except RuntimeError:
            pass   # the runtime hands the error out once more
        t.batch(10)
        t.batch(10)
    finally:
        if graph:
            cu.cuGraphDestroy(graph)
        if stream:
            cu.cuStreamDestroy_v2(stream)
        lib.gpu_free(d_ids)
        t.vram.free()
