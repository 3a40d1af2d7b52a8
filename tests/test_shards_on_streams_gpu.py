"""Shards of one process on streams of their own: a batch takes every SM for all its ticks only while no other shard's
work is under way, and stays bit-exact either way."""
import numpy as np
import pytest

import oracle
from axicor_gb300 import _native as N
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W

pytestmark = pytest.mark.gpu

ONE_LAUNCH = 6


class Brain:
    """6,400 neurons (a resident grid of blocks in a batch that has the GPU to itself), in step with the oracle."""

    def __init__(self, seed):
        self.w = W.small(dims=(20, 20, 16), slots=24, inputs=64, p=0.1, seed=seed)
        self.lay, self.state, self.heads = S.generate_brain(self.w.spec())
        self.n, self.A = self.lay.padded_n, self.lay.total_axons
        self.vram = S.VramState(self.n, self.A)
        self.vram.upload_state(self.state)
        self.vram.upload_axon_heads(self.heads)
        self.eng, self.tick, self.words = S.ShardEngine(self.vram), 0, 2
        # before the runs: an allocation between two of them would wait for the first
        self.io = {t: S.IoDeviceBuffers(self.words, 0, 0, t) for t in (4, 8, 1500)}

    def start(self, ticks, stream=None, use_graph=True):
        io = self.io[ticks]
        bm = S.input_bitmask(self.w.seed, self.tick, ticks, 64, self.w.rate_q32)
        own = self.eng.stream
        self.eng.stream = stream or own
        self.eng.step_day_phase_batch(ticks, io, bm, None, None, self.lay.virtual_offset, 64, None, 1, 0, self.tick,
                                      use_graph=use_graph)
        self.eng.stream = own
        self.tick += ticks
        return self.tick - ticks, ticks, bm

    def check(self, *runs):
        for tick, ticks, bm in runs:
            oracle.run_ticks(self.state, self.heads, self.w.lut, self.n, self.A, 1, tick, ticks, bm, self.words,
                             self.lay.virtual_offset, 64)
        N.lib().gpu_device_synchronize()
        assert np.array_equal(self.vram.download_heads(), self.heads)
        assert np.array_equal(self.vram.download_state(), self.state)
        return int(self.vram.forms(reset=True)[ONE_LAUNCH])


def test_a_batch_beside_another_shards_work(gpu):
    a, b = Brain(1), Brain(2)
    S.upload_lut(a.w.lut)
    try:
        assert a.check(a.start(8)) == 8 and b.check(b.start(8)) == 8, "alone: one launch"
        long = a.start(1500)        # some 15 ms of GPU time, queued
        beside = b.start(8)
        assert b.check(beside) == 0, "beside another shard's batch: the kernel chain"
        assert a.check(long) == 1500
        assert b.check(b.start(8)) == 8, "alone again"
        long = a.start(1500)
        assert b.check(b.start(8, stream=a.eng.stream)) == 8, "behind it on the same stream"
        assert a.check(long) == 1500
        ticks = a.start(4, use_graph=False)
        assert b.check(b.start(8)) == 0, "after another shard's per-tick calls"
        assert b.check(b.start(8)) == 8
        a.check(ticks)
    finally:
        a.vram.free()
        b.vram.free()


def test_a_freed_shard_is_forgotten(gpu):
    a, b = Brain(3), Brain(4)
    S.upload_lut(a.w.lut)
    try:
        long = a.start(1500)
        a.check(long)
        a.start(8)
        a.eng.synchronize()
        a.vram.free()
        assert b.check(b.start(8)) == 8
    finally:
        a.vram.free()
        b.vram.free()
