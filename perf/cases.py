"""The work that a user of this engine has it do, as cases that can be timed and compared.

A case is one pass through a public entry point on a brain that lives on the GPU: a batch of ticks of one shard
(``ShardEngine.step_day_phase_batch``, with its native loop or, as an unmodified caller of the drop-in boundary
does, one ``cu_step_day_phase`` per tick), of a zone's shards, of a population or of the learned-schedule engine; a
Night Phase sort-and-prune; a gradient of the activity predictor.  Sizes are those of ``axicor_gb300/workloads.py``
(16k, 1.5M and 8M neurons, populations of 1k to 100k), the smallest of the tests, and odd ones between.

The brains are drawn on the GPU with the statistics of ``workloads.py``: presynaptic axons with probability
proportional to exp(-distance / 4 voxels), segment 1 + distance / 2, weights of 50..800 signed by the presynaptic
type, one input to an input voxel.  ``prepare`` runs a brain's first ticks, so that a pass meets it in the regime
that its parameters lead to: saturated (every neuron fires as soon as its refractory period ends), or quiet
(homeostasis on: under one neuron in a hundred fires per tick).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from axicor_gb300 import _native as N
from axicor_gb300 import learned as L
from axicor_gb300 import shard as S
from axicor_gb300 import workloads as W

#: inertia falling over all ranks: no weight ever stops moving
GRADED = (128, 120, 100, 90, 80, 70, 60, 50, 40, 30, 20, 10, 8, 6, 4, 2)


def listed():
    return [
        # the smallest brains of the tests, stepped by an unmodified caller: one cu_step_day_phase per tick
        {"name": "tick-2k", "kind": "tick", "x": 16, "y": 16, "z": 8, "slots": 64, "inputs": 64, "outputs": 64,
         "ticks": 20, "warm": 200, "regime": "saturated"},
        # an agent's brain: 16k neurons, the batch loop
        {"name": "batch-16k", "kind": "batch", "x": 32, "y": 32, "z": 16, "slots": 128, "inputs": 256, "outputs": 256,
         "ticks": 100, "warm": 700, "regime": "saturated"},
        # the headline brain of the benchmark, in its settled regime
        {"name": "batch-1.5M", "kind": "batch", "x": 128, "y": 128, "z": 92, "slots": 100, "inputs": 4096,
         "outputs": 4096, "ticks": 100, "warm": 800, "regime": "saturated"},
        # the largest brain, short batches (20 ticks to a host round trip)
        {"name": "batch-8M", "kind": "batch", "x": 200, "y": 200, "z": 200, "slots": 128, "inputs": 8192,
         "outputs": 4096, "ticks": 20, "warm": 700, "regime": "saturated"},
        # a brain that learns all its life: every weight moves at every spike, dopamine, network spikes, odd sizes
        {"name": "plastic-500k", "kind": "batch", "x": 87, "y": 83, "z": 71, "slots": 96, "inputs": 1001,
         "outputs": 999, "ticks": 20, "warm": 100, "regime": "plastic"},
        # the headline brain kept quiet by homeostasis, input rate following a 100-tick cycle
        {"name": "quiet-1.5M", "kind": "batch", "x": 128, "y": 128, "z": 92, "slots": 100, "inputs": 4096,
         "outputs": 4096, "ticks": 100, "warm": 400, "regime": "quiet"},
        # the headline brain behind the drop-in boundary
        {"name": "tick-1.5M", "kind": "tick", "x": 128, "y": 128, "z": 92, "slots": 100, "inputs": 4096,
         "outputs": 4096, "ticks": 10, "warm": 800, "regime": "saturated"},
        # independent brains of 1k to 100k neurons stepped together
        {"name": "population-32", "kind": "population", "brains": 32, "ticks": 100, "warm": 600, "seed": 2},
        # the learned schedule on a quiet brain (the sparse form's regime)
        {"name": "learned-400k", "kind": "learned", "x": 96, "y": 64, "z": 64, "slots": 96, "inputs": 2048,
         "ticks": 100, "warm": 300, "collect": 100, "regime": "quiet"},
        # a zone: four shards with ghost axons between them; several neuron types of different propagation lengths,
        # adaptive leak, heartbeats and network spikes
        {"name": "zone-4", "kind": "zone", "shards": 4, "x": 37, "y": 37, "z": 37, "slots": 80, "inputs": 512,
         "outputs": 512, "ghosts": 1024, "ticks": 20, "warm": 200, "regime": "mixed"},
        # Night Phase: every neuron's slots sorted by weight and the weak ones pruned
        {"name": "night-1M", "kind": "night", "x": 101, "y": 103, "z": 97, "slots": 100, "inputs": 1024},
        # a training step's forward and backward of the activity predictor
        {"name": "mlp-grad-100k", "kind": "mlp", "count": 100_000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tick", "batch", "batch", "batch", "population", "learned", "zone", "night", "mlp"])
    if kind == "mlp":
        return {"kind": "mlp", "count": _log(rng, 1000, 200_000)}
    if kind == "population":
        return {"kind": "population", "brains": rng.randint(4, 32), "ticks": rng.choice([20, 50, 100]), "warm": 400,
                "seed": rng.randint(3, 1 << 20)}
    top = {"tick": 1_500_000, "batch": 2_000_000, "learned": 800_000, "zone": 100_000, "night": 2_000_000}[kind]
    edge = _log(rng, 1500, top) ** (1.0 / 3.0)
    x, y = (max(8, int(round(edge * rng.uniform(0.8, 1.25)))) for _ in range(2))
    z = max(8, int(round(edge ** 3 / (x * y))))
    n = x * y * z
    c = {"kind": kind, "x": x, "y": y, "z": z, "slots": rng.randint(24, 128), "inputs": rng.randint(32, max(33, n // 64))}
    if kind == "night":
        return c
    c.update(ticks=rng.choice([10, 20, 50]) if kind != "tick" else rng.choice([5, 10, 20]), warm=rng.choice([100, 300, 700]),
             regime=rng.choice(["saturated", "plastic", "quiet", "mixed"]))
    if kind == "learned":
        c.update(regime=rng.choice(["quiet", "saturated"]), collect=50, ticks=50)
        return c
    c["outputs"] = rng.randint(1, min(n, 4096))
    if kind == "zone":
        c.update(shards=rng.randint(2, 4), ghosts=rng.randint(1, min(1024, c["inputs"] // 2)))
    return c


# ---------------------------------------------------------------------------
# brains
# ---------------------------------------------------------------------------
def _lut(case):
    r = case.get("regime", "saturated")
    lut = W.default_lut()
    if r == "quiet":
        for v in (0, 1):
            lut[v]["homeostasis_penalty"] = 16000
            lut[v]["homeostasis_decay"] = 80
    if r in ("plastic", "mixed"):
        for v in (0, 1):
            lut[v]["inertia_curve"] = np.array(GRADED, np.uint8)
            lut[v]["d1_affinity"], lut[v]["d2_affinity"] = 64, 32
    if r == "mixed":
        lut[2], lut[3] = lut[0].copy(), lut[1].copy()
        lut[2]["signal_propagation_length"] = 6
        lut[2]["adaptive_mode"], lut[2]["adaptive_leak_gain"], lut[2]["adaptive_leak_max"] = 1, 32, 400
        lut[2]["homeostasis_penalty"], lut[2]["homeostasis_decay"] = 900, 40
        lut[3]["signal_propagation_length"] = 3
        lut[3]["spontaneous_firing_period_ticks"] = 211
    return lut


_lut_on_gpu = None


def _use_lut(lut):
    """The process LUT, uploaded at boot as a program does: not again for another brain of the same types."""
    global _lut_on_gpu
    if _lut_on_gpu != lut.tobytes():
        S.upload_lut(lut)
        _lut_on_gpu = lut.tobytes()


def _rates(case):
    return W.sinusoid_rates() if case.get("regime") == "quiet" else np.array([W.p_q32(0.05)], np.uint32)


class _Mem:
    """Device memory of a shard for torch (__cuda_array_interface__); keeps its owner alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3,
                                         "strides": None}


def _view(owner, ptr, shape, typestr):
    return torch.as_tensor(_Mem(owner, int(ptr), shape, typestr), device="cuda")


class _Owner:
    """A shard's memory and what a program keeps beside it; freed when nothing refers to it any more."""

    def __init__(self, vram):
        self.vram = vram


_tables = {}


def _offset_table():
    """Voxel offsets (dx, dy, dz) and segments, drawn with probability proportional to exp(-d / 4) within 48
    voxels, as 2^22 quantiles."""
    if "t" not in _tables:
        r = torch.arange(-48, 49, device="cuda", dtype=torch.float32)
        dx, dy, dz = torch.meshgrid(r, r, r, indexing="ij")
        d = torch.sqrt(dx * dx + dy * dy + dz * dz)
        keep = (d > 0) & (d <= 48)
        dx, dy, dz, d = dx[keep], dy[keep], dz[keep], d[keep]
        cdf = torch.cumsum(torch.exp(-d.double() / 4.0), 0)
        q = (torch.arange(1 << 22, device="cuda", dtype=torch.float64) + 0.5) / (1 << 22) * cdf[-1]
        i = torch.searchsorted(cdf, q)
        _tables["t"] = (torch.stack([dx, dy, dz])[:, i].to(torch.int32), (1 + (d[i].to(torch.int32) >> 1)))
    return _tables["t"]


class _Brain:
    """One shard with a seeded brain, its engine and its batch I/O."""

    def __init__(self, dims, slots, inputs, seed, lut, types=2, ghosts=0):
        x, y, z = dims
        n = x * y * z
        self.n, self.slots, self.nv = n, slots, inputs - ghosts
        self.N = (n + 63) // 64 * 64
        self.A = (self.N + inputs + 31) // 32 * 32
        self.voff, self.ghost0 = self.N, self.N + self.nv
        self.vram = S.VramState(self.N, self.A)
        own, p, M = _Owner(self.vram), self.vram.ptrs, self.N
        self.volt = _view(own, p.soma_voltage, (M,), "<i4")
        self.flags = _view(own, p.soma_flags, (M,), "|u1")
        self.thr = _view(own, p.threshold_offset, (M,), "<i4")
        self.timers = _view(own, p.timers, (M,), "|u1")
        s2a = _view(own, p.soma_to_axon, (M,), "<i4")
        self.targets = _view(own, p.dendrite_targets, (128, M), "<i4")
        self.weights = _view(own, p.dendrite_weights, (128, M), "<i2")
        self.dtimers = _view(own, p.dendrite_timers, (128, M), "|u1")
        self.heads = _view(own, p.axon_heads, (self.A, 8), "<i4")
        self.blob = _view(own, p.soma_voltage, (S.BYTES_PER_NEURON * M // 4,), "<i4")   # the whole .state
        g = torch.Generator(device="cuda").manual_seed(seed)
        u = torch.rand(n, device="cuda", generator=g)
        inh = u < 0.2
        kind = inh.to(torch.uint8)
        if types == 4:   # a third of each kind has the second excitatory / inhibitory type
            kind += 2 * (torch.rand(n, device="cuda", generator=g) < 1 / 3).to(torch.uint8)
        self.flags[:n] = kind << 4
        s2a.fill_(-1)
        s2a[:n] = torch.arange(n, device="cuda", dtype=torch.int32)
        # input v sits on a voxel of its own; half of the draws of that voxel take the input
        inputs = min(inputs, n)
        site = torch.randperm(n, device="cuda", generator=g)[:inputs]
        input_at = torch.full((n,), -1, device="cuda", dtype=torch.int32)
        input_at[site] = torch.arange(inputs, device="cuda", dtype=torch.int32)
        off, seg = _offset_table()
        me = torch.arange(n, device="cuda", dtype=torch.int32)
        px, py, pz = me % x, (me // x) % y, me // (x * y)
        for s in range(slots):
            k = torch.randint(1 << 22, (n,), device="cuda", generator=g)
            o = off[:, k]
            pre = ((px + o[0]) % x) + x * (((py + o[1]) % y) + y * ((pz + o[2]) % z))
            pre = torch.where(pre == me, (pre + 1) % n, pre)
            w = torch.randint(50, 801, (n,), device="cuda", generator=g, dtype=torch.int32)
            iv = input_at[pre]
            from_input = (iv >= 0) & (w & 1 == 1)
            w = torch.where(inh[pre] & ~from_input, -w, w)
            axon = torch.where(from_input, self.voff + iv, pre)
            self.targets[s, :n] = (seg[k] << 24) | (axon + 1)
            self.weights[s, :n] = w.to(torch.int16)
        torch.cuda.synchronize()
        N.lib().axc_shard_invalidate(C.byref(p))   # the blob was written without the library
        _use_lut(lut)

    def outputs(self):
        return {"voltage": self.volt, "flags": self.flags, "threshold": self.thr, "timers": self.timers,
                "weights": self.weights[:self.slots], "heads": self.heads}


class _Loop:
    """What ShardEngine's caller keeps for its batches: the engine, device I/O buffers, the next inputs."""

    def __init__(self, brain, case, seed, network=0):
        self.b, self.ticks, self.words = brain, case["ticks"], (brain.nv + 31) // 32
        self.network = network
        self.eng = S.ShardEngine(brain.vram)
        self.n_out = case.get("outputs", 0)
        ids = np.linspace(0, brain.n - 1, self.n_out).astype(np.uint32)
        self.ids = torch.from_numpy(ids.view(np.int32)).cuda()
        self.seed, self.rates, self.tick = seed, _rates(case), 0
        self.dopamine = 20 if case.get("regime") in ("plastic", "mixed") else 0
        self.open(case["ticks"], 8)

    def open(self, ticks, batches):
        """I/O buffers and `batches` batches' inputs of `ticks` ticks from here."""
        self.ticks = ticks
        self.io = S.IoDeviceBuffers(self.words, max(self.network, 0), self.n_out, ticks)
        bm = S.input_bitmask(self.seed, self.tick, ticks * batches, self.b.nv, self.rates)
        self.bms = [S.PinnedBuffer(self.words * ticks, np.uint32) for _ in range(batches)]
        for i, b in enumerate(self.bms):
            b.array[:] = bm[i * b.len:(i + 1) * b.len]
        self.out = S.PinnedBuffer(max(self.n_out * ticks, 1), np.uint8)
        self.spikes = self.counts = None
        if self.network:
            r = np.random.default_rng(self.seed)
            self.spikes = [r.integers(0, self.b.A, ticks * self.network, dtype=np.uint32) for _ in range(batches)]
            self.counts = [r.integers(0, self.network + 1, ticks, dtype=np.uint32) for _ in range(batches)]

    def step(self, graph):
        i = (self.tick // self.ticks) % len(self.bms)
        self.eng.step_day_phase_batch(
            self.ticks, self.io, self.bms[i].array, self.spikes[i] if self.spikes else None,
            self.counts[i] if self.counts else None, self.b.voff, self.b.nv, self.ids.data_ptr() if self.n_out else None,
            1, self.dopamine, self.tick, h_output_history=self.out.array if self.n_out else None, use_graph=graph)
        self.tick += self.ticks

    def warm(self, ticks):
        if ticks:
            per, n_out, self.n_out = self.ticks, self.n_out, 0
            self.open(min(ticks, 50), -(-ticks // min(ticks, 50)))
            for _ in range(len(self.bms)):
                self.step(True)
            self.eng.synchronize()
            self.n_out, self.tick = n_out, -(-self.tick // per) * per
            self.open(per, 8)


def _dims(c):
    return (c["x"], c["y"], c["z"])


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _prepare_mlp(case, seed)
    if kind == "population":
        return _Population(case, seed)
    if kind == "zone":
        return _Zone(case, seed)
    lut = _lut(case)
    b = _Brain(_dims(case), case["slots"], case["inputs"], seed, lut, 4 if case.get("regime") == "mixed" else 2)
    if kind == "night":
        return _Night(b, seed)
    if kind == "learned":
        return _Learned(b, case, seed)
    loop = _Loop(b, case, seed, network=64 if case["regime"] in ("plastic", "mixed") else 0)
    loop.warm(case["warm"])
    return _Shard(loop, kind == "batch")


def run(state):
    return state.run()


class _Shard:
    def __init__(self, loop, graph):
        self.loop, self.graph = loop, graph

    def run(self):
        self.loop.step(self.graph)
        return {"readout": self.loop.out.array, **self.loop.b.outputs()}


class _Night:
    """A brain after a day: weights spread over the whole range, the weak and the strong mixed in each row."""

    def __init__(self, b, seed):
        self.b = b
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        for s in range(b.slots):
            m = torch.randint(0, 4096, (b.N,), device="cuda", generator=g, dtype=torch.int32)
            b.weights[s] = torch.where(b.weights[s] < 0, -m, m).to(torch.int16)
            b.dtimers[s] = (m & 0xFF).to(torch.uint8)
        torch.cuda.synchronize()
        N.lib().axc_shard_invalidate(C.byref(b.vram.ptrs))

    def run(self):
        N.lib().launch_sort_and_prune(C.byref(self.b.vram.ptrs), self.b.N, 100)
        return {"targets": self.b.targets, "weights": self.b.weights, "timers": self.b.dtimers, "flags": self.b.flags}


class _Learned:
    def __init__(self, b, case, seed):
        self.b, self.ticks = b, case["ticks"]
        words = (b.nv + 31) // 32
        rows = case["warm"] + case["collect"] + case["ticks"]
        bm = S.input_bitmask(seed, 0, rows, b.nv, _rates(case))
        self.bm = torch.from_numpy(bm.view(np.int32)).cuda()
        self.tick0 = case["warm"] + case["collect"]
        self.eng = L.LearnedEngine(b.vram, b.N, b.A, b.voff, b.nv, self.bm.data_ptr(), words, rows,
                                   sample_capacity=20_000)
        self.eng.set_policy(L.Policy(policy=0))
        self.eng.run(0, case["warm"], 50)
        self.eng.collect(True, sample_every=2, reset=True)
        self.eng.run(case["warm"], case["collect"], 50)
        self.eng.collect(False)
        self.eng.train(epochs=4, batch=512, lr=2e-3, seed=5)
        self.eng.set_policy(L.Policy(policy=-1))

    def run(self):
        self.eng.run(self.tick0, self.ticks, 50)
        return self.b.outputs()


class _Population:
    """Brains of workloads.population: 1k to 100k neurons, each with its own types and inputs."""

    def __init__(self, case, seed):
        self.ticks, self.warm = case["ticks"], case["warm"]
        rows = self.warm + self.ticks
        self.brains, self.keep, descs = [], [], []
        for i, w in enumerate(W.population(seed=case["seed"], count=case["brains"], ticks=rows)):
            b = _Brain(w.dims, w.slots, w.num_inputs, seed * 1000 + i, W.default_lut())
            words = (b.nv + 31) // 32
            bm = torch.from_numpy(S.input_bitmask(seed + i, 0, rows, b.nv, w.rate_q32).view(np.int32)).cuda()
            lut = torch.from_numpy(np.ascontiguousarray(w.lut).view(np.uint8)).cuda()
            d = N.AxcPopBrainDesc()
            d.vram, d.padded_n, d.total_axons = b.vram.ptrs, b.N, b.A
            d.virtual_offset, d.num_virtual = b.voff, b.nv
            d.d_input_bitmask, d.words_per_tick, d.bitmask_ticks = bm.data_ptr(), words, rows
            d.v_seg, d.d_lut, d.dopamine, d.tick_base = 1, lut.data_ptr(), 0, 0
            self.brains.append(b)
            self.keep += [bm, lut]
            descs.append(d)
        torch.cuda.synchronize()
        h = C.c_void_p()
        N.check(N.lib().axc_population_create((N.AxcPopBrainDesc * len(descs))(*descs), len(descs), C.byref(h)),
                "axc_population_create")
        self.handle = h.value
        if self.warm:
            N.check(N.lib().axc_population_run(self.handle, 0, self.warm, 50, None), "axc_population_run")

    def run(self):
        N.check(N.lib().axc_population_run(self.handle, self.warm, self.ticks, min(self.ticks, 50), None),
                "axc_population_run")
        return [(b.blob, b.heads) for b in self.brains]

    def __del__(self):
        try:
            if self.handle:
                torch.cuda.synchronize()
                N.lib().axc_population_destroy(self.handle)
        except Exception:
            pass


class _Zone:
    def __init__(self, case, seed):
        self.case = case
        lut = _lut(case)
        self.loops = []
        for i in range(case["shards"]):
            b = _Brain(_dims(case), case["slots"], case["inputs"] + case["ghosts"], seed * 100 + i, lut,
                       4 if case["regime"] == "mixed" else 2, ghosts=case["ghosts"])
            self.loops.append(_Loop(b, case, seed * 100 + i, network=32))
            self.loops[-1].warm(case["warm"])
        rng = np.random.default_rng(seed)
        n, g = len(self.loops), case["ghosts"]
        self.idx, routes = [], []
        for i in range(n):
            dst = self.loops[(i + 1) % n].b
            src = torch.from_numpy(rng.choice(self.loops[i].b.n, size=g, replace=False).astype(np.int32)).cuda()
            to = torch.arange(dst.ghost0, dst.ghost0 + g, device="cuda", dtype=torch.int32)
            self.idx += [src, to]
            routes.append(N.AxcGhostRoute(i, (i + 1) % n, src.data_ptr(), to.data_ptr(), g))
        self.routes = (N.AxcGhostRoute * n)(*routes)
        self.shards = (N.AxcZoneShard * n)()
        torch.cuda.synchronize()

    def run(self):
        for z, lp in zip(self.shards, self.loops):
            i = (lp.tick // lp.ticks) % len(lp.bms)
            z.vram, z.padded_n, z.total_axons, z.io = lp.b.vram.ptrs, lp.b.N, lp.b.A, lp.io.as_struct()
            z.h_input_bitmask = lp.bms[i].as_ptr()
            z.h_incoming_spikes, z.h_spike_counts = N.ptr(lp.spikes[i]), N.ptr(lp.counts[i])
            z.virtual_offset, z.num_virtual_axons = lp.b.voff, lp.b.nv
            z.mapped_soma_ids_device, z.v_seg, z.dopamine = lp.ids.data_ptr(), 1, lp.dopamine
            z.h_output_history = lp.out.as_ptr()
        ticks, tick = self.loops[0].ticks, self.loops[0].tick
        N.check(N.lib().axc_step_zone_batch(self.shards, len(self.loops), self.routes, len(self.loops), ticks, tick,
                                            self.loops[0].eng.stream), "axc_step_zone_batch")
        for lp in self.loops:
            lp.tick += ticks
        return [{"readout": lp.out.array, **lp.b.outputs()} for lp in self.loops]


def _mlp_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.randn(N.lib().axc_mlp_param_count(), device="cuda", generator=g) * 0.1
    x = torch.rand(case["count"], L.FEATURES, device="cuda", generator=g)
    y = torch.rand(case["count"], device="cuda", generator=g)
    return p, x, y


class _prepare_mlp:
    def __init__(self, case, seed):
        self.p, self.x, self.y = _mlp_inputs(case, seed)
        self.grad, self.loss = torch.zeros_like(self.p), torch.zeros(1, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        N.check(N.lib().axc_mlp_loss_grad(self.p.data_ptr(), self.x.data_ptr(), self.y.data_ptr(), self.y.numel(),
                                          self.grad.data_ptr(), self.loss.data_ptr(), None), "axc_mlp_loss_grad")
        return {"loss": self.loss, "grad": self.grad}


def exact(case, seed):
    """The predictor's loss and gradient in 64 bits (parameters and inputs rounded to BF16, as they are stored);
    the engine's other outputs are integers that two right answers share bit for bit."""
    if case["kind"] != "mlp":
        return None
    p, x, y = (t.double() for t in _mlp_inputs(case, seed))
    p, x = p.bfloat16().double(), x.bfloat16().double()
    f, h = L.FEATURES, L.HIDDEN
    w1, b1, w2, b2 = p[:h * f].view(h, f), p[h * f:h * f + h], p[h * f + h:h * f + 2 * h], p[-1]
    pre = x @ w1.T + b1
    act = pre.clamp(min=0)
    err = act @ w2 + b2 + x[:, 8] - y
    d = 2.0 * err / y.numel()
    da = d[:, None] * w2 * (pre > 0)
    grad = torch.cat([(da.T @ x).reshape(-1), da.sum(0), act.T @ d, d.sum().reshape(1)])
    return {"loss": (err * err).mean().reshape(1), "grad": grad}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _brain_work(n, slots, inputs, moves):
    """The dendrites read once (target 4 B, weight 2 B; 2 B written where the weights move), soma state read and
    written once (voltage, threshold, flags, timer; axon id read), heads read and written once."""
    return n * slots * (6 + (2 if moves else 0)) + n * 24 + (n + inputs) * 64


def work(case):
    if case["kind"] == "mlp":
        c, f, h = case["count"], L.FEATURES, L.HIDDEN
        return {"bytes": c * (f + 1) * 4 + 2 * 4 * (h * f + 2 * h + 1), "flops": c * (4 * f * h + 6 * h)}
    if case["kind"] == "population":
        ws = W.population(seed=case["seed"], count=case["brains"], ticks=1)
        return {"bytes": sum(_brain_work(w.num_neurons, w.slots, w.num_inputs, False) for w in ws)
                + case["ticks"] * sum(w.num_inputs for w in ws) / 8, "flops": 0}
    n = case["x"] * case["y"] * case["z"]
    if case["kind"] == "night":
        return {"bytes": n * (2 * 128 * 7 + 2), "flops": 0}
    one = _brain_work(n, case["slots"], case["inputs"], case["regime"] in ("plastic", "mixed"))
    one += case["ticks"] * (case["inputs"] / 8 + case.get("outputs", 0))
    return {"bytes": one * case.get("shards", 1) + 128 * case.get("ghosts", 0) * case.get("shards", 0), "flops": 0}
