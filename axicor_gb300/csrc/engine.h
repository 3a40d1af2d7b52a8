// engine.h — internal declarations shared by the engine's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <tuple>
#include <type_traits>
#include <utility>

#include "../../include/axicor_day.h"
#include "per_device.h"

namespace axc {

// Launches kernel k and returns the status of that launch alone
// (cudaLaunchKernel's return value), without reading or clearing an error
// that an earlier call left pending.  Arguments convert to the kernel's
// parameter types.
template <typename... P, typename... A, size_t... I>
cudaError_t launch_k_impl(void (*k)(P...), dim3 g, dim3 b, cudaStream_t s, std::index_sequence<I...>, A&&... a) {
  std::tuple<std::decay_t<P>...> t(static_cast<std::decay_t<P>>(std::forward<A>(a))...);
  void* args[sizeof...(P) > 0 ? sizeof...(P) : 1] = {static_cast<void*>(&std::get<I>(t))...};
  return cudaLaunchKernel(reinterpret_cast<const void*>(k), g, b, args, 0, s);
}
template <typename... P, typename... A>
cudaError_t launch_k(void (*k)(P...), dim3 g, dim3 b, cudaStream_t s, A&&... a) {
  static_assert(sizeof...(P) == sizeof...(A), "one argument per kernel parameter");
  return launch_k_impl(k, g, b, s, std::index_sequence_for<P...>{}, std::forward<A>(a)...);
}

// Control block of one shard in device memory.
struct ShardCtl {
  uint32_t spike_count;   // spikers listed by the last update stage
  uint32_t err;           // AXC_ERR_* bits, sticky until read with clear
  uint32_t tick_base;     // batch mode: global tick of tick 0 of the batch
  int32_t dopamine;       // batch mode: dopamine of the batch
  uint32_t fix_count;     // row engine: GSOP slots deferred to the fix-up stage
  uint32_t fix_overflow;  // row engine: the fix-up list overflowed, rescan the spikers
  alignas(8) uint32_t eval_act[2][2];  // row engine, tick k (slot k & 1): [0] non-refractory neurons listed, [1] axons
                           // with a head on a segment of the batch (8-byte aligned pairs: one atomic adds both)
  uint32_t row_smax;      // row engine: longest row (slots before the first empty) of the batch
  uint32_t seg_max;       // row engine: largest segment of a live slot in the batch
  unsigned long long row_sum;  // row engine: checksum of the batch's targets (slot order)
  uint32_t pmax;          // row engine: largest signal_propagation_length of the LUT (batch start)
  uint32_t barrier;       // row engine: arrivals at the barriers of k_rows_small's resident grid
  unsigned long long ctr[8];  // statistics, see axc_shard_counters
  uint32_t dense[2];      // row engine: axons of tick k (slot k & 1) off the lit set the row layout assumed
  unsigned long long pfx_total;   // row engine: slots of the rows tested on every tick (batch start)
  unsigned long long slot_total;  // row engine: live slots of the rows (batch start)
  uint32_t lay_now;       // row engine: this batch lays the row copy out anew (layout_decide)
  uint32_t lay_since;     // row engine: ticks since the last layout
  uint32_t lay_every;     // row engine: ticks between layouts while the lit-sum criterion holds
  uint32_t lay_wait;      // row engine: ticks a layout must last while it does not hold
  uint32_t lay_lit;       // row engine: fully-lit axons when the layout was made
  uint32_t dec_ticks;     // row engine: ticks of the last decision
  uint32_t lay_forced;    // row engine: the layout was forced
  uint32_t gave_up;       // row engine: a barrier of k_rows_small's resident grid ran out of tries
  unsigned long long mov_total;   // row engine: movable slots of the rows (batch start)
  unsigned long long lit_seen;    // row engine: ctr[6] at the last decision
  unsigned long long lay_work;    // row engine: tested and movable slots of the layout before the current one
  unsigned long long gsop_same[2];  // row engine: 4-slot groups the 8-lane pass's GSOP visited and left as they
                                    // were, and all it visited, since the last decision
  uint32_t mixed_len;     // row engine: a neuron with slots has another signal_propagation_length than pmax
  uint32_t streak;        // row engine: consecutive ticks that the sparse form could have run (sparse_tick)
  uint32_t idx_ok;        // row engine: an inverted index was built (it holds while idx_sum == lay_sum)
  uint32_t busy;          // row engine: consecutive ticks that it could not have run, up to kBusyStreak
  uint32_t ix_run;        // row engine: the graph that runs has the sparse form's kernels
  uint32_t busy_told;     // row engine: the host's pinned word says that busy reached kBusyStreak
  unsigned long long lay_sum, idx_sum;  // row engine: checksum of the rows' targets by position; the index's rows'
  const uint32_t* ix_off; // inverted index of the rows (RowIndex)
  const uint16_t* ix_seg;
  const uint32_t* ix_ent;
  uint32_t lay_segs;      // row engine: layouts since the last forced one, up to 2 (keep_segs)
  uint32_t pad3;
  unsigned long long forms[8];   // row engine: ticks per form, one-launch ticks, layouts (axc_shard_forms)
};

// Inverted index of the row copy: per axon the row slots that target it
// (n * 128 + row position), those of one segment together, for the sparse
// form of a tick (row_engine.cuh).  The learned engine's: allocated when its
// brain first turns quiet (576 bytes a neuron and axon, room for 128 slots a row
// whatever it holds; the batch and per-tick paths allocate nothing beyond the row
// copy).
struct RowIndex {
  void* base = nullptr;
  uint32_t* off = nullptr;  // [A+1] first entry of an axon
  uint32_t* cur = nullptr;  // [A] fill cursor (build)
  uint32_t* bsum = nullptr; // scan block sums (build)
  uint16_t* seg = nullptr;  // [A][32] entries of an axon before segment s (s = 31: all segments >= 31);
                            // kSegUnsorted in [0]: too many entries, unsorted
  uint32_t* ent = nullptr;  // [N * 128], the live slots first
};

// Neuron-major copy of the dendrites used by the batch engine for the length
// of one batch (row_engine.cuh).
struct RowCache {
  uint32_t N = 0, A = 0;
  void* base = nullptr;
  uint32_t* rt = nullptr;   // [N][128] targets, neuron-major
  int16_t* rw = nullptr;    // [N][128] weights, neuron-major
  uint16_t* cnt = nullptr;  // [N] slots before the first empty target; bit 15: an invalid target, 14: split (kRowSplit)
  uint2* mask2 = nullptr;   // [A+1] split segment-hit masks (heads 0..6 | head 7); [A] dummy
  uint32_t* axw = nullptr;  // [A] owners and used segments of the axon (kAxOwned); population: somas that own it
  uint32_t* eval = nullptr; // [N] non-refractory neurons of the tick
  uint32_t* fix = nullptr;  // [kFixCap] deferred GSOP slots (n*128 + slot)
  uint32_t* lit = nullptr;  // [A/32+1] fully-lit axons of the tick, one bit each
  uint32_t* live = nullptr; // [A/32+1] axons with a head on a segment of the batch this tick, one bit each
  uint32_t* evb = nullptr;  // [N/32+1] neurons evaluated this tick, one bit each
  int32_t* acc = nullptr;   // [N] input current of the sparse form (zero between ticks)
  uint32_t* gs_n = nullptr; // [N] spikers with 1..8 slots GSOP may move (a thread each)
  uint32_t* gd_n = nullptr; // [N] spikers with more (8 lanes each)
  uint4* amask = nullptr;   // [N] row positions (bit q) whose weights GSOP may move (set at batch start)
  uint8_t* lfz = nullptr;   // [N] number of those slots (set at batch start)
  uint4* omask = nullptr;   // [N] columnar slots placed first in the row (the movable ones; all when unpermuted)
  uint32_t* wcnt = nullptr; // [2][kMaxUpdateWarps] spikers each warp of the update pass listed (gs_n, gd_n)
  int2* rec = nullptr;      // [N] x: wrapping sum of the row's lit-sum weights, y: its groups' bounds (build_row)
  uint4* lmask = nullptr;   // [N] the columnar slots of omask placed before the others (movable, lit)
  uint32_t* alit = nullptr; // [A/32+1] axons fully lit in every one of the last ticks (kLitWindow)
  uint32_t* xlit = nullptr; // [A/32+1] axons (of alit) taken as fully lit when the row layout was made
  RowIndex ix;
  bool ix_failed = false;   // no room for the index: not tried again
  uint8_t* posmap = nullptr;  // [N][128] row position of each columnar slot (learned engine only; own allocation)
};

// Per-shard scratch owned by the engine, next to the reference-visible
// state.  Sized for (padded_n, total_axons).
struct ShardScratch {
  uint32_t padded_n = 0;
  uint32_t total_axons = 0;
  void* base = nullptr;        // single allocation
  uint32_t* seg_mask = nullptr;  // [A] segment-hit mask of the propagated heads
  uint32_t* pend = nullptr;      // [A] soma pushes pending for the push stage
  uint32_t* incoming = nullptr;  // [A] network spike pushes pending for the axon stage
  uint32_t* spikers = nullptr;   // [N] ids of the neurons that spiked this tick
  ShardCtl* ctl = nullptr;
  uint32_t* batch_counts = nullptr;  // [batch_cap] per-tick network spike counts
  uint32_t batch_cap = 0;
  uint32_t* h_counts_pinned = nullptr;  // pinned: [0] the device asks for an inverted index (RowIndex), [1] busy_told
  bool ix_run = false;                  // ShardCtl::ix_run as last set
  void* graph_cache = nullptr;          // batch engine graphs (batch_engine.cu)
  RowCache* rows = nullptr;             // batch engine neuron-major dendrites
  // Per-tick entry point (cu_step_day_phase): its row cache lives across calls.
  // It is valid while nothing else wrote the shard's targets, weights, flags or
  // soma_to_axon and the LUT is the one it was built with; every entry point
  // of this library that writes them clears the flag.
  std::atomic<bool> tick_rows_valid{false};
  uint64_t tick_rows_lut = 0;           // LUT generation the per-tick row cache was built with
  uint32_t tick_parity = 0;             // per-tick calls alternate the row engine's list slots
  uint32_t tick_since_build = 0;        // per-tick calls since the row copy was laid out
  const void* state_base = nullptr;     // the shard's .state allocation (invalidation by address)
  size_t state_bytes = 0;
  // Batch path: the row copy (layout, weights, lit-sum sums) is kept from one
  // batch to the next while it matches the shard's memory and the LUT (the
  // device decides each batch whether to lay it out anew: layout_decide).
  // Cleared by every route that clears tick_rows_valid, and by the per-tick
  // entry point; the next batch then lays the rows out for sure.
  std::atomic<bool> batch_rows_valid{false};
  uint64_t batch_rows_lut = 0;           // LUT generation of the batch layout
  // What others_running looks at (batch_engine.cu, under its lock).
  cudaEvent_t work_done = nullptr;      // behind the shard's last batch or run
  cudaStream_t work_stream = nullptr;
  bool work_listed = false;             // not known to be done
  uint64_t own_ticks = 0;               // per-tick calls of this shard, of all others at its last batch
  uint64_t other_ticks = 0;
};

// The shards of a process share the GPU: a batch that takes every SM for all of its
// ticks (k_rows_small's resident grid) would make the others' wait, kernel by kernel
// they run beside each other (four shards of 16,384 saturated neurons on streams of
// their own: 39.0 us a tick of all four in resident grids, 18.4 in chains).
// Behind a batch's, run's or zone's launches on st, and for each per-tick call:
void work_started(ShardScratch& s, cudaStream_t st);
void tick_started(ShardScratch& s);
// Another shard's batch or run is under way on another stream, or another shard was
// stepped tick by tick since this one's last batch.
bool others_running(ShardScratch& s, cudaStream_t st);
void work_created(ShardScratch& s);   // a new shard: the ticks before it are none of its batches'
void work_forget(ShardScratch& s);

constexpr uint32_t kLitWindow = 32;   // last ticks before a layout in which an axon must have been fully lit
constexpr uint32_t kBatchRelayoutMin = 100, kBatchRelayoutMax = 1600;   // ticks between batch layouts

uint64_t lut_generation();

// Whether the next batch must lay the row copy out anew whatever the device
// decides (the kept copy is stale or from another LUT); marks the copy the
// batch leaves as valid.
inline bool batch_rows_force(ShardScratch& s) {
  const uint64_t gen = lut_generation();
  const bool force = !(s.batch_rows_valid.load() && s.batch_rows_lut == gen);
  s.batch_rows_lut = gen;
  s.batch_rows_valid.store(true);
  return force;
}

#ifdef __CUDACC__
#define AXC_HD __host__ __device__
#else
#define AXC_HD
#endif

// The current layout meets the lit-sum criterion: at most an eighth of the live
// slots are tested one by one.
AXC_HD inline bool layout_met(const ShardCtl* c) { return c->slot_total > 0 && c->pfx_total * 8ull <= c->slot_total; }

// The layout decision for the next `ticks` ticks (lit: always-lit axons of the last
// ticks, counted when forced or not met; index: the ticks may run the sparse form).
// A new layout when forced; every lay_every ticks, doubling from
// kBatchRelayoutMin to kBatchRelayoutMax, while the current one meets the
// lit-sum criterion (at most an eighth of the live slots tested); while it does
// not, when a tenth more axons are fully lit than when it was made; while it
// does, when axons it took as lit were dark on half of the ticks; and in both
// cases when an eighth of the groups of movable slots that GSOP visited since the
// last decision no longer moved; but for these at most every lay_wait ticks,
// doubling from 16 while the new layouts gain less than a tenth, and at least
// every kBatchRelayoutMax.  A brain whose weights never freeze, or that is
// quiet, so keeps its layout instead of paying for one each batch (1.6 ms at
// 1.5M neurons).  The layout kernels of the batch return at once when lay_now is 0.
AXC_HD inline void layout_decision(ShardCtl* c, uint32_t force, uint32_t ticks, uint32_t lit, bool index) {
  // the layout meets the criterion, and its lit axons stayed lit on most ticks since the last decision
  const bool met = layout_met(c);
  const unsigned long long lit6 = c->ctr[6] < c->lit_seen ? c->ctr[6] : c->ctr[6] - c->lit_seen;
  const bool missed = met && lit6 * 2ull < c->dec_ticks;   // ticks with dark axons
  if (!index) c->streak = 0;   // of the learned engine's last ticks
  bool build = force;
  const bool froze = c->gsop_same[0] > 0 && c->gsop_same[0] * 8ull >= c->gsop_same[1];
  if (!force && met) {
    build = c->lay_since >= c->lay_every || ((froze || missed) && c->lay_since >= c->lay_wait);
  } else if (!force) {
    const bool grew = (unsigned long long)lit * 10ull > (unsigned long long)c->lay_lit * 11ull;
    // (the sparse form reads no more than the movable slots of a few spikers: its rows stay)
    build = (c->lay_since >= kBatchRelayoutMax && c->streak == 0u) ||
            (c->lay_since >= c->lay_wait && (froze || grew) && c->slot_total > 0);
  }
  if (build && (force || !met)) c->lay_lit = force ? 0u : lit;   // a forced layout leaves movable slots out
  // the last layout left a tenth fewer tested and movable slots than the one before
  const bool paid = (c->pfx_total + c->mov_total) * 10ull < c->lay_work * 9ull;
  if (build) {
    const uint32_t twice = 2u * c->lay_every;
    c->lay_every = (force || !met || c->lay_every < kBatchRelayoutMin) ? kBatchRelayoutMin
                   : twice < kBatchRelayoutMax                          ? twice
                                                                        : kBatchRelayoutMax;
    const uint32_t wait = 2u * c->lay_wait < kBatchRelayoutMax ? 2u * c->lay_wait : kBatchRelayoutMax;
    c->lay_wait = force ? 0u : (paid || c->lay_wait < 16u) ? 16u : wait;
    c->lay_work = c->pfx_total + c->mov_total;
    c->lay_since = 0;
  }
  if (build) {
    c->lay_forced = force;
    c->lay_segs = force ? 0u : c->lay_segs < 2u ? c->lay_segs + 1u : 2u;
  }
  c->gsop_same[0] = c->gsop_same[1] = 0;
  c->lit_seen = c->ctr[6];
  c->dec_ticks = ticks;
  c->lay_since += ticks;
  c->lay_now = build ? 1u : 0u;
}

#ifdef __CUDACC__
// The decision on the device, by one block before the batch (lit: the always-lit
// axons of the last ticks, a bit each, of A).
__device__ __forceinline__ void layout_decide(ShardCtl* c, uint32_t force, uint32_t ticks, const uint32_t* lit,
                                              uint32_t A, bool index) {
  __shared__ uint32_t s_lit;
  uint32_t n = 0;
  if (threadIdx.x == 0) s_lit = 0;
  __syncthreads();
  if (force || !layout_met(c)) {
    for (uint32_t i = threadIdx.x; i < (A + 31) / 32; i += blockDim.x) n += __popc(lit[i]);
    n = __reduce_add_sync(0xFFFFFFFFu, n);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&s_lit, n);
  }
  __syncthreads();
  if (threadIdx.x == 0) layout_decision(c, force, ticks, s_lit, index);
}
#endif

constexpr uint32_t kFixCap = 1u << 22;  // deferred GSOP slots per tick before the rescan path
constexpr uint32_t kMaxUpdateWarps = 32u * 1024u;  // warps of the update pass (32 per SM)

// Row engine (row_engine.cuh, compiled in day_phase.cu).  A (re)allocation
// drops the batch engine's captured graphs, which hold the old addresses; the
// new buffers are zeroed on `stream` (the legacy stream: zeroed before return).
cudaError_t rows_alloc(ShardScratch& s, uint32_t N, uint32_t A, bool with_fix, cudaStream_t stream);
void rows_free(ShardScratch& s);
// Allocates the row copy's position map (row position of every columnar slot),
// written by every later row copy of the shard that asks for it.
cudaError_t rows_posmap(ShardScratch& s, cudaStream_t stream);
// row_sum: also compute the targets checksum (ShardCtl::row_sum) the learned engine checks its index against;
// with_posmap: also write the position map (when it is allocated); conditional: the layout kernels lay
// the rows out only when the device's decision (ShardCtl::lay_now, layout_decide) says so, and
// otherwise keep the copy (only the per-tick lists are reset).
cudaError_t launch_rows_begin(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, cudaStream_t stream,
                              bool row_sum = false, bool permute = true, bool with_posmap = true,
                              bool conditional = false);
// The device's layout decision outside a batch's control kernel (per-tick calls).
cudaError_t launch_rows_decide(ShardScratch& s, uint32_t A, bool force, uint32_t ticks, cudaStream_t stream);
cudaError_t launch_rows_end(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, cudaStream_t stream);

// Before a learned chunk of a shard with rows, on its stream: when the device
// asked for an inverted index, lays the rows out if the device's decision says
// so (as the chunk's own conditional layout would) and builds the index; else
// nothing.
cudaError_t rows_index_wish(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, cudaStream_t stream,
                            bool row_sum, bool with_posmap);
// The pinned word the device asks through.
cudaError_t rows_wish_alloc(ShardScratch& s);

// Tries of the update pass's first wait for its staged bitmap; returns the previous value.
uint32_t set_first_wait_limit(uint32_t tries);
// Tries of the barriers of k_rows_small's resident grid; returns the previous value.
uint32_t set_barrier_limit(uint32_t tries);

// Registry keyed by the axon_heads pointer.  Created by cu_allocate_shard;
// created lazily (and sized) for shards whose memory the caller allocated.
ShardScratch* scratch_for(const ShardVramPtrs* vram, uint32_t padded_n, uint32_t total_axons,
                          cudaError_t* err);
void scratch_release(const void* heads_key);
void graph_cache_free(ShardScratch* s);  // batch_engine.cu
void graph_cache_drop(ShardScratch* s);  // batch_engine.cu: destroys the captured graphs only
uint32_t fix_capacity();                 // batch_engine.cu: deferred-GSOP list capacity in use

// The row caches of a shard (per-tick and batch) no longer match its memory (shard_api.cu).
inline void rows_touched(ShardScratch& s) {
  s.tick_rows_valid.store(false);
  s.batch_rows_valid.store(false);
}
// A batch or run that returned an error may not have made the layout that it was to
// make (batch_rows_force counts it as made): the next one makes it.
inline void batch_undone(ShardScratch* s) {
  if (s) rows_touched(*s);
}
// Marks every shard whose .state allocation overlaps [dst, dst + size).
void invalidate_overlapping(const void* dst, size_t size);
// Looks up a shard's scratch without creating it (nullptr if none).
ShardScratch* scratch_find(const ShardVramPtrs* vram);

// Tick stages (day_phase.cu).  When dctl_batch is true the tick number,
// dopamine and network spike count come from the shard's device control
// block (tick = ctl->tick_base + k, count = batch_counts[k]).
struct TickArgs {
  uint32_t padded_n, total_axons, v_seg, tick;
  const uint32_t* input_bitmask;
  uint32_t virtual_offset, num_virtual;
  const uint32_t* incoming_spikes;
  uint32_t num_incoming;      // per-tick mode
  uint32_t max_incoming;      // batch mode: capacity of the tick's schedule row
  const uint32_t* mapped_soma_ids;
  uint8_t* output_history;
  uint32_t num_outputs;
  int16_t dopamine;
  bool batch;                 // read tick/dopamine/count from the device control block
  uint32_t k;                 // tick index inside the batch
  bool rows;                  // use the neuron-major row engine (batch mode only)
  uint32_t fix_cap;           // row engine: deferred-GSOP list capacity (<= kFixCap)
  bool lit_new;               // row engine: the window of always-lit axons (RowCache::alit) starts at this tick
  bool shared_gpu;            // row engine: other shards' ticks run beside this one's
  bool index;                 // row engine: count active axons, for the sparse form (the learned engine's plain graph)
  bool sparse;                // row engine: and launch its kernels
  bool defer_push;            // row engine: leave this tick's soma pushes to the next tick's prologue
                              // (never on the last tick of a batch)
};

// ev (optional): 6 events recorded around the stages (incoming, axons,
// update, push, gsop) for per-kernel timing.
constexpr int kTickStages = 5;
cudaError_t launch_tick(const ShardVramPtrs& v, ShardScratch& s, const TickArgs& a, cudaStream_t stream,
                        cudaEvent_t* ev = nullptr);
// Small brains: `ticks` ticks from a (its arrays those of the first; words of the
// input per tick) in one launch, where rows_small says so.
bool rows_small(uint32_t N, uint32_t A, bool whole_gpu, bool batch);
// Its cluster or resident grid does not fit after all (a context that may not use
// every SM): the kernel chain runs the ticks.
inline bool launch_refused(cudaError_t e) {
  return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorInvalidClusterSize ||
         e == cudaErrorLaunchOutOfResources || e == cudaErrorInvalidConfiguration || e == cudaErrorNotSupported;
}
cudaError_t launch_rows_small(const ShardVramPtrs& v, ShardScratch& s, const TickArgs& a, uint32_t ticks,
                              uint32_t words, cudaStream_t stream);
cudaError_t launch_reset_burst(const ShardVramPtrs& v, uint32_t padded_n, cudaStream_t stream);

// One shard's batch: the arguments of axc_step_day_phase_batch (batch_engine.cu).
struct BatchArgs {
  const ShardVramPtrs* vram;
  uint32_t padded_n, total_axons, ticks;
  const AxcIoBuffers* io;
  const uint32_t *h_bm, *h_in, *h_counts;
  uint32_t voff, nv;
  const uint32_t* ids;
  uint32_t v_seg;
  int16_t dopamine;
  uint32_t tick_base;
};
cudaError_t batch_prepare(const BatchArgs& b, ShardScratch** out_s, uint32_t* out_rows, cudaStream_t stream);
// whole_gpu: the batch may hold every SM (no other shard's branch runs beside it).
// one_launch: a small brain's ticks may run in one launch; a capture that is refused
// with it (launch_refused) is made again without.
cudaError_t batch_capture(const BatchArgs& b, ShardScratch& s, uint32_t rows, uint32_t fix_cap, cudaStream_t cap,
                          bool whole_gpu, bool one_launch);
// dst[dst_indices[i]] = src[src_indices[i]] for src_indices[i] < 2^31 (side_kernels.cu, bindings.cu:341-368).
cudaError_t ghost_sync(const BurstHeads8* src_heads, BurstHeads8* dst_heads, const uint32_t* src_indices,
                       const uint32_t* dst_indices, uint32_t count, cudaStream_t stream);
cudaError_t launch_spike_list_sorted(const ShardVramPtrs& v, uint32_t padded_n, uint32_t* out_ids,
                                     uint32_t* out_count, cudaStream_t stream);

// Stand-alone stages for the legacy per-kernel launchers (ffi.rs:193-233).
cudaError_t launch_push_incoming(BurstHeads8* heads, ShardScratch& s, uint32_t A, const uint32_t* ids,
                                 uint32_t count, cudaStream_t stream);
cudaError_t launch_propagate_only(BurstHeads8* heads, uint32_t A, uint32_t v_seg, cudaStream_t stream);
cudaError_t launch_update_stage(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, uint32_t tick,
                                cudaStream_t stream);
cudaError_t launch_gsop_stage(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, int16_t dopamine,
                              cudaStream_t stream);

// LUT access for host code (day_phase.cu owns the __constant__ symbol).  Every
// upload advances the LUT generation.
cudaError_t lut_upload(const VariantParameters* lut, cudaStream_t stream, bool async);
uint64_t lut_generation();

int current_device();
int sm_count();   // of the current device

}  // namespace axc
