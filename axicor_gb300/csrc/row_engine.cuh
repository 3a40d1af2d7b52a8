// row_engine.cuh — the batch engine's neuron-major tick (compiled as part of
// day_phase.cu: it uses that translation unit's __constant__ LUT and helpers).
//
// Why: in the reference layout dendrite slot i of all neurons is one row
// ([slot][neuron], memory.rs:71-86), so a 32-byte sector holds 8 neurons'
// targets.  In steady state only the non-refractory quarter of the neurons is
// evaluated each tick, yet nearly every sector is fetched, and GSOP re-reads
// the spikers' slots with one sector per slot.  For the length of one batch the
// engine keeps a neuron-major copy ([neuron][128]) of targets and weights:
//
//   layout       k_rows_mult       owners of each axon (none, one, several)
//                k_rows_build      columnar -> rows in groups by what a tick has to
//                                  test and GSOP may move (build_row)
//   per tick     k_rows_prologue_plain  the previous tick's soma pushes, axon
//                                  pushes + propagation + split masks, fully-lit
//                                  bitmap, refractory countdown, list of
//                                  evaluated neurons
//                k_rows_update     8 lanes per evaluated neuron: gather/sum, GLIF,
//                                  GSOP of the movable slots
//                k_rows_update_lsum  the same, a thread per neuron, on ticks that
//                                  test few slots (tick_form)
//                k_sparse_*        the same from an inverted index, on the learned
//                                  engine's quiet ticks
//                k_rows_fixup      readout, the GSOP slots whose result depends on
//                                  same-tick pushes
//                k_rows_push       the spikers' pushes (a batch's last tick only;
//                                  otherwise the next prologue applies them)
//   small brains k_rows_small      all of that for a batch's ticks in one launch
//   batch end    k_rows_writeback  weights rows -> columnar
//
// GSOP against same-tick pushes.  GSOP must see the heads after this tick's
// soma pushes (physics.cu:281-373 runs after the update kernel).  A push
// inserts a 0 head and drops h7, so for an axon owned by one soma the result
// can only change when segment 0 is involved or h7 is the only head in the
// tail.  The axon stage writes two masks per axon — hits of heads 0..6 and
// hits of head 7 — so GSOP knows, per slot, the "no push" and "one push"
// outcomes.  When they agree the weight is updated at once; otherwise the slot
// is left untouched and listed, and k_rows_fixup applies it with the actual
// push count (and from the original weight).  Axons owned by two or more
// somas, variants whose length differs from the LUT maximum or exceeds 16
// (where the cooling shift can be non-zero) and segments >= 31 take the exact
// general path.

namespace axc {
namespace {

constexpr uint32_t kRowStride = AXC_MAX_DENDRITES;   // slots per neuron row
constexpr uint32_t kInf = 0xFFFFFFFFu;

// Programmatic dependent launch inside a tick's kernel chain (prologue ->
// 8-lane pass -> lit-sum pass -> fix-up -> push).  A kernel
// launched with launch_chain(pdl = true) may be scheduled while the kernel
// before it on the stream still runs; its first statement is chain_wait(),
// which returns once that kernel has completed and its writes are visible, so
// only the launch and the block scheduling overlap.  Every block passes
// chain_wait() before it can exit, so a kernel's completion implies its
// predecessor's, and the chain stays ordered end to end.  chain_open() then
// lets the next kernel of the chain be scheduled (after this grid's last block
// started and passed its own wait); it only matters when that kernel is
// launched with the attribute.  In a kernel launched without it (the prologue,
// every kernel of a captured batch) chain_wait() returns at once: the stream
// finished the predecessor before the kernel started.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_open() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... Args>
static void launch_chain(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool pdl,
                         Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  // a failed launch also leaves its error for cudaGetLastError, which the
  // launch sequences return
  cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}
// Axon word axw[a], set by the layout: a soma owns the axon; two or more do; bits
// 1..30: a used slot of the shard targets that segment of it.  The axon is fully
// lit when heads 0..6 cover those segments (not every segment that some axon
// uses: after two pushes close together the eight heads reach less far, but few
// axons have slots on their last segments).
constexpr uint32_t kAxOwned = 1u, kAxShared = 0x80000000u, kAxSegs = 0x7FFFFFFEu;
// Segments 1..used_segs count as used on every axon, so that a layout asks for the
// words of the targets beyond them only (a third of the benchmark's slots are past 7,
// one in 16 past 12; asking for all of them was 450 us of a layout of 1.5M neurons).
// Seven heads one tick apart reach segment 7, two ticks apart 13: an axon lit on its
// own segments at every tick is lit on those too.  A forced layout takes the larger
// number: it is the one that a write, a LUT or a change of path makes a program wait
// for, and the next layout, if it pays, marks the rest.  The layouts after that keep
// the marks: the targets are the same until something forces a layout (keep_segs).
constexpr uint32_t kUsedSegs = 7, kUsedSegsForced = 12;
__device__ __forceinline__ uint32_t used_segs(const ShardCtl* ctl, uint32_t cond) {
  return cond && !ctl->lay_forced ? kUsedSegs : kUsedSegsForced;
}
__device__ __forceinline__ bool keep_segs(const ShardCtl* ctl, uint32_t cond) { return cond && ctl->lay_segs == 2u; }
__device__ __forceinline__ uint32_t ax_owners(uint32_t axw) { return (axw & kAxOwned) + (axw >> 31); }
constexpr uint32_t kRowBad = 0x8000u;    // cnt flag: the row holds an invalid target
constexpr uint32_t kRowSplit = 0x4000u;  // cnt flag: its movable slots are in two groups (build_row), not in slot order

// Bytes of the fully-lit bitmap of A axons as staged in shared memory (one
// bit per axon and a spare word, rounded up to the bulk copy's 16 bytes; the
// global bitmap is allocated at least this large).
__host__ __device__ __forceinline__ uint32_t lit_smem_bytes(uint32_t A) { return (((A >> 5) + 1) * 4 + 15) & ~15u; }

// physics.cu:322-371 for one slot given the minimum in-tail distance md.
__device__ __forceinline__ int16_t gsop_weight(int16_t w16, uint32_t md, const VariantParameters& p, int32_t bm,
                                               int32_t raw_pot, int32_t final_dep) {
  const bool active = md != kInf;
  const int32_t sign = w16 >= 0 ? 1 : -1;
  int32_t abs_w = (int32_t)w16;
  if (abs_w < 0) abs_w = -abs_w;
  uint32_t rank = (uint32_t)abs_w >> 11;
  if (rank > 15) rank = 15;
  const int32_t inertia = p.inertia_curve[rank];
  const int32_t delta_pot = wmul(wmul(raw_pot, inertia), bm) >> 7;
  const int32_t delta_dep = wmul(wmul(final_dep, inertia), bm) >> 7;
  const uint32_t cs = active ? (md >> 4) : 0u;
  int32_t delta = active ? (delta_pot >> cs) : wsub(0, delta_dep);
  delta = wmul(delta, 128) >> (7u + cs);
  int32_t new_abs = wadd(abs_w, delta);
  new_abs = new_abs & ~(new_abs >> 31);
  if (new_abs > 32767) new_abs = 32767;
  return (int16_t)wmul(new_abs, sign);
}

__device__ __forceinline__ uint32_t md_of(const uint32_t h[8], uint32_t s, uint32_t len) {
  uint32_t md = kInf;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const uint32_t d = h[q] - s;
    md = min(md, d < len ? d : kInf);
  }
  return md;
}

// Minimum distances with no push and with one push (0, h0..h6).
__device__ __forceinline__ void md_pair(const BurstHeads8* heads, uint32_t a, uint32_t s, uint32_t len,
                                        uint32_t* md0, uint32_t* md1) {
  uint32_t h[8];
  load_heads(heads, a, h);
  uint32_t m06 = kInf;
#pragma unroll
  for (int q = 0; q < 7; q++) {
    const uint32_t d = h[q] - s;
    m06 = min(m06, d < len ? d : kInf);
  }
  const uint32_t d7 = h[7] - s;
  *md0 = min(m06, d7 < len ? d7 : kInf);
  const uint32_t dz = 0u - s;
  *md1 = min(m06, dz < len ? dz : kInf);
}

// Write-through of GSOP's weight changes to the reference's columnar blob
// (dendrite_weights[slot][N]), used by the per-tick entry point, whose row
// cache outlives the call: after every tick the blob must hold the weights the
// reference would hold.  w == nullptr: no write-through (the batch paths write
// every weight back at batch end).
struct ColWT {
  int16_t* w = nullptr;         // columnar weights of the shard
  const uint4* om = nullptr;    // per neuron: the columnar slots placed first in its row,
  const uint4* lm = nullptr;    // and those of them placed before the others
  uint32_t N = 0;
};

// The r-th set bit (0-based, r < popc) of a word: a binary search over the counts
// (__fns walks the bits: 15 of the 37 us of a plastic per-tick call at 6,000 neurons).
__device__ __forceinline__ uint32_t nth_bit32(uint32_t m, uint32_t r) {
  uint32_t pos = 0;
#pragma unroll
  for (uint32_t st = 16; st > 0; st >>= 1) {
    const uint32_t c = __popc(m & ((1u << st) - 1u));
    if (r >= c) {
      r -= c;
      pos += st;
      m >>= st;
    }
  }
  return pos;
}

// The r-th set bit (0-based) of a 128-bit mask.
__device__ __forceinline__ uint32_t nth_bit128(uint4 m, uint32_t r) {
  uint32_t w = m.x, base = 0;
  uint32_t c = __popc(w);
  if (r >= c) { r -= c; w = m.y; base = 32; c = __popc(w); }
  if (base == 32u && r >= c) { r -= c; w = m.z; base = 64; c = __popc(w); }
  if (base == 64u && r >= c) { r -= c; w = m.w; base = 96; }
  return base + nth_bit32(w, r);
}

// Columnar slot of row position pos < lf, in a row whose movable slots are om,
// those of lm first and then the others, each in slot order.
__device__ __forceinline__ uint32_t col_of_pos(uint4 om, uint4 lm, uint32_t pos) {
  const uint32_t nl = __popc(lm.x) + __popc(lm.y) + __popc(lm.z) + __popc(lm.w);
  return pos < nl ? nth_bit128(lm, pos)
                  : nth_bit128(make_uint4(om.x & ~lm.x, om.y & ~lm.y, om.z & ~lm.z, om.w & ~lm.w), pos - nl);
}

__device__ __forceinline__ void col_write(const ColWT& wt, uint32_t n, uint32_t pos, int16_t w) {
  const uint32_t q = col_of_pos(wt.om[n], wt.lm[n], pos);
  wt.w[(size_t)q * wt.N + n] = w;
}

// The columnar slots of consecutive row positions: the first by search, each further
// one the mask's next bit.
struct ColRun {
  uint4 m;
  uint32_t cur, base, left;   // the word's bits not yet passed, its first slot, positions before the other mask

  __device__ __forceinline__ uint32_t word() const {
    return base == 0u ? m.x : base == 32u ? m.y : base == 64u ? m.z : m.w;
  }
  __device__ __forceinline__ void others(const ColWT& wt, uint32_t n) {
    const uint4 om = wt.om[n], lm = wt.lm[n];
    m = make_uint4(om.x & ~lm.x, om.y & ~lm.y, om.z & ~lm.z, om.w & ~lm.w);
    left = kRowStride;
  }
  __device__ __forceinline__ ColRun(const ColWT& wt, uint32_t n, uint32_t pos) {
    m = wt.lm[n];
    const uint32_t nl = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
    uint32_t r = pos;
    if (pos < nl) {
      left = nl - pos;
    } else {
      r = pos - nl;
      others(wt, n);
    }
    base = nth_bit128(m, r);
    const uint32_t bit = base & 31u;
    base -= bit;
    cur = word() & (~0u << bit);
  }
  __device__ __forceinline__ uint32_t next(const ColWT& wt, uint32_t n) {
    if (left-- == 0u) {
      others(wt, n);
      left--;
      base = 0;
      cur = m.x;
    }
    while (cur == 0u && base < 96u) {
      base += 32u;
      cur = word();
    }
    const uint32_t q = base + __ffs(cur) - 1u;
    cur &= cur - 1u;
    return q;
  }
};

// The lit-sum form runs tick k when the rows' tested slots are few (at most
// an eighth of the live slots: otherwise the 8-lane pass is faster) and every
// axon the row layout took as fully lit is fully lit this tick; with a few of
// them dark (a network spike on an axon that its soma keeps lit moves its
// oldest heads on) the rows are checked slot by slot (kFormVerify), with many, or in
// rows of up to 32 slots, by the dense pass (504,000 plastic neurons, 32 slots: 31.7 us
// a tick against 36.8 checked; tick_form has the other sizes).  Every thread
// of both update kernels asks at its start; the words were written by
// earlier kernels and no kernel that asks writes them, so cached loads (in
// L1 after the first warp of an SM) serve it: uncached loads sent every
// warp's request to the one L2 slice that holds the control block, a few
// microseconds per launch.
__device__ __forceinline__ bool lit_layout(unsigned long long tested, unsigned long long slots) {
  return slots > 0 && tested * 8ull <= slots;
}

// The sparse form can run tick k: fewer than half as many axons have a head on
// a segment of the batch as neurons are evaluated.  The dense pass tests every
// slot of the evaluated neurons (~4.5 ns a thousand slots at 1.5M neurons), the
// sparse form walks the hit segments' entries of the active axons.  The two
// words were written by the prologue.
__device__ __forceinline__ bool sparse_tick(uint32_t eval, uint32_t active) { return active * 2u < eval; }

// The inverted index matches the rows: it was built, from a layout with the
// same targets at the same row positions (0: a layout without the checksum).
__device__ __forceinline__ bool index_built(const ShardCtl* ctl) {
  return ctl->idx_ok && ctl->lay_sum != 0ull && ctl->idx_sum == ctl->lay_sum;
}
// And this graph can use it.
__device__ __forceinline__ bool index_ok(const ShardCtl* ctl) { return ctl->ix_run && index_built(ctl); }

// Per-neuron GSOP constants (physics.cu:290-345).
struct GsopConsts {
  int32_t bm, raw_pot, final_dep;
};

__device__ __forceinline__ GsopConsts gsop_consts(uint8_t flags, const VariantParameters& p, int32_t dopamine) {
  GsopConsts g;
  const uint32_t burst = (flags >> 1) & 0x07;
  g.bm = burst > 0 ? (int32_t)burst : 1;
  const int32_t pot_mod = wmul(dopamine, (int32_t)p.d1_affinity) >> 7;
  const int32_t dep_mod = wmul(dopamine, (int32_t)p.d2_affinity) >> 7;
  g.raw_pot = wadd((int32_t)p.gsop_potentiation, pot_mod);
  const int32_t raw_dep = wsub((int32_t)p.gsop_depression, dep_mod);
  g.final_dep = raw_dep & ~(raw_dep >> 31);
  return g;
}

// Split segment-hit masks of one axon's (propagated) heads for length P:
// x: bits 0..30 = segments hit by heads 0..6, bit 31 = some head (0..7) may hit
//    a segment >= 31;  y: bits 0..30 = segments hit by head 7, bit 31 = the axon
//    is owned by two or more somas.  An axon owned by no soma cannot be pushed
//    between update and GSOP, so its head-7 hits are folded into x.
__device__ __forceinline__ uint2 split_masks(const uint32_t h[8], uint32_t P, uint32_t mult) {
  uint32_t x = 0, y = 0;
  if (P != 0) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const uint32_t v = h[k];
      if (v < 255u + P) {
        const uint32_t lo = (v + 1u > P) ? v + 1u - P : 0u;
        uint32_t bits = 0;
        if (lo <= 30u) {
          const uint32_t top = min(v, 30u);
          bits = ((2u << top) - 1u) & ~((1u << lo) - 1u);
        }
        if (k < 7) x |= bits; else y |= bits;
        if (v >= 31u) x |= 0x80000000u;
      }
    }
  }
  if (mult == 0) { x |= y; y = 0; }
  if (mult >= 2) y |= 0x80000000u;
  return make_uint2(x, y);
}

// True when the update pass may apply GSOP to this slot on the spot.
// fast: hit/no-hit decides (variant length == LUT max <= 16, segment < 31,
// axon not multiply owned) and the one-push outcome equals the no-push one.
__device__ __forceinline__ bool fast_class(uint32_t s, uint2 m, bool gsop_fast) {
  return gsop_fast && s < 31u && !(m.y >> 31);
}

__device__ __forceinline__ bool fast_sensitive(uint32_t s, uint2 m) {
  const bool a0 = ((m.x | m.y) >> s) & 1u;
  const bool a1 = (s == 0u) || ((m.x >> s) & 1u);
  return a0 != a1;
}

// Control block and per-tick buffers of the learned-schedule engine
// (learned.cuh): the prologue accumulates per-tile activity into them and, on
// a sparse tick, compacts the active axons into per-tile segments whose sizes
// the predictor chose before the tick.
struct LearnCtl {
  uint32_t mode;          // this tick: 0 dense row pass, 1 sparse axon-driven gather
  uint32_t overflow;      // a tile outgrew its pre-sized segment: the tick runs dense
  uint32_t spk_count;     // sparse tick: spikers listed for GSOP
  uint32_t stale;         // the inverted index no longer matches the targets
  uint32_t ticks_seen;    // ticks completed with features since the history began
  uint32_t samples;       // (features, target) pairs recorded
  uint32_t sample_cap;
  uint32_t sample_every;  // record every k-th tick
  int32_t policy;         // -1 predictor, 0 always dense, 1 always sparse (exact capacities)
  uint32_t collect;       // record pairs while running
  float ratio;            // sparse when ratio * predicted active synapses < evaluated slots
  float margin;           // capacity = prediction * (1 + margin) + slack
  uint32_t slack;
  uint32_t T;             // tiles of 1024 axons (= neurons)
  uint32_t prev_mode;     // the previous tick's schedule
  uint32_t prev_learned;  // the previous tick's schedule came from the predictor
  uint32_t feat_done;     // the features kernel ran after the previous tick
  uint32_t pad0, pad1, pad2, pad3;
  unsigned long long eval_next;   // evaluated slots of the next tick (features kernel)
  unsigned long long eval_now;    // evaluated slots of this tick
  unsigned long long row_sum;     // targets checksum the inverted index was built from
  float pred_total;               // sum of the tile predictions for this tick (synapses)
  float inrate[9];                // input spike fraction of ticks t, t-1, ..., t-8
  unsigned long long stat[12];
};

struct LearnDev {
  LearnCtl* ctl;
  const uint32_t* inv_off;  // [A+1] inverted index offsets (slots whose target is axon a)
  uint32_t* yacc;           // [T] active synapses of the tile's axons this tick
  uint32_t* bacc;           // [T] heads in flight on the tile's axons this tick
  uint32_t* fill;           // [T] axons compacted into the tile's segment
  const uint32_t* cap;      // [T] the tile's capacity in synapses
  uint32_t* alist;          // active axons of a sparse tick, tile j at [1024 j, 1024 j + fill[j])
  uint32_t* evbits;         // [N/32+1] evaluated neurons of the tick
};

// The form of tick k, the same for every kernel that asks after the prologue.
// lc: the learned engine's control block (its planned sparse ticks), or null;
// index: the tick may run sparse by the exact counts (the learned engine's
// graphs, whose memory holds the inverted index).
// The kernels that run a tick count it by its form (ShardCtl::forms).
enum TickForm {
  kFormDense = 0,     // k_rows_update: every slot tested
  kFormLitSum = 1,    // k_rows_update_lsum: a thread per neuron
  kFormSparse = 2,    // k_sparse_hits, k_sparse_neurons
  kFormScatter = 3,   // the learned engine's kernels without the rows' index
  kFormLitRows = 4,   // k_rows_update: lit_row_step
  kFormVerify = 5     // the same, with dark axons: each lit slot is looked up
};
constexpr int kCountSmall = 6, kCountLayout = 7;   // forms[]: ticks inside k_rows_small; layouts of the rows

// One thread of a tick's kernel.
__device__ __forceinline__ void count_form(ShardCtl* ctl, int form) { atomicAdd(&ctl->forms[form], 1ull); }

// The control words are read at once (volatile, so that no load waits behind the
// branch on another) through L1, as lit_layout's comment says.
__device__ __forceinline__ unsigned long long ctl_ld64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ctl_ld32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// kFormLitRows where more than a sixteenth of the live slots are movable or
// tested: a settled brain has 0.5 % of them so, one that learns all its life
// nearly all.  kFormVerify while so few axons are dark that less than one row in
// kDarkRows has a slot on one: such a row is tested a second time and holds up its
// warp's other three.  A tick of 504,000 plastic neurons with 64 network spikes: 32.6
// us checked and 37.8 dense at 33 slots a row, 39.0 and 42.2 at 64, 53.6 and 53.4 at
// 96, 64.5 and 62.0 at 128; of 61,000 at 100 slots, with the same spikes, 26.4 and 21.1;
// with a hundredth of the axons dark 1.5M settled neurons took 240 checked, 163 dense.
constexpr uint32_t kDarkRows = 128;
__device__ __forceinline__ TickForm tick_form(const ShardCtl* ctl, uint32_t k, uint32_t A, const LearnCtl* lc,
                                              uint32_t index) {
  const unsigned long long p = ctl_ld64(&ctl->pfx_total), c = ctl_ld64(&ctl->slot_total), m = ctl_ld64(&ctl->mov_total);
  const uint32_t dark = ctl_ld32(&ctl->dense[k & 1]), smax = ctl_ld32(&ctl->row_smax);
  if (lc && lc->mode == 1u && !lc->overflow) return index_ok(ctl) ? kFormSparse : kFormScatter;
  if (lit_layout(p, c)) {
    if (!dark) return (m + p) * 16ull > c ? kFormLitRows : kFormLitSum;
    return smax > 32u && (unsigned long long)dark * smax * kDarkRows <= A ? kFormVerify : kFormDense;
  }
  return index && index_ok(ctl) && sparse_tick(ctl->eval_act[k & 1][0], ctl->eval_act[k & 1][1]) ? kFormSparse : kFormDense;
}

// 64-bit mix of one live slot for the targets checksum (order-independent sum).
__device__ __forceinline__ unsigned long long slot_mix(uint32_t t, uint32_t r) {
  unsigned long long x = ((unsigned long long)t << 32) ^ (unsigned long long)r;
  x *= 0x9E3779B97F4A7C15ull;
  x ^= x >> 31;
  x *= 0xBF58476D1CE4E5B9ull;
  return x ^ (x >> 29);
}

// ---------------------------------------------------------------------------
// batch start / end: the row copy
// ---------------------------------------------------------------------------
// Smallest |w| from which every inertia rank of variant v is 0 (0x10000:
// none): GSOP moves such a weight by 0 whatever the hit, distance, burst or
// dopamine (physics.cu:336-371), except -32768, which the clamp turns into
// -32767.
__device__ __forceinline__ int32_t frozen_from(const VariantParameters& p) {
  int r0 = 16;
  while (r0 > 0 && p.inertia_curve[r0 - 1] == 0) r0--;
  return r0 < 16 ? r0 * 2048 : 0x10000;
}

// thr <= |w| <= 32767, in plain signed comparisons (-32768 is not frozen: the
// clamp moves it).
__device__ __forceinline__ bool frozen_weight(int16_t w16, int32_t thr) {
  const int32_t w = w16;
  return w != -32768 && (w >= thr || w <= -thr);
}

// Row position of columnar slot q (lane = q & 31) when the slots of mask o
// come first, in slot order, and the others follow in slot order: word = the
// 32 bits of o holding q, pre = set bits of o before that word, lf = set bits
// of o in all.
__device__ __forceinline__ uint32_t row_pos(uint32_t word, uint32_t lane, uint32_t q, uint32_t pre, uint32_t lf) {
  const uint32_t below = pre + __popc(word & ((1u << lane) - 1u));
  return ((word >> lane) & 1u) ? below : lf + q - below;
}

// One neuron's row of the row copy, by one warp, from the staged columns (column
// j, c used slots): placement, and the neuron's cnt / amask / omask / lfz.
// A slot is movable when GSOP may still move its weight, and lit (stage_columns)
// when it has a segment in 1..30, belongs to a neuron whose variant
// length is the LUT maximum, and targets an axon that xlit marks as fully lit:
// while that axon stays fully lit (the prologue checks it every tick) the slot
// is a hit, and GSOP takes its delta from the rank table (movable slots only
// with mov_lit).  With permute the row
// holds, each group in slot order,
//   [0, lm)    movable, lit: hits, their weights read each tick
//   [lm, lf)   movable, not lit: tested each tick
//   [lf, end)  frozen, not lit: tested each tick
//   [end, c)   frozen, lit: hits whose weights are summed once (rec[n].x)
// and rec[n].y = lm | lf << 8 | end << 16; lmask marks the columnar slots of the
// first group.  Without permute every slot keeps its position.
// Returns, in every lane, the row's largest segment, (want_sum) its targets
// checksums by columnar slot and by row position, and its tested slots.
struct RowBuilt {
  uint32_t smx;
  unsigned long long hsum;
  uint32_t pfx;
  uint32_t lf;
  unsigned long long psum;
};

__device__ __forceinline__ uint32_t popc4(const uint32_t (&m)[4]) {
  return __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
}

// 32 neurons' columns staged in shared memory, with a class byte a slot.
struct SlotStage {
  uint32_t t[AXC_MAX_DENDRITES][33];
  int16_t w[AXC_MAX_DENDRITES][34];
  uint8_t k[AXC_MAX_DENDRITES][36];   // kSlotMov | kSlotLit | kSlotBad
  uint32_t cnt[32];                   // used slots of the neurons
  int32_t fz[32];                     // frozen_from of their variants
  uint32_t lit[32];                   // their lit slots may be taken as such
};
constexpr uint32_t kSlotMov = 1u, kSlotLit = 2u, kSlotBad = 4u;

// Columns -> stage, by a 256-thread block that has set cnt (AXC_MAX_DENDRITES),
// fz and lit: 32 slots of the 32 neurons a round, until every neuron has met its
// first empty target.  A thread has four targets and weights of the next round in
// flight while it looks up the four of this one (xlit: the lit axons; axw: marks
// the axon's segment as used, beyond the first `used`), so a round costs the latency
// of one gather.
__device__ __forceinline__ void stage_columns(SlotStage& st, const uint32_t* __restrict__ targets,
                                              const int16_t* __restrict__ weights, uint32_t N, uint32_t n0, uint32_t A,
                                              const uint32_t* __restrict__ xlit, bool mov_lit, uint32_t* axw,
                                              uint32_t used) {
  const uint32_t col = threadIdx.x & 31, r0 = threadIdx.x >> 5, n = n0 + col;
  const int32_t fz = st.fz[col];
  const bool lit_on = xlit && st.lit[col];
  uint32_t t[4];
  int16_t w[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const size_t at = (size_t)(8 * i + r0) * N + n;
    t[i] = n < N ? __ldcs(targets + at) : 0u;
    w[i] = n < N ? __ldcs(weights + at) : (int16_t)0;
  }
#pragma unroll 1
  for (uint32_t ch = 0; ch < AXC_MAX_DENDRITES / 32; ch++) {
    uint32_t tn[4] = {0, 0, 0, 0};
    int16_t wn[4] = {0, 0, 0, 0};
    if (ch + 1 < AXC_MAX_DENDRITES / 32 && n < N) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const size_t at = (size_t)((ch + 1) * 32 + 8 * i + r0) * N + n;
        tn[i] = __ldcs(targets + at);
        wn[i] = __ldcs(weights + at);
      }
    }
    uint32_t lw[4], aw[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t a = (t[i] & AXC_TARGET_AXON_MASK) - 1u, seg = t[i] >> AXC_TARGET_SEG_SHIFT;
      const bool in = a < A && seg - 1u < 30u;
      lw[i] = in && lit_on ? __ldg(xlit + (a >> 5)) : 0u;
      aw[i] = in && axw && seg > used ? axw[a] : 0xFFFFFFFFu;   // (a stale word only costs an atomic that changes nothing)
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t r = ch * 32 + 8 * i + r0;
      const uint32_t a = (t[i] & AXC_TARGET_AXON_MASK) - 1u, seg = t[i] >> AXC_TARGET_SEG_SHIFT;
      if (!((aw[i] >> (seg & 31u)) & 1u)) atomicOr(axw + a, 1u << seg);
      const bool mov = !frozen_weight(w[i], fz);
      const bool lit = ((lw[i] >> (a & 31u)) & 1u) && (mov_lit || !mov);
      // an invalid axon id (field 0 or >= A) points at the dummy mask entry A,
      // which sends the slot down the exact path (hit_exact / gsop_general skip it)
      const bool bad = a >= A;
      st.t[r][col] = bad && t[i] ? (t[i] & ~AXC_TARGET_AXON_MASK) | (A + 1u) : t[i];
      st.w[r][col] = w[i];
      st.k[r][col] = (uint8_t)((mov ? kSlotMov : 0u) | (lit ? kSlotLit : 0u) | (bad ? kSlotBad : 0u));
      if (t[i] == 0) atomicMin(&st.cnt[col], r);
      t[i] = tn[i];
      w[i] = wn[i];
    }
    __syncthreads();
    const int mine = threadIdx.x < 32 ? (st.cnt[threadIdx.x] < (ch + 1) * 32) : 1;
    if (__syncthreads_and(mine)) break;
  }
}

__device__ __forceinline__ RowBuilt build_row(const SlotStage& st, uint32_t j, uint32_t n, uint32_t c, bool want_sum,
                                              bool permute, uint32_t* __restrict__ rt, int16_t* __restrict__ rw,
                                              uint16_t* __restrict__ cnt, uint4* __restrict__ amask,
                                              uint4* __restrict__ omask, uint8_t* __restrict__ lfz,
                                              int2* __restrict__ rec = nullptr, uint4* __restrict__ lmask = nullptr,
                                              uint8_t* __restrict__ posmap = nullptr) {
  const uint32_t lane = threadIdx.x & 31;
  bool bad = false;
  uint32_t smx = 0, rsum = 0;
  unsigned long long hsum = 0, psum = 0;
  uint32_t t[4], mv[4], lt[4], all[4];   // movable / lit / used slots, by columnar position
  int16_t w[4];
#pragma unroll
  for (int ch = 0; ch < 4; ch++) {
    const uint32_t q = 32u * ch + lane;
    all[ch] = c >= 32u * ch + 32u ? kFull : c > 32u * ch ? (1u << (c - 32u * ch)) - 1u : 0u;
    uint32_t k = 0;
    t[ch] = 0;
    w[ch] = 0;
    if (q < c) {
      t[ch] = st.t[q][j];
      w[ch] = st.w[q][j];
      k = st.k[q][j];
      bad |= (k & kSlotBad) != 0u;
      smx = max(smx, t[ch] >> AXC_TARGET_SEG_SHIFT);
      if (want_sum) hsum += slot_mix(t[ch], n * kRowStride + q);
      if ((k & (kSlotLit | kSlotMov)) == kSlotLit) rsum += (uint32_t)(int32_t)w[ch];
    }
    mv[ch] = __ballot_sync(kFull, (k & kSlotMov) != 0u);
    lt[ch] = permute ? __ballot_sync(kFull, (k & kSlotLit) != 0u) : 0u;
  }
  bad = __any_sync(kFull, bad);
  smx = __reduce_max_sync(kFull, smx);
  rsum = __reduce_add_sync(kFull, rsum);
  if (want_sum) hsum = warp_sum(hsum);
  if (bad) {
#pragma unroll
    for (int ch = 0; ch < 4; ch++) { mv[ch] = all[ch]; lt[ch] = 0u; }
    rsum = 0;
  }
  uint32_t g0[4], g1[4], g2[4];   // the first three groups
#pragma unroll
  for (int ch = 0; ch < 4; ch++) {
    g0[ch] = mv[ch] & lt[ch];
    g1[ch] = mv[ch] & ~lt[ch];
    g2[ch] = all[ch] & ~mv[ch] & ~lt[ch];
  }
  const uint32_t lm = popc4(g0), lf = lm + popc4(g1), end = lf + popc4(g2);
  const uint32_t below = (1u << lane) - 1u, bit = 1u << lane;
  // one group holds the whole row (a plastic brain, a quiet one, a settled one):
  // every slot keeps its place
  const bool moved = permute && lm != c && !(lm == 0u && lf == c) && !(lf == 0u && (end == c || end == 0u));
  uint32_t p0 = 0, p1 = lm, p2 = lf, p3 = end, am[4];
#pragma unroll
  for (int ch = 0; ch < 4; ch++) {
    const uint32_t q = 32u * ch + lane;
    uint32_t pos = q;
    if (moved) {
      const uint32_t g3 = all[ch] & ~(g0[ch] | g1[ch] | g2[ch]);
      if (g0[ch] & bit) pos = p0 + __popc(g0[ch] & below);
      else if (g1[ch] & bit) pos = p1 + __popc(g1[ch] & below);
      else if (g2[ch] & bit) pos = p2 + __popc(g2[ch] & below);
      else pos = p3 + __popc(g3 & below);
      p0 += __popc(g0[ch]);
      p1 += __popc(g1[ch]);
      p2 += __popc(g2[ch]);
      p3 += __popc(g3);
    }
    if (q < c) {
      if (want_sum && moved) psum += slot_mix(t[ch], n * kRowStride + pos);
      rt[(size_t)n * kRowStride + pos] = t[ch];
      rw[(size_t)n * kRowStride + pos] = w[ch];
      if (posmap) posmap[(size_t)n * kRowStride + q] = (uint8_t)pos;
    }
    // the movable slots by row position: the first lf positions, or mv itself
    const uint32_t lo = 32u * ch;
    am[ch] = permute ? (lf >= lo + 32u ? kFull : (lf > lo ? (1u << (lf - lo)) - 1u : 0u)) : mv[ch];
  }
  if (lane == 0) {
    cnt[n] = (uint16_t)(c | (bad ? kRowBad : 0u) | (lm > 0u && lm < lf ? kRowSplit : 0u));
    amask[n] = make_uint4(am[0], am[1], am[2], am[3]);
    omask[n] = permute ? make_uint4(mv[0], mv[1], mv[2], mv[3]) : make_uint4(all[0], all[1], all[2], all[3]);
    if (lmask) lmask[n] = permute ? make_uint4(g0[0], g0[1], g0[2], g0[3]) : make_uint4(all[0], all[1], all[2], all[3]);
    lfz[n] = (uint8_t)lf;
    if (rec) rec[n] = make_int2((int32_t)rsum, (int32_t)(lm | (lf << 8) | (end << 16)));
  }
  if (want_sum) psum = moved ? warp_sum(psum) : hsum;   // the same slots at the same places
  return RowBuilt{smx, hsum, end - lm, lf, psum};
}

// Batch end, 32 neurons from n0 by a 256-thread block: weights rows -> columnar
// for the slots of omask (the first group of the row, in slot order).  Those
// are the only slots whose weights GSOP can have changed (the others are frozen
// or, without permute, omask holds every used slot).
__device__ __forceinline__ void writeback_tile(int16_t* __restrict__ weights, uint32_t N, uint32_t n0,
                                               const int16_t* __restrict__ rw, const uint16_t* __restrict__ cnt,
                                               const uint4* __restrict__ omask, int16_t (*s_w)[34],
                                               uint32_t* s_c) {
  __shared__ uint4 s_om[32];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t j = warp; j < 32; j += 8) {
    const uint32_t n = n0 + j;
    const uint32_t c = n < N ? (cnt[n] & 0xFFu) : 0u;
    const uint4 om = c ? omask[n] : make_uint4(0, 0, 0, 0);
    if (lane == 0) {
      s_c[j] = (om.x | om.y | om.z | om.w) ? c : 0u;
      s_om[j] = om;
    }
    const uint32_t o[4] = {om.x, om.y, om.z, om.w};
    uint32_t pre = 0;
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      const uint32_t q = 32u * ch + lane;
      if (q < c && ((o[ch] >> lane) & 1u))
        s_w[q][j] = rw[(size_t)n * kRowStride + pre + __popc(o[ch] & ((1u << lane) - 1u))];
      pre += __popc(o[ch]);
    }
  }
  __syncthreads();
  uint32_t cmax = 0;
  for (int j = 0; j < 32; j++) cmax = max(cmax, s_c[j]);
  const uint32_t c_mine = s_c[lane];
  const uint4 om = s_om[lane];
  const uint32_t o[4] = {om.x, om.y, om.z, om.w};
  for (uint32_t r = warp; r < cmax; r += 8)
    if (r < c_mine && ((o[r >> 5] >> (r & 31u)) & 1u)) weights[(size_t)r * N + n0 + lane] = s_w[r][lane];
}

// Batch start: columnar -> rows, tiles of 32 neurons by 256-thread blocks (stage_columns,
// build_row), four resident on an SM and up to four tiles a block (`per`; as many as
// leave each SM its blocks): with a block a tile the batches that keep their layout paid
// 27 us at 1.5M neurons and 135 at 8M for blocks that only return (8 and 35 now), and a
// layout of 8M took 8.8 ms against 8.5.  What the rows add up to is kept in shared
// memory (176 bytes of spills a thread with it in registers, 100 without).
// A slot whose weight GSOP may still move (not frozen_weight, or any slot of a row with
// an invalid target) is movable; weights only freeze, so the marks hold for the whole
// batch.  The dendrite sum (a wrapping i32 sum) and GSOP (per slot) do not depend on the
// order of a row.
// Per neuron: cnt = used slots (| kRowBad | kRowSplit), lfz = movable slots, amask = their
// row positions, omask = the columnar slots placed first (read by the
// write-back; every used slot when the row keeps the columnar order).
constexpr int kBuildBlocks = 4;
constexpr uint32_t kBuildTiles = 4;

__global__ void __launch_bounds__(256, kBuildBlocks) k_rows_build(const uint32_t* __restrict__ targets,
                                                    const int16_t* __restrict__ weights,
                                                    const uint8_t* __restrict__ flags, uint32_t N,
                                                    uint32_t* __restrict__ rt, int16_t* __restrict__ rw,
                                                    uint16_t* __restrict__ cnt, uint4* __restrict__ amask,
                                                    uint4* __restrict__ omask, uint8_t* __restrict__ lfz,
                                                    ShardCtl* __restrict__ ctl, uint32_t A, uint32_t want_sum,
                                                    uint32_t permute, const uint32_t* __restrict__ xlit,
                                                    int2* __restrict__ rec, uint4* __restrict__ lmask,
                                                    uint8_t* __restrict__ posmap, uint32_t* axw, uint32_t cond,
                                                    uint32_t per) {
  if (cond && !ctl->lay_now) return;   // the batch keeps the last layout
  if (keep_segs(ctl, cond)) axw = nullptr;
  __shared__ SlotStage st;
  const uint32_t pmax = lut_pmax(), used = used_segs(ctl, cond);
  // movable slots join the lit groups (no cooling step up to length 16), except in
  // a layout that was forced: the window of always-lit axons is from before what
  // forced it (a LUT, new targets)
  const bool mov_lit = pmax <= 16u && cond && !ctl->lay_forced;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // the block's longest row, largest segment, tested and live slots and (when
  // asked) targets checksum, a warp's each; one atomic each per block
  __shared__ uint32_t s_bc[8], s_bs[8], s_bp[8], s_bl[8], s_bx[8], s_bm[8];
  __shared__ unsigned long long s_bh[8], s_bq[8];
  if (threadIdx.x < 8) {
    s_bc[threadIdx.x] = s_bs[threadIdx.x] = s_bp[threadIdx.x] = s_bl[threadIdx.x] = s_bx[threadIdx.x] = 0;
    s_bm[threadIdx.x] = 0;
    s_bh[threadIdx.x] = s_bq[threadIdx.x] = 0;
  }
  const uint32_t n_end = min(N, (blockIdx.x + 1u) * (32u * per));
#pragma unroll 1
  for (uint32_t n0 = blockIdx.x * (32u * per); n0 < n_end; n0 += 32u) {
    __syncthreads();   // the previous tile's rows are built
    if (threadIdx.x < 32) {
      const uint32_t n = n0 + threadIdx.x;
      const VariantParameters& vp = VARIANT_LUT[n < N ? flags[n] >> 4 : 0];
      st.cnt[threadIdx.x] = AXC_MAX_DENDRITES;
      st.fz[threadIdx.x] = frozen_from(vp);
      st.lit[threadIdx.x] = vp.signal_propagation_length == pmax ? 1u : 0u;
    }
    __syncthreads();
    stage_columns(st, targets, weights, N, n0, A, xlit, mov_lit, axw, used);
    for (uint32_t j = warp; j < 32; j += 8) {
      const uint32_t n = n0 + j;
      if (n >= N) continue;
      const uint32_t c = st.cnt[j];
      const RowBuilt rb = build_row(st, j, n, c, want_sum != 0u, permute != 0u, rt, rw, cnt, amask, omask, lfz, rec,
                                    lmask, posmap);
      if (lane == 0 && c) {   // in shared memory: registers are short
        s_bc[warp] = max(s_bc[warp], c);
        s_bs[warp] = max(s_bs[warp], rb.smx);
        s_bp[warp] += rb.pfx;
        s_bl[warp] += c;
        s_bm[warp] += rb.lf;
        s_bx[warp] |= st.lit[j] == 0u;
        if (want_sum) {
          s_bh[warp] += rb.hsum + slot_mix(c, n);
          s_bq[warp] += rb.psum + slot_mix(c, ~n);
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t bc = 0, bs = 0, bp = 0, bl = 0, bx = 0, bm = 0;
    unsigned long long bh = 0, bq = 0;
    for (int q = 0; q < 8; q++) {
      bc = max(bc, s_bc[q]);
      bs = max(bs, s_bs[q]);
      bh += s_bh[q];
      bp += s_bp[q];
      bl += s_bl[q];
      bx |= s_bx[q];
      bm += s_bm[q];
      bq += s_bq[q];
    }
    if (bc > *(volatile uint32_t*)&ctl->row_smax) atomicMax(&ctl->row_smax, bc);
    if (bs > *(volatile uint32_t*)&ctl->seg_max) atomicMax(&ctl->seg_max, bs);
    if (want_sum) atomicAdd(&ctl->row_sum, bh);
    if (bp) atomicAdd(&ctl->pfx_total, (unsigned long long)bp);
    if (bl) atomicAdd(&ctl->slot_total, (unsigned long long)bl);
    if (bx) ctl->mixed_len = 1u;
    if (bm) atomicAdd(&ctl->mov_total, (unsigned long long)bm);
    if (bq) atomicAdd(&ctl->lay_sum, bq);
  }
}

// Layout start: the axon words cleared and, for permuted rows, the axons
// that were fully lit in every one of the last ticks the rows saw (up to
// kLitWindow of them: one that flickers would send every tick it is dark to the
// dense pass) taken as the lit set of the layout (the prologue checks every tick
// that they still are).
__global__ void __launch_bounds__(256) k_rows_prep(const ShardCtl* __restrict__ ctl, uint32_t* __restrict__ axw,
                                                   uint32_t A, const uint32_t* __restrict__ alit,
                                                   uint32_t* __restrict__ xlit, uint32_t cond) {
  if (cond && !ctl->lay_now) return;
  const uint32_t words = A / 32 + 1, used = (2u << used_segs(ctl, cond)) - 2u;
  const bool keep = keep_segs(ctl, cond);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < A; i += gridDim.x * blockDim.x) {
    axw[i] = keep ? axw[i] & kAxSegs : used;
    if (xlit && i < words) xlit[i] = alit[i];
  }
}

__global__ void __launch_bounds__(256) k_rows_mult(const uint32_t* __restrict__ s2a, uint32_t N, uint32_t A,
                                                   uint32_t* __restrict__ axw, uint2* __restrict__ mask2,
                                                   ShardCtl* __restrict__ ctl, uint32_t cond) {
  if (cond && !ctl->lay_now) return;
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n == 0) {
    mask2[A] = make_uint2(0u, 0x80000000u);   // dummy entry of invalid targets: no hit, exact path
    count_form(ctl, kCountLayout);
    ctl->row_smax = 0;
    ctl->seg_max = 0;
    ctl->row_sum = 0;
    ctl->pmax = lut_pmax();
    ctl->pfx_total = 0;
    ctl->slot_total = 0;
    ctl->mixed_len = 0;
    ctl->mov_total = 0;
    ctl->lay_sum = 0;   // the index holds while the layout it was built from does (checksum)
  }
  if (n >= N) return;
  const uint32_t a = s2a[n];
  if (a < A && (atomicOr(&axw[a], kAxOwned) & kAxOwned)) atomicOr(&axw[a], kAxShared);
}

// Batch end: weights rows -> columnar.  The slots of lmask[n] (in slot order) and
// then the others of omask[n] are the row's first positions, the only slots
// whose weights GSOP can have changed.  Two kernels, one of which returns at once: a
// thread per neuron where the rows have few such slots (a neuron without any, every
// one of a frozen row, costs one 16-byte load and two bytes of cnt, and lmask is read
// of split rows only; 8M settled neurons: 76 us, 88 with lmask read of every row that
// moves, 176 through the tiles' registers and shared memory), else tiles of 32
// neurons: rows read whole, columns written 64 bytes a warp (512k plastic neurons: 100
// us against 228).
__device__ __forceinline__ bool writeback_tiled(const ShardCtl* ctl, uint32_t N) {
  return ctl->mov_total + ctl->pfx_total > 24ull * N;
}

__global__ void __launch_bounds__(256) k_rows_writeback(int16_t* __restrict__ weights, uint32_t N,
                                                        const int16_t* __restrict__ rw,
                                                        const uint16_t* __restrict__ cnt,
                                                        const uint4* __restrict__ omask,
                                                        const uint4* __restrict__ lmask,
                                                        const ShardCtl* __restrict__ ctl, uint32_t* __restrict__ pend,
                                                        uint32_t* __restrict__ incoming, uint32_t A) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  const uint4 om = n < N ? omask[n] : make_uint4(0, 0, 0, 0);   // asked for beside the control block
  const uint32_t cw = n < N ? cnt[n] : 0u;
  const bool tiled = writeback_tiled(ctl, N);
  if (ctl->gave_up)   // pushes of ticks that never ended
    for (uint32_t a = n; a < A; a += gridDim.x * blockDim.x) pend[a] = incoming[a] = 0u;
  if (tiled || !(om.x | om.y | om.z | om.w)) return;
  const uint4 lm = cw & kRowSplit ? lmask[n] : make_uint4(0, 0, 0, 0);   // else one run, in slot order
  const uint32_t o[4] = {om.x, om.y, om.z, om.w}, x[4] = {lm.x, lm.y, lm.z, lm.w};
  const int16_t* row = rw + (size_t)n * kRowStride;
  uint32_t k = 0;
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      uint32_t b = pass ? o[ch] & ~x[ch] : x[ch];
      while (b) {
        const uint32_t q = 32u * ch + (uint32_t)(__ffs(b) - 1);
        b &= b - 1u;
        weights[(size_t)q * N + n] = row[k++];
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_rows_writeback_tiles(int16_t* __restrict__ weights, uint32_t N,
                                                              const int16_t* __restrict__ rw,
                                                              const uint4* __restrict__ omask,
                                                              const uint4* __restrict__ lmask,
                                                              ShardCtl* __restrict__ ctl) {
  __shared__ int16_t s_w[AXC_MAX_DENDRITES][34];
  __shared__ uint32_t s_m[32][4];
  if (blockIdx.x == 0 && threadIdx.x == 0 && ctl->gave_up) ctl->gave_up = 0u;   // cleared by the kernel before
  if (!writeback_tiled(ctl, N)) return;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t t0 = blockIdx.x * 32u; t0 < N; t0 += gridDim.x * 32u) {
    int16_t v[4][4];   // four neurons a warp, every load first
    uint32_t m[4][4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const uint32_t nn = t0 + warp * 4u + e;
      const uint4 a = nn < N ? omask[nn] : make_uint4(0, 0, 0, 0), b = nn < N ? lmask[nn] : make_uint4(0, 0, 0, 0);
      const uint32_t o[4] = {a.x, a.y, a.z, a.w}, x[4] = {b.x, b.y, b.z, b.w};
      uint32_t px = 0, po = popc4(x);
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        m[e][ch] = o[ch];
        const uint32_t rest = o[ch] & ~x[ch], below = (1u << lane) - 1u;
        const uint32_t pos = ((x[ch] >> lane) & 1u) ? px + __popc(x[ch] & below) : po + __popc(rest & below);
        v[e][ch] = ((o[ch] >> lane) & 1u) ? rw[(size_t)nn * kRowStride + pos] : (int16_t)0;
        px += __popc(x[ch]);
        po += __popc(rest);
      }
    }
    __syncthreads();   // the previous 32 are written
#pragma unroll
    for (int e = 0; e < 4; e++) {
#pragma unroll
      for (int ch = 0; ch < 4; ch++) {
        s_w[32u * ch + lane][warp * 4u + e] = v[e][ch];
        if (lane == 0) s_m[warp * 4u + e][ch] = m[e][ch];
      }
    }
    __syncthreads();
    uint32_t c[4];
#pragma unroll
    for (int ch = 0; ch < 4; ch++) c[ch] = s_m[lane][ch];
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t r = warp + 8u * i;
      if ((c[i >> 2] >> (r & 31u)) & 1u) weights[(size_t)r * N + t0 + lane] = s_w[r][lane];
    }
  }
}

// Learned engine, in the prologue: per-tile active synapses and heads in
// flight; on a sparse tick, the block's active axons go into its tile's
// segment (a 256-thread block lies inside one 1024-axon tile).  A tile whose
// active synapses exceed the capacity the predictor gave it sets the overflow
// flag.
__device__ __forceinline__ void learn_axons(const LearnDev& L, uint32_t i, uint32_t A, uint32_t fan,
                                            uint32_t inflight) {
  __shared__ uint32_t s_red[3][8];
  __shared__ uint32_t s_base2;
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const bool act = fan != 0u;
  const uint32_t ball = __ballot_sync(kFull, act);
  const uint32_t f = warp_sum(fan), b = warp_sum(inflight);
  if (lane == 0) { s_red[0][w] = f; s_red[1][w] = b; s_red[2][w] = __popc(ball); }
  __syncthreads();
  const uint32_t i0 = blockIdx.x * blockDim.x;
  const uint32_t j = i0 >> 10;
  const bool sparse = L.ctl->mode == 1u;
  if (threadIdx.x == 0) {
    uint32_t tf = 0, tb = 0, tc = 0;
    for (int q = 0; q < 8; q++) {
      tf += s_red[0][q];
      tb += s_red[1][q];
      const uint32_t c = s_red[2][q];
      s_red[2][q] = tc;
      tc += c;
    }
    s_base2 = 0;
    if (i0 < A) {
      const uint32_t old = atomicAdd(&L.yacc[j], tf);
      atomicAdd(&L.bacc[j], tb);
      if (sparse) {
        if (tc) s_base2 = atomicAdd(&L.fill[j], tc);
        if (old + tf > L.cap[j]) L.ctl->overflow = 1u;
      }
    }
  }
  __syncthreads();
  // an axon is appended once per tick, so a tile's segment never exceeds its 1024 axons
  if (sparse && act) L.alist[(size_t)j * 1024u + s_base2 + s_red[2][w] + __popc(ball & ((1u << lane) - 1u))] = i;
}

// 32 axons' bits of the window of always-lit axons (RowCache::alit).
__device__ __forceinline__ void always_lit(uint32_t* word, uint32_t lit, uint32_t first) {
  if (first) *word = lit;
  else if (lit != 0xFFFFFFFFu) atomicAnd(word, lit);
}

// Counts a prologue block's evaluated neurons and active axons of tick k with
// one atomic; returns the block's first position in the evaluated list.
__device__ __forceinline__ uint32_t append_count(ShardCtl* ctl, uint32_t k, uint32_t eval, uint32_t act) {
  if (!(eval | act)) return 0u;
  return (uint32_t)atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->eval_act[k & 1][0]),
                             ((unsigned long long)act << 32) | eval);
}

// ---------------------------------------------------------------------------
// per tick 1/4 of the learned engine's own graphs: axons (inject, network pushes,
// propagate, split masks) and somas (refractory countdown, list of neurons to
// evaluate), with learn_axons' per-tile activity and, on sparse ticks, the
// compaction of the active axons.  The list entry positions are reserved once
// per block.  The plain engine runs k_rows_prologue_plain.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_rows_prologue(BurstHeads8* __restrict__ heads, uint32_t A, uint32_t v_seg,
                                                       const uint32_t* __restrict__ bitmask, uint32_t voff,
                                                       uint32_t nv, uint32_t* __restrict__ incoming,
                                                       const uint32_t* __restrict__ batch_counts, uint32_t k,
                                                       uint2* __restrict__ mask2, const uint32_t* __restrict__ axw,
                                                       uint8_t* __restrict__ flags, uint8_t* __restrict__ timers,
                                                       uint32_t N, uint32_t* __restrict__ eval,
                                                       ShardCtl* __restrict__ ctl, uint32_t raise_err,
                                                       uint32_t* __restrict__ lit_bits, LearnDev L,
                                                       uint32_t* __restrict__ pend_apply,
                                                       const uint32_t* __restrict__ xlit,
                                                       uint32_t* __restrict__ live, uint32_t* __restrict__ evb,
                                                       uint32_t* __restrict__ alit, uint32_t alit_new) {
  __shared__ uint32_t s_base;
  __shared__ uint32_t s_warp[8], s_act[8];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t xw = (xlit && i < A) ? __ldg(xlit + (i >> 5)) : 0u;   // axons the row layout took as fully lit
  // every load first, with no barrier before them: heads, owners, pending
  // pushes, input bit; the batch constants are read by every thread (the LUT's
  // largest length and the largest segment, both set by the row copy)
  uint4 hx = make_uint4(0, 0, 0, 0), hy = hx;
  uint32_t own = 0, pc = 0, ibit = 0;
  const uint8_t tm = i < N ? timers[i] : (uint8_t)0;
  if (i < A) {
    const uint4* p = reinterpret_cast<const uint4*>(heads + i);
    hx = p[0];
    hy = p[1];
    own = __ldg(axw + i);
    if (pend_apply) pc = pend_apply[i];   // the previous tick's soma pushes (pushes commute)
    if (bitmask) {
      const uint32_t v = i - voff;
      if (v < nv) ibit = (__ldg(bitmask + (v >> 5)) >> (v & 31u)) & 1u;
    }
  }
  const uint32_t pmax = ctl->pmax, seg_max = ctl->seg_max;
  // segments the batch's slots use: 0..seg_max (bit 31: any segment >= 31)
  const uint32_t act = seg_max >= 31u ? 0xFFFFFFFFu : ((2u << seg_max) - 1u);
  const bool inc = batch_counts && batch_counts[k] > 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->ctr[0] += 1;
    if (raise_err) atomicOr(&ctl->err, raise_err);
    ctl->fix_count = 0;      // the previous tick's fix-up is done
    ctl->fix_overflow = 0;
  }
  bool lit = false, on = false;
  uint32_t fan = 0, inflight = 0;   // active synapses and heads in flight of axon i
  if (i < A) {
    uint32_t h[8] = {hx.x, hx.y, hx.z, hx.w, hy.x, hy.y, hy.z, hy.w};
    uint32_t npush = ibit + pc;
    if (pc) pend_apply[i] = 0;
    if (inc) {
      const uint32_t c = incoming[i];
      if (c) { npush += c; incoming[i] = 0; }
    }
    push_n(h, npush);
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (h[j] != AXC_AXON_SENTINEL) h[j] += v_seg;
    uint4* p = reinterpret_cast<uint4*>(heads + i);
    p[0] = make_uint4(h[0], h[1], h[2], h[3]);
    p[1] = make_uint4(h[4], h[5], h[6], h[7]);
    const uint2 m = split_masks(h, pmax, ax_owners(own));
    mask2[i] = m;
    // fully lit: heads 0..6 hit every segment 1..30 the axon's slots use and at
    // most one soma owns the axon, so for those segments the hit is 1 and one
    // push cannot change it
    lit = (m.x & own & kAxSegs) == (own & kAxSegs) && !(m.y >> 31);
    // active: some head covers a segment that a slot of the batch uses
    on = ((m.x | (m.y & 0x7FFFFFFFu)) & act) != 0u;
    if (on) fan = __ldg(L.inv_off + i + 1) - __ldg(L.inv_off + i);
#pragma unroll
    for (int j = 0; j < 8; j++) inflight += h[j] < 255u + pmax ? 1u : 0u;
  }
  learn_axons(L, i, A, fan, inflight);
  if (lit_bits) {
    const uint32_t lb = __ballot_sync(kFull, lit);
    if ((threadIdx.x & 31) == 0 && i < A) {
      lit_bits[i >> 5] = lb;
      always_lit(alit + (i >> 5), lb, alit_new);
      if (xw & ~lb) atomicAdd(&ctl->dense[k & 1], (uint32_t)__popc(xw & ~lb));   // the lit-sum form cannot run this tick
    }
  }
  bool ev = false;
  if (i < N) {
    if (tm > 0) {                                 // physics.cu:168-174 after the burst reset
      timers[i] = (uint8_t)(tm - 1);
      flags[i] = flags[i] & 0xF0;
    } else {
      ev = true;
    }
  }
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t ballot = __ballot_sync(kFull, ev), onb = __ballot_sync(kFull, on);
  if (lane == 0) {
    if (i < N) L.evbits[i >> 5] = evb[i >> 5] = ballot;
    if (i < A) live[i >> 5] = onb;
    s_warp[w] = __popc(ballot);
    s_act[w] = __popc(onb);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0, on_tot = 0;
    for (int q = 0; q < 8; q++) { const uint32_t c = s_warp[q]; s_warp[q] = tot; tot += c; on_tot += s_act[q]; }
    s_base = append_count(ctl, k, tot, on_tot);
  }
  __syncthreads();
  if (ev) eval[s_base + s_warp[w] + __popc(ballot & ((1u << lane) - 1u))] = i;
}

// ---------------------------------------------------------------------------
// per tick 2/4: 8 lanes per evaluated neuron, lane g holds slots
// 32j + 4g .. 32j + 4g + 3 (j = 0..3) of the neuron's row in registers.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t word_of(const uint4& v, int i) {
  return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}
__device__ __forceinline__ int16_t half_of(const uint2& v, int i) {
  const uint32_t w = (i < 2) ? v.x : v.y;
  return (int16_t)((i & 1) ? (w >> 16) : (w & 0xFFFFu));
}
__device__ __forceinline__ void set_half(uint2& v, int i, int16_t x) {
  uint32_t& w = (i < 2) ? v.x : v.y;
  w = (i & 1) ? ((w & 0x0000FFFFu) | ((uint32_t)(uint16_t)x << 16)) : ((w & 0xFFFF0000u) | (uint16_t)x);
}

// Rare paths of the update pass, kept out of line so that the hot loop keeps
// its registers.
__device__ __noinline__ bool hit_exact(const BurstHeads8* heads, uint32_t A, uint32_t a, uint32_t s,
                                       uint32_t prop) {
  return a < A && heads_hit(heads, a, s, prop);
}

// General GSOP of one slot with exact distances.  Returns 0 when applied, 1
// when the slot must be deferred to the fix-up stage (its result depends on
// same-tick pushes), 2 when the target is invalid (skipped, physics.cu would
// read out of bounds).
__device__ __noinline__ int gsop_general(const BurstHeads8* heads, const uint2* mask2, uint32_t A, uint32_t a,
                                         uint32_t s, const VariantParameters& p, uint8_t flags, int32_t dopamine,
                                         int16_t* w16) {
  if (a >= A) return 2;
  const uint2 m = mask2[a];
  uint32_t md, md1;
  md_pair(heads, a, s, p.signal_propagation_length, &md, &md1);
  if ((m.y >> 31) || md != md1) return 1;
  const GsopConsts gc = gsop_consts((uint8_t)((flags & 0xF0) | 0x05), p, dopamine);
  *w16 = gsop_weight(*w16, md, p, gc.bm, gc.raw_pot, gc.final_dep);
  return 0;
}

// GSOP deltas per variant and inertia rank for a spiker (flags type | 0b101:
// burst multiplier 2, physics.cu:255, 271-273, 290-291; physics.cu:336-349).
// Called by the first 256 threads of the block.
// The LUT's largest signal_propagation_length; seen by all after the next barrier.
__device__ __forceinline__ void pmax_of(uint32_t* dst, const VariantParameters* lut) {
  if (threadIdx.x < 32) {
    const uint32_t m = __reduce_max_sync(kFull, lut[threadIdx.x & 15].signal_propagation_length);
    if (threadIdx.x == 0) *dst = m;
  }
}

__device__ __forceinline__ void build_gtab(int2 (*gtab)[16], const VariantParameters* lut, int32_t dopamine) {
  if (threadIdx.x < 256) {
    const uint32_t v = threadIdx.x >> 4, r = threadIdx.x & 15;
    const GsopConsts g = gsop_consts((uint8_t)((v << 4) | 0x05), lut[v], dopamine);
    const int32_t inertia = lut[v].inertia_curve[r];
    gtab[v][r] = make_int2(wmul(wmul(g.raw_pot, inertia), g.bm) >> 7, wmul(wmul(g.final_dep, inertia), g.bm) >> 7);
  }
}

// How the 8 lanes of a neuron hold its row, from the shard's longest row
// smax: F full rounds of 32 slots (lane g: slots 32j+4g..32j+4g+3, one vector
// load each of targets and weights) and, for rows that end inside a round, TR
// single-slot rounds (lane g: slot 32F+g+8t) kept in the round-3 registers
// (T[3].x / T[3].y, the two halves of W[3].x).  A 100-slot row takes 3 full
// rounds and one single-slot round instead of 4 full rounds, three quarters of
// whose last round would be empty; a tail of more than 16 slots takes a full
// round.
struct RowShape {
  uint32_t F, TR;
};

__device__ __forceinline__ RowShape row_shape(uint32_t smax) {
  uint32_t F = smax >> 5, tail = smax & 31u;
  if (tail > 16u) {
    F++;
    tail = 0;
  }
  return RowShape{F, (tail + 7u) >> 3};
}

__device__ __forceinline__ void row_load(uint4 (&T)[4], uint2 (&W)[4], const uint32_t* rt_n, const int16_t* rw_n,
                                         uint32_t g8, bool valid, RowShape sh, uint32_t smax) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    T[j] = make_uint4(0, 0, 0, 0);
    W[j] = make_uint2(0, 0);
    if (valid && (uint32_t)j < sh.F && 32u * j + 4u * g8 < smax) {
      T[j] = __ldg(reinterpret_cast<const uint4*>(rt_n + 32 * j + 4 * g8));
      W[j] = *reinterpret_cast<const uint2*>(rw_n + 32 * j + 4 * g8);
    }
  }
  if (sh.F < 4u && valid) {
    const uint32_t q0 = 32u * sh.F + g8;
    if (sh.TR > 0u && q0 < smax) {
      T[3].x = __ldg(rt_n + q0);
      W[3].x = (uint16_t)rw_n[q0];
    }
    if (sh.TR > 1u && q0 + 8u < smax) {
      T[3].y = __ldg(rt_n + q0 + 8);
      W[3].x |= (uint32_t)(uint16_t)rw_n[q0 + 8] << 16;
    }
  }
}

// Bulk copy global -> shared completed on an mbarrier (cp.async.bulk, the
// untiled TMA path: 16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bulk_to_smem(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for phase `parity` of bar at most `tries` tries (default kWaitLimit); false: gave up.
constexpr uint32_t kWaitLimit = 1u << 16;
// Tries of the update pass's first wait for the staged bitmap
// (axc_row_engine_wait_limit; tests set 0 to take the give-up path).  The
// drain wait before the block exits always has kWaitLimit tries.
__device__ uint32_t g_first_wait_limit = kWaitLimit;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t tries = kWaitLimit) {
  for (uint32_t it = 0; it < tries; it++)
    if (mbar_test(bar, parity)) return true;
  return false;
}

// The dendrite pass over the slots one lane holds (row_shape) of a row with c
// used slots: returns the lane's share of the input current and sets, per slot
// (bit 4j+i; single-slot round t: bit 12+t), hitb = the segment is hit and
// slowb = GSOP needs the exact path (physics.cu:186-207 for the hit test).
template <bool LIT>
__device__ __forceinline__ int32_t row_slots(const uint4 (&T)[4], const uint2 (&W)[4], uint32_t c, uint32_t g8,
                                             RowShape sh, const uint2* mask2, const uint32_t* s_lit,
                                             uint32_t seg_hi, bool exact, bool gfast, uint32_t prop,
                                             const BurstHeads8* heads, uint32_t A, uint32_t& hitb_out,
                                             uint32_t& slowb_out, bool lit_on = true) {
  int32_t i_in = 0;
  const bool glit = LIT && lit_on && gfast;   // the fully-lit shortcut applies
  uint32_t hitb = 0, slowb = 0;   // bit 4j+i
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if ((uint32_t)j >= sh.F) continue;
    const uint32_t q0 = 32u * j + 4u * g8;
    uint2 m[4];
    bool lit[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t t = word_of(T[j], i);
      const uint32_t ax = (t & AXC_TARGET_AXON_MASK) - 1u;   // invalid ids were redirected to A
      lit[i] = glit && ((t >> AXC_TARGET_SEG_SHIFT) - 1u) < seg_hi && ((s_lit[ax >> 5] >> (ax & 31u)) & 1u);
      m[i] = (q0 + i < c && !lit[i]) ? mask2[ax] : make_uint2(0, 0);
    }
    uint32_t need = 0;   // live slots off the fully-lit path
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (q0 + i >= c) continue;
      if (LIT && lit[i]) {                      // segment 1..30 of a fully lit axon: hit, fast GSOP
        i_in = wadd(i_in, (int32_t)half_of(W[j], i));
        hitb |= 1u << (4 * j + i);
      } else {
        need |= 1u << i;
      }
    }
    // warp-uniform: most rounds have every slot of the warp's four rows on the
    // fully-lit path, and skip the mask path as a whole
    if (LIT && !__any_sync(kFull, need)) continue;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (!((need >> i) & 1u)) continue;
      const uint32_t t = word_of(T[j], i);
      const uint32_t s = t >> AXC_TARGET_SEG_SHIFT;
      const uint32_t sh = min(s, 31u);
      const uint32_t bx = (m[i].x >> sh) & 1u, by = (m[i].y >> sh) & 1u;
      bool hit = (bx | by) != 0u;              // bit 31 (s >= 31): "may hit", tested below
      if (hit && (s >= 31u || !exact))
        hit = hit_exact(heads, A, (t & AXC_TARGET_AXON_MASK) - 1u, s, prop);
      if (hit) {
        i_in = wadd(i_in, (int32_t)half_of(W[j], i));
        hitb |= 1u << (4 * j + i);
      }
      // fast GSOP: hit decides, and one same-tick push could not change it
      const bool fast = gfast && s < 31u && !(m[i].y >> 31) && (bx || by == (s == 0u));
      slowb |= fast ? 0u : (1u << (4 * j + i));
    }
  }
  if (sh.F < 4u) {
    // single-slot tail rounds t = 0, 1: slot 32F + g8 + 8t, bit 12 + t
    uint2 m[2];
    uint32_t need = 0;
#pragma unroll
    for (int t = 0; t < 2; t++) {
      m[t] = make_uint2(0, 0);
      const uint32_t q = 32u * sh.F + g8 + 8u * t;
      if ((uint32_t)t >= sh.TR || q >= c) continue;
      const uint32_t tw = t ? T[3].y : T[3].x;
      const uint32_t ax = (tw & AXC_TARGET_AXON_MASK) - 1u;
      if (glit && ((tw >> AXC_TARGET_SEG_SHIFT) - 1u) < seg_hi && ((s_lit[ax >> 5] >> (ax & 31u)) & 1u)) {
        i_in = wadd(i_in, (int32_t)half_of(W[3], t));
        hitb |= 1u << (12 + t);
      } else {
        m[t] = mask2[ax];
        need |= 1u << t;
      }
    }
    if (!LIT || __any_sync(kFull, need)) {
#pragma unroll
      for (int t = 0; t < 2; t++) {
        if (!((need >> t) & 1u)) continue;
        const uint32_t tw = t ? T[3].y : T[3].x;
        const uint32_t b = 1u << (12 + t);
        const int32_t w = (int32_t)half_of(W[3], t);
        const uint32_t s = tw >> AXC_TARGET_SEG_SHIFT;
        const uint32_t shv = min(s, 31u);
        const uint32_t bx = (m[t].x >> shv) & 1u, by = (m[t].y >> shv) & 1u;
        bool hit = (bx | by) != 0u;
        if (hit && (s >= 31u || !exact)) hit = hit_exact(heads, A, (tw & AXC_TARGET_AXON_MASK) - 1u, s, prop);
        if (hit) {
          i_in = wadd(i_in, w);
          hitb |= b;
        }
        const bool fast = gfast && s < 31u && !(m[t].y >> 31) && (bx || by == (s == 0u));
        slowb |= fast ? 0u : b;
      }
    }
  }
  hitb_out = hitb;
  slowb_out = slowb;
  return i_in;
}

// GLIF of one evaluated (non-refractory) neuron, physics.cu:209-275.
struct GlifOut {
  int32_t v, thr;
  int glif, spike;
};

__device__ __forceinline__ GlifOut glif_step(const VariantParameters& p, int32_t v0, int32_t thr0, int32_t i_in,
                                             uint32_t tick, uint32_t n) {
  GlifOut o;
  const int32_t decayed = wsub(thr0, (int32_t)p.homeostasis_decay);
  int32_t thr = decayed & ~(decayed >> 31);
  int32_t leak = p.leak_rate;
  if (p.adaptive_mode == 1) {
    leak = wadd(leak, wmul(thr, (int32_t)p.adaptive_leak_gain) >> 8);
    const int32_t over = wsub(leak, p.adaptive_leak_max);
    leak = wsub(leak, over & ~(over >> 31));
  }
  int32_t v = wadd(v0, i_in);
  const int32_t diff = wsub(v, p.rest_potential);
  const int32_t sign = (diff > 0) - (diff < 0);
  int32_t leaked = wsub(wmul(diff, sign), leak);
  leaked = leaked & ~(leaked >> 31);
  v = wadd(p.rest_potential, wmul(sign, leaked));
  const int glif = v >= wadd(p.threshold, thr) ? 1 : 0;
  const uint32_t period = p.spontaneous_firing_period_ticks;
  const int hb = (period > 0 && ((tick + n * 104729u) % period) == 0) ? 1 : 0;
  if (glif) {
    v = p.rest_potential;
    thr = wadd(thr, p.homeostasis_penalty);
  }
  o.v = v;
  o.thr = thr;
  o.glif = glif;
  o.spike = glif | hb;
  return o;
}

// GSOP of a spiker's slots held by this lane (physics.cu:281-373): fast slots
// from the gtab deltas, slow ones on the exact path or deferred to the fix-up
// list.  same: 4-slot groups visited << 16 | those that kept their weights.
// Writes the changed weights back to the row (rt_n / rw_n: the neuron's row);
// returns the slots done.
template <bool WT = false>
__device__ __forceinline__ uint32_t row_gsop(uint2 (&W)[4], uint32_t hitb, uint32_t slowb,
                                             uint32_t c, uint32_t g8, RowShape sh, const int2 (*gtab)[16],
                                             uint32_t var, const uint32_t* rt_n, int16_t* rw_n,
                                             const BurstHeads8* heads, const uint2* mask2, uint32_t A,
                                             const VariantParameters& p, uint8_t flags, int32_t dopamine,
                                             ShardCtl* ctl, uint32_t* fix, uint32_t fix_cap, uint32_t n,
                                             uint32_t& same, const ColWT& wt = ColWT{}) {
  uint32_t gdone = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if ((uint32_t)j >= sh.F) continue;
    const uint32_t q0 = 32u * j + 4u * g8;
    if (q0 >= c) continue;
    uint2 wj = W[j];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t b = 1u << (4 * j + i);
      if (q0 + i >= c) continue;
      const int16_t w16 = half_of(wj, i);
      if (!(slowb & b)) {
        // cooling shift 0: delta = +potentiation or -depression of the weight's rank
        const int32_t aw = w16 < 0 ? -(int32_t)w16 : (int32_t)w16;
        const int2 e = gtab[var][min((uint32_t)aw >> 11, 15u)];
        int32_t na = aw + ((hitb & b) ? e.x : -e.y);
        na = min(max(na, 0), 32767);
        set_half(wj, i, (int16_t)(w16 < 0 ? -na : na));
        gdone++;
        continue;
      }
      const uint32_t t = __ldg(rt_n + q0 + i);
      int16_t nw = w16;
      const int r = gsop_general(heads, mask2, A, (t & AXC_TARGET_AXON_MASK) - 1u, t >> AXC_TARGET_SEG_SHIFT, p,
                                 flags, dopamine, &nw);
      if (r == 2) continue;
      gdone++;
      if (r == 1) {
        const uint32_t slot = atomicAdd(&ctl->fix_count, 1u);
        if (slot < fix_cap) fix[slot] = (uint32_t)((size_t)n * kRowStride + q0 + i);
        else ctl->fix_overflow = 1u;
        continue;
      }
      set_half(wj, i, nw);
    }
    same += 0x10000u;   // visited, and (low half) left as they were
    if (wj.x == W[j].x && wj.y == W[j].y) {
      same++;
    } else {
      *reinterpret_cast<uint2*>(rw_n + q0) = wj;
      if (WT) {
        ColRun cols(wt, n, q0);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          if (q0 + i >= c) break;
          const uint32_t q = cols.next(wt, n);
          if (half_of(wj, i) != half_of(W[j], i)) wt.w[(size_t)q * wt.N + n] = half_of(wj, i);
        }
      }
    }
  }
  if (sh.F < 4u) {
#pragma unroll
    for (int t = 0; t < 2; t++) {
      if ((uint32_t)t >= sh.TR) continue;
      const uint32_t q = 32u * sh.F + g8 + 8u * t;
      if (q >= c) continue;
      const uint32_t b = 1u << (12 + t);
      const int16_t w16 = half_of(W[3], t);
      int16_t nw = w16;
      if (!(slowb & b)) {
        const int32_t aw = w16 < 0 ? -(int32_t)w16 : (int32_t)w16;
        const int2 e = gtab[var][min((uint32_t)aw >> 11, 15u)];
        int32_t na = aw + ((hitb & b) ? e.x : -e.y);
        na = min(max(na, 0), 32767);
        nw = (int16_t)(w16 < 0 ? -na : na);
        gdone++;
      } else {
        const uint32_t tw = __ldg(rt_n + q);
        const int r = gsop_general(heads, mask2, A, (tw & AXC_TARGET_AXON_MASK) - 1u, tw >> AXC_TARGET_SEG_SHIFT,
                                   p, flags, dopamine, &nw);
        if (r == 2) continue;
        gdone++;
        if (r == 1) {
          const uint32_t slot = atomicAdd(&ctl->fix_count, 1u);
          if (slot < fix_cap) fix[slot] = (uint32_t)((size_t)n * kRowStride + q);
          else ctl->fix_overflow = 1u;
          continue;
        }
      }
      if (nw != w16) {
        rw_n[q] = nw;
        if (WT) col_write(wt, n, q, nw);
      }
    }
  }
  return gdone;
}

// The hit test of one slot as the 8-lane pass makes it (row_slots): the
// fully-lit shortcut for segments 1..seg_hi of variants whose length is the LUT
// maximum (<= 16), else the tick's split masks and, where they do not decide,
// the eight heads.  *fast: GSOP may take the slot's delta from the gtab table
// (the hit decides and one same-tick push cannot change it).
__device__ __forceinline__ bool slot_hit(uint32_t t, bool exact, bool gfast, uint32_t prop, uint32_t seg_hi,
                                         const uint32_t* lit_bits, const uint2* mask2,
                                         const BurstHeads8* heads, uint32_t A, bool* fast) {
  const uint32_t s = t >> AXC_TARGET_SEG_SHIFT;
  const uint32_t ax = (t & AXC_TARGET_AXON_MASK) - 1u;   // invalid ids were redirected to A (dummy mask entry)
  if (gfast && (s - 1u) < seg_hi && ((lit_bits[ax >> 5] >> (ax & 31u)) & 1u)) {
    *fast = true;
    return true;
  }
  const uint2 m = mask2[ax];
  const uint32_t sh = min(s, 31u);
  const uint32_t bx = (m.x >> sh) & 1u, by = (m.y >> sh) & 1u;
  bool hit = (bx | by) != 0u;
  if (hit && (s >= 31u || !exact)) hit = hit_exact(heads, A, ax, s, prop);
  *fast = gfast && s < 31u && !(m.y >> 31) && (bx || by == (s == 0u));
  return hit;
}

// GSOP (physics.cu:281-373) of row position q of spiker n, weight w16, target
// *t: the rank's delta where the hit decides (fast), else the exact path or the
// fix-up list.  Returns the slots done (0: an invalid target).
template <bool WT>
__device__ __forceinline__ uint32_t gsop_slot(int16_t w16, const uint32_t* t, int16_t* w, bool hit, bool fast,
                                              const int2* gtab_v, const BurstHeads8* heads, const uint2* mask2,
                                              uint32_t A, const VariantParameters& p, uint8_t flags, int32_t dopamine,
                                              ShardCtl* ctl, uint32_t* fix, uint32_t fix_cap, uint32_t n, uint32_t q,
                                              const ColWT& wt) {
  int16_t nw = w16;
  if (fast) {
    const int32_t aw = w16 < 0 ? -(int32_t)w16 : (int32_t)w16;
    const int2 e = gtab_v[min((uint32_t)aw >> 11, 15u)];
    int32_t na = aw + (hit ? e.x : -e.y);
    na = min(max(na, 0), 32767);
    nw = (int16_t)(w16 < 0 ? -na : na);
  } else {
    const uint32_t tt = *t;
    const int r = gsop_general(heads, mask2, A, (tt & AXC_TARGET_AXON_MASK) - 1u, tt >> AXC_TARGET_SEG_SHIFT, p, flags,
                               dopamine, &nw);
    if (r == 2) return 0u;
    if (r == 1) {
      const uint32_t slot = atomicAdd(&ctl->fix_count, 1u);
      if (slot < fix_cap) fix[slot] = (uint32_t)((size_t)n * kRowStride + q);
      else ctl->fix_overflow = 1u;
      return 1u;
    }
  }
  if (nw != w16) {
    *w = nw;
    if (WT) col_write(wt, n, q, nw);
  }
  return 1u;
}

struct LsumCount {
  uint32_t ev_slots, hits, nspk, gdone, nev, err, tested, same;
};

// The state of a neuron after GLIF and its spike's push.
__device__ __forceinline__ void neuron_store(const ShardVramPtrs& P, uint32_t n, const GlifOut& o, uint8_t flags,
                                             const VariantParameters& p, uint32_t my_axon, uint32_t A, uint32_t* pend,
                                             LsumCount& k) {
  P.soma_voltage[n] = o.v;
  P.soma_flags[n] = (uint8_t)((flags & 0xF0) | (o.spike ? 0x05 : 0x00));
  P.threshold_offset[n] = o.thr;
  P.timers[n] = o.glif ? p.refractory_period : 0;
  if (!o.spike) return;
  k.nspk++;
  if (my_axon != AXC_NO_AXON) {
    if (my_axon < A) atomicAdd(&pend[my_axon], 1u);
    else k.err |= AXC_ERR_SOMA_AXON;
  }
}

// GSOP of a movable lit slot: a hit within the first 16 segments' cooling step,
// so the weight takes its rank's potentiation.
__device__ __forceinline__ int16_t gsop_lit(int16_t w16, const int2* gtab_v) {
  const int32_t aw = w16 < 0 ? -(int32_t)w16 : (int32_t)w16;
  int32_t na = aw + gtab_v[min((uint32_t)aw >> 11, 15u)].x;
  na = min(max(na, 0), 32767);
  return (int16_t)(w16 < 0 ? -na : na);
}

// GSOP of two movable lit slots in one register (gsop_lit for each half), for
// potentiations 0..16383 (tab: per rank 0..16, in the low half): |w| is w xor its
// sign mask plus one where negative, the sums stay below 2^16, and a weight that
// was negative stays at least 1 in size, so no half carries into the other.
__device__ __forceinline__ uint32_t gsop_lit2(uint32_t w, const uint32_t* tab) {
  uint32_t s;   // 0xFFFF in a negative half (prmt with the sign-replicating selectors 8 + byte)
  asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(s) : "r"(w));
  const uint32_t aw = (w ^ s) + (s & 0x00010001u);
  const uint32_t d = __byte_perm(tab[(aw >> 11) & 31u], tab[aw >> 27], 0x5410);
  const uint32_t na = __vminu2(aw + d, 0x7FFF7FFFu);
  return (na ^ s) + (s & 0x00010001u);
}

// One step of the lit rows, 8 lanes per neuron: lane g8 holds row positions
// 64 r + 8 g8 .. + 7 (r = 0, 1), the movable slots' weights in two 16-byte
// registers.  VERIFY: the row's lit slots are looked up in the tick's fully-lit
// bitmap (s_lit; lit_on false: not there); a row with a dark one is tested slot
// by slot.  tab (null: some potentiation does not fit) serves GSOP two slots at a
// time.  All 32 lanes take part.
// Bound by instructions: 12.3M movable lit slots a tick (512k neurons, 96 slots,
// a quarter evaluated) cost ~15 each with the look-up, where the slot-by-slot
// pass spent ~85.
template <bool VERIFY, bool WT>
__device__ __forceinline__ void lit_row_step(const ShardVramPtrs& P, uint32_t A, const uint32_t* __restrict__ rt,
                                             int16_t* rw, const uint16_t* __restrict__ cnt,
                                             const uint2* mask2, uint32_t* pend,
                                             uint32_t* fix, ShardCtl* ctl, uint32_t fix_cap,
                                             const int2* __restrict__ rec, const ColWT& wt,
                                             const VariantParameters* lut, const int2 (*gtab)[16],
                                             const uint32_t (*tab)[17], uint32_t pmax, uint32_t smax, uint32_t tick,
                                             int32_t dopamine, uint32_t n, bool valid, const uint32_t* s_lit,
                                             bool lit_on, LsumCount& kc) {
  const uint32_t g8 = threadIdx.x & 7u;
  // every load of the neuron at once; the movable slots are most of the row
  const uint8_t flags = P.soma_flags[n];
  const uint32_t cw = cnt[n];
  const int2 ls = __ldg(rec + n);
  const int32_t thr0 = P.threshold_offset[n];
  const int32_t v0 = P.soma_voltage[n];
  const uint32_t my_axon = __ldg(P.soma_to_axon + n);
  const uint32_t* rt_n = rt + (size_t)n * kRowStride;
  int16_t* rw_n = rw + (size_t)n * kRowStride;
  uint4 W[2], T[VERIFY ? 4 : 1];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const bool in = 64u * r + 8u * g8 < smax;
    W[r] = in ? *reinterpret_cast<const uint4*>(rw_n + 64 * r + 8 * g8) : make_uint4(0, 0, 0, 0);
    if (VERIFY) {
#pragma unroll
      for (int x = 0; x < 2; x++)
        T[2 * r + x] = in ? __ldg(reinterpret_cast<const uint4*>(rt_n + 64 * r + 8 * g8) + x) : make_uint4(0, 0, 0, 0);
    }
  }
  const uint32_t c = cw & 0xFFu, y = (uint32_t)ls.y;
  const uint32_t lm = y & 0xFFu, lf = (y >> 8) & 0xFFu, end = (y >> 16) & 0xFFu;
  const uint32_t var = flags >> 4;
  const VariantParameters& p = lut[var];
  const uint32_t prop = p.signal_propagation_length;
  const bool exact = prop == pmax;
  const bool gfast = exact && prop <= 16u;
  int32_t i_in = g8 == 0 ? ls.x : 0;
  uint32_t all_lit = 1u;   // bit 0: every lit slot looked up so far is on a fully-lit axon
  // movable lit slots: positions 0 .. lm - 1
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const uint32_t q0 = 64u * r + 8u * g8;
    if (q0 + 8u <= lm) {
#pragma unroll
      for (int h = 0; h < 4; h++) i_in = __dp2a_lo((int)word_of(W[r], h), 0x0101, i_in);
      if (VERIFY && lit_on) {
#pragma unroll
        for (int h = 0; h < 8; h++) {
          const uint32_t u = word_of(T[2 * r + (h >> 2)], h & 3) - 1u;   // axon in the low 24 bits
          all_lit &= s_lit[(u & AXC_TARGET_AXON_MASK) >> 5] >> (u & 31u);
        }
      }
    } else if (q0 < lm) {
#pragma unroll 1
      for (uint32_t q = q0; q < lm; q++) {
        i_in = wadd(i_in, (int32_t)rw_n[q]);
        if (VERIFY && lit_on) {
          const uint32_t u = __ldg(rt_n + q) - 1u;
          all_lit &= s_lit[(u & AXC_TARGET_AXON_MASK) >> 5] >> (u & 31u);
        }
      }
    }
  }
  bool dark = false;   // the row is tested slot by slot
  if (VERIFY) {
    // the frozen lit slots end .. c - 1 (few or none where most slots move)
    if (lit_on)
      for (uint32_t q = end + g8; q < c; q += 8u) {
        const uint32_t u = __ldg(rt_n + q) - 1u;
        all_lit &= s_lit[(u & AXC_TARGET_AXON_MASK) >> 5] >> (u & 31u);
      }
    const uint32_t b = __ballot_sync(kFull, !lit_on || !(all_lit & 1u));
    dark = (b >> (threadIdx.x & 24u)) & 0xFFu;
  }
  // tested slots: positions lm .. end - 1, one a lane; of a dark row every slot
  const uint32_t q0 = dark ? 0u : lm, nt = dark ? c : end - lm;
  if (dark) i_in = 0;
  uint32_t hb = 0, fb = 0;   // bit r: this lane's r-th tested slot is a hit / in GSOP's fast class
  // four a lane at a time, each load of the four before any is waited for (slot
  // -> mask is a chain of two cache misses, and one such row in a warp's slice
  // would hold up its block)
  for (uint32_t x0 = 0; x0 < nt; x0 += 32u) {
    uint32_t t[4];
    int32_t w[4];
    uint2 m[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t x = x0 + 8u * u + g8;
      t[u] = x < nt ? __ldg(rt_n + q0 + x) : 0u;
      w[u] = x < nt ? (int32_t)rw_n[q0 + x] : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)   // invalid ids were redirected to A (dummy mask entry)
      m[u] = x0 + 8u * u + g8 < nt ? mask2[(t[u] & AXC_TARGET_AXON_MASK) - 1u] : make_uint2(0, 0);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (x0 + 8u * u + g8 >= nt) continue;
      const uint32_t s = t[u] >> AXC_TARGET_SEG_SHIFT, sh = min(s, 31u);
      const uint32_t bx = (m[u].x >> sh) & 1u, by = (m[u].y >> sh) & 1u;
      bool hit = (bx | by) != 0u;              // bit 31 (s >= 31): "may hit", tested below
      if (hit && (s >= 31u || !exact)) hit = hit_exact(P.axon_heads, A, (t[u] & AXC_TARGET_AXON_MASK) - 1u, s, prop);
      const uint32_t bit = 1u << (x0 / 8u + u);
      if (hit) {
        i_in = wadd(i_in, w[u]);
        hb |= bit;
      }
      fb |= gfast && s < 31u && !(m[u].y >> 31) && (bx || by == (s == 0u)) ? bit : 0u;
    }
  }
  i_in = wadd(i_in, __shfl_xor_sync(kFull, i_in, 1));
  i_in = wadd(i_in, __shfl_xor_sync(kFull, i_in, 2));
  i_in = wadd(i_in, __shfl_xor_sync(kFull, i_in, 4));
  if (!valid) return;
  kc.hits += __popc(hb);
  const GlifOut o = glif_step(p, v0, thr0, i_in, tick, n);
  if (g8 == 0) {
    if (cw & kRowBad) kc.err |= AXC_ERR_TARGET_RANGE;
    kc.ev_slots += c;
    if (!dark) kc.hits += (c - end) + lm;
    kc.tested += nt;
    kc.nev++;
    neuron_store(P, n, o, flags, p, my_axon, A, pend, kc);
    if (o.spike) kc.gdone += (c - lf) + (dark ? 0u : lm);   // the frozen slots are left as they are
  }
  if (!o.spike) return;
  if (!dark) {
#pragma unroll
    for (int r = 0; r < 2; r++) {
      const uint32_t qr = 64u * r + 8u * g8;
      if (qr + 8u <= lm && tab) {
        const uint4 nw = make_uint4(gsop_lit2(W[r].x, tab[var]), gsop_lit2(W[r].y, tab[var]),
                                    gsop_lit2(W[r].z, tab[var]), gsop_lit2(W[r].w, tab[var]));
        kc.same += 0x10000u;   // groups visited << 16 | left as they were
        if (nw.x == W[r].x && nw.y == W[r].y && nw.z == W[r].z && nw.w == W[r].w) {
          kc.same++;
          continue;
        }
        *reinterpret_cast<uint4*>(rw_n + qr) = nw;
        if (WT) {
          ColRun cols(wt, n, qr);
#pragma unroll 1
          for (uint32_t h = 0; h < 8; h++) {
            const uint32_t q = cols.next(wt, n);
            const int16_t a = (int16_t)(word_of(nw, h >> 1) >> (16u * (h & 1u)));
            if (a != (int16_t)(word_of(W[r], h >> 1) >> (16u * (h & 1u)))) wt.w[(size_t)q * wt.N + n] = a;
          }
        }
      } else {
#pragma unroll 1
        for (uint32_t q = qr; q < min(qr + 8u, lm); q++) {
          const int16_t w16 = rw_n[q];
          const int16_t nw = gsop_lit(w16, gtab[var]);
          if (nw == w16) continue;
          rw_n[q] = nw;
          if (WT) col_write(wt, n, q, nw);
        }
      }
    }
  }
  // the movable ones among the tested slots
  const uint32_t mt = dark ? lf : lf - lm;
  for (uint32_t x = g8, r = 0; x < mt; x += 8u, r++)
    kc.gdone += gsop_slot<WT>(rw_n[q0 + x], rt_n + q0 + x, rw_n + q0 + x, (hb >> r) & 1u, (fb >> r) & 1u, gtab[var],
                              P.axon_heads, mask2, A, p, flags, dopamine, ctl, fix, fix_cap, n, q0 + x, wt);
}

// The potentiations of gtab for gsop_lit2; false (in every thread) when one does
// not fit.  Called by all threads of the block.
__device__ __forceinline__ bool build_ptab(uint32_t (*tab)[17], const int2 (*gtab)[16]) {
  bool ok = true;
  for (uint32_t i = threadIdx.x; i < 16u * 17u; i += blockDim.x) {
    const int32_t x = gtab[i / 17u][min(i % 17u, 15u)].x;
    ok = ok && x >= 0 && x <= 16383;
    tab[i / 17u][i % 17u] = (uint32_t)x;
  }
  return __syncthreads_and(ok);
}

// Sums per-thread counters over a block: v[0..5] into ctr[1..5] and ctr[7] (evaluated
// slots, hits, spikes, GSOP slots, evaluated neurons, tested slots), v[6..7] into
// gsop_same.  Two warp reductions, one barrier and one atomic per counter: 64-bit
// shuffles and a serial sum over 32 warps were 8,000 cycles of the 8-lane pass.
template <int NC>
__device__ __forceinline__ void block_counts(const uint32_t (&v)[NC], unsigned long long* ctr,
                                             unsigned long long* gsop_same = nullptr) {
  __shared__ uint32_t red[NC][32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int c = 0; c < NC; c++) {
    const uint32_t x = __reduce_add_sync(kFull, v[c]);
    if (lane == 0) red[c][w] = x;
  }
  __syncthreads();
  if (w < (uint32_t)NC) {
    const uint32_t sum = __reduce_add_sync(kFull, lane < nw ? red[w][lane] : 0u);
    unsigned long long* dst = w < 5u ? ctr + 1 + w : w == 5u ? ctr + 7 : gsop_same + (w - 6u);
    if (lane == 0 && sum) atomicAdd(dst, (unsigned long long)sum);
  }
}

// What a pass reads of the control block, asked for in one go.
struct PassCtl {
  uint32_t tick, smax, seg_max;
};
__device__ __forceinline__ PassCtl pass_ctl(const ShardCtl* ctl, uint32_t k) {
  return {ctl_ld32(&ctl->tick_base) + k, ctl_ld32(&ctl->row_smax), ctl_ld32(&ctl->seg_max)};
}

// The 8-lane pass over the tick's evaluated neurons, one form of three (dense,
// lit rows, checked lit rows).  s_lit: the tick's fully-lit bitmap (one bit per
// axon), in shared memory where it fits, else in global memory; lit_on false: it
// did not arrive, the pass does without it (results exact).  Slots whose axon is
// fully lit need no mask gather from L2.
// WT: write GSOP's changes through to the columnar blob (the per-tick entry point).
// Warp wid of the nwarps that share the list; counts: this thread's (block_counts).
template <bool WT>
__device__ __forceinline__ void rows_update(TickForm form, uint32_t wid, uint32_t nwarps, const PassCtl& pc,
                                            const ShardVramPtrs& P, uint32_t A, const uint32_t* rt, int16_t* rw,
                                            const uint16_t* cnt, const uint2* mask2, const uint32_t* eval,
                                            uint32_t ecount, uint32_t* pend, uint32_t* fix, ShardCtl* ctl,
                                            uint32_t fix_cap, const uint8_t* lfz, const ColWT& wt, const int2* rec,
                                            const VariantParameters* lut, const int2 (*gtab)[16],
                                            const uint32_t (*ptab)[17], uint32_t pmax, int32_t dopamine,
                                            const uint32_t* s_lit, bool lit_on, uint32_t (&counts)[8]) {
  const uint32_t tick = pc.tick;
  const uint32_t smax = pc.smax;   // longest row of the shard: rows are loaded up to here
  const RowShape sh = row_shape(smax);
  const uint32_t seg_hi = min(pc.seg_max, 30u);   // lit bits cover segments 1..seg_hi
  const uint32_t lane = threadIdx.x & 31, g8 = lane & 7, grp = lane >> 3;
  // Four neurons a step.  The warps take the steps in turn, which evens out a short
  // list; of a long one each has a slice of its own.
  const uint32_t per_warp = ecount < 64u * nwarps ? 0u : (((ecount + nwarps - 1) / nwarps) + 3u) & ~3u;
  const uint32_t step = per_warp ? 4u : 4u * nwarps;
  const uint32_t beg = per_warp ? wid * per_warp : 4u * wid;
  const uint32_t end = per_warp ? min(beg + per_warp, ecount) : ecount;
  uint32_t ev_slots = 0, hits = 0, nspk = 0, gdone = 0, nev = 0, err = 0;
  uint32_t same = 0;         // row_gsop
  uint32_t lit_tested = 0;
  if (form != kFormDense) {
    LsumCount kc = {0, 0, 0, 0, 0, 0, 0, 0};
    if (form == kFormVerify) {
      for (uint32_t i0 = beg; i0 < end; i0 += step)
        lit_row_step<true, WT>(P, A, rt, rw, cnt, mask2, pend, fix, ctl, fix_cap, rec, wt, lut, gtab,
                               ptab, pmax, smax, tick, dopamine,
                               eval[min(i0 + grp, end - 1u)], i0 + grp < end, s_lit, lit_on, kc);
    } else {
      if (blockIdx.x == 0 && threadIdx.x == 0) ctl->ctr[6] += 1;   // ticks on the lit-sum form
      for (uint32_t i0 = beg; i0 < end; i0 += step)
        lit_row_step<false, WT>(P, A, rt, rw, cnt, mask2, pend, fix, ctl, fix_cap, rec, wt, lut, gtab,
                                ptab, pmax, smax, tick, dopamine,
                                eval[min(i0 + grp, end - 1u)], i0 + grp < end, nullptr, false, kc);
      lit_tested = kc.tested;
    }
    ev_slots = kc.ev_slots;
    hits = kc.hits;
    nspk = kc.nspk;
    gdone = kc.gdone;
    nev = kc.nev;
    err |= kc.err;
    same = kc.same;
  }
  for (uint32_t base = beg; form == kFormDense && base < end; base += 8u * step) {
    const uint32_t at = base + (lane >> 2) * step + (lane & 3u);   // eight steps' neurons, one a lane
    const uint32_t mine = at < end ? eval[at] : 0u;
    for (uint32_t sub = 0; sub < 8 && base + sub * step < end; sub++) {
      const bool valid = base + sub * step + grp < end;
      const uint32_t n = __shfl_sync(kFull, mine, 4u * sub + grp);
      // every load of the neuron at once: state, count, and its row up to smax
      const uint8_t flags = P.soma_flags[n];
      const uint32_t cw = valid ? cnt[n] : 0u;
      const uint32_t lf = lfz[n];
      const int32_t thr0 = P.threshold_offset[n];
      const int32_t v0 = P.soma_voltage[n];
      const uint32_t* rt_n = rt + (size_t)n * kRowStride;
      int16_t* rw_n = rw + (size_t)n * kRowStride;
      uint4 T[4];
      uint2 W[4];
      row_load(T, W, rt_n, rw_n, g8, valid, sh, smax);
      const uint32_t c = cw & 0xFFu;
      const uint32_t var = flags >> 4;
      const VariantParameters& p = lut[var];
      const uint32_t prop = p.signal_propagation_length;
      const bool exact = prop == pmax;
      const bool gfast = exact && prop <= 16u;
      if (cw & kRowBad) err |= AXC_ERR_TARGET_RANGE;
      uint32_t hitb, slowb;
      // the fully-lit test reads the bitmap from shared memory (LIT) or, when it
      // did not fit there, from global memory (1 bit per axon: far fewer bytes
      // to keep in L1/L2 than the 8-byte masks)
      int32_t i_in = row_slots<true>(T, W, c, g8, sh, mask2, s_lit, seg_hi, exact, gfast, prop,
                                     P.axon_heads, A, hitb, slowb, lit_on);
      i_in = wadd(i_in, __shfl_xor_sync(kFull, i_in, 1));
      i_in = wadd(i_in, __shfl_xor_sync(kFull, i_in, 2));
      i_in = wadd(i_in, __shfl_xor_sync(kFull, i_in, 4));
      if (g8 == 0 && valid) { ev_slots += c; nev++; }
      hits += __popc(hitb);
      // GLIF (physics.cu:209-275); the neuron is not refractory
      int spike = 0;
      if (valid) {
        const GlifOut o = glif_step(p, v0, thr0, i_in, tick, n);
        spike = o.spike;
        if (g8 == 0) {
          P.soma_voltage[n] = o.v;
          P.soma_flags[n] = (uint8_t)((flags & 0xF0) | (spike ? 0x05 : 0x00));
          P.threshold_offset[n] = o.thr;
          P.timers[n] = o.glif ? p.refractory_period : 0;
          if (spike) {
            nspk++;
            const uint32_t my_axon = P.soma_to_axon[n];
            if (my_axon != AXC_NO_AXON) {
              if (my_axon < A) atomicAdd(&pend[my_axon], 1u);
              else err |= AXC_ERR_SOMA_AXON;
            }
          }
        }
      }
      // GSOP (physics.cu:281-373) of the spiker's movable slots, the first lf
      // of its row; frozen slots (GSOP leaves them as they are) are counted
      if (spike && lf > 0u)
        gdone += row_gsop<WT>(W, hitb, slowb, lf, g8, sh, gtab, var, rt_n, rw_n, P.axon_heads, mask2, A, p, flags,
                              dopamine, ctl, fix, fix_cap, n, same, wt);
      if (spike && g8 == 0) gdone += c - lf;
    }
  }
  if (!lit_on) err |= AXC_ERR_WAIT_LIMIT;
  const uint32_t err_any = __reduce_or_sync(kFull, err);
  if (err_any && lane == 0) atomicOr(&ctl->err, err_any);
  counts[0] = ev_slots;
  counts[1] = hits;
  counts[2] = nspk;
  counts[3] = gdone;
  counts[4] = nev;
  counts[5] = lit_tested;
  counts[6] = same & 0xFFFFu;
  counts[7] = same >> 16;
}

// LIT: 1024-thread blocks (one per SM) that first copy the prologue's
// fully-lit bitmap into shared memory.
template <bool LIT, bool WT>
__global__ void __launch_bounds__(LIT ? 1024 : 256, LIT ? 1 : 4)
    k_rows_update(ShardVramPtrs P, uint32_t A, const uint32_t* __restrict__ rt, int16_t* __restrict__ rw,
                  const uint16_t* __restrict__ cnt, const uint2* __restrict__ mask2, const uint32_t* __restrict__ eval,
                  uint32_t* __restrict__ pend, uint32_t* __restrict__ fix, ShardCtl* __restrict__ ctl, uint32_t k,
                  uint32_t fix_cap, const uint32_t* __restrict__ lit_bits, const LearnCtl* __restrict__ lc,
                  const uint8_t* __restrict__ lfz, ColWT wt, uint32_t index, const int2* __restrict__ rec,
                  uint32_t unit) {
  __shared__ VariantParameters lut[16];
  __shared__ int2 gtab[16][16];
  __shared__ uint32_t ptab[16][17];
  __shared__ uint32_t s_pmax;
  __shared__ uint64_t s_bar;
  extern __shared__ __align__(128) uint32_t s_lit[];
  chain_wait();
  chain_open();
  const PassCtl pc = pass_ctl(ctl, k);
  const uint32_t ecount = ctl_ld32(&ctl->eval_act[k & 1][0]);
  const TickForm form = tick_form(ctl, k, A, lc, index);
  // else k_rows_update_lsum or the learned engine's kernels run this tick
  if (form != kFormDense && form != kFormLitRows && form != kFormVerify) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) count_form(ctl, form);
  if (LIT && threadIdx.x == 0) mbar_init(&s_bar, 1);
  lut_to_smem(lut);
  __syncthreads();
  // the fully-lit bitmap: one bulk copy into shared memory
  if (LIT && threadIdx.x == 0) bulk_to_smem(s_lit, lit_bits, lit_smem_bytes(A), &s_bar);
  const int32_t dopamine = (int32_t)(int16_t)ctl->dopamine;
  pmax_of(&s_pmax, lut);
  build_gtab(gtab, lut, dopamine);
  __syncthreads();
  const bool packed = form != kFormDense && build_ptab(ptab, gtab);
  const bool lit_on = !LIT || mbar_wait_bounded(&s_bar, 0, g_first_wait_limit);
  uint32_t counts[8];
  // An equal, contiguous part of the list per block, a multiple of `unit` neurons: 4
  // where the shard has the GPU to itself (6,000 plastic neurons, 1,500 of them
  // evaluated, sat on 12 SMs), else whole steps of the block, so that fewer blocks
  // stand in the way of the other shards' (four zone shards of 100,000: 2,160 us per
  // 20 ticks against 2,450).  The neighbours in a part, whose targets are near each
  // other, share an L1.
  const uint32_t part = ((ecount + gridDim.x - 1) / gridDim.x + unit - 1u) / unit * unit;
  const uint32_t first = min(blockIdx.x * part, ecount);
  rows_update<WT>(form, threadIdx.x >> 5, blockDim.x >> 5, pc, P, A, rt, rw, cnt, mask2, eval + first,
                  min(part, ecount - first), pend, fix, ctl, fix_cap, lfz, wt, rec, lut, gtab, packed ? ptab : nullptr,
                  s_pmax, dopamine, LIT ? s_lit : lit_bits, lit_on, counts);
  block_counts(counts, ctl->ctr, ctl->gsop_same);
  // a wait that gave up: the copy must land before the block exits
  if (LIT && !lit_on && !mbar_wait_bounded(&s_bar, 0)) atomicOr(&ctl->err, AXC_ERR_WAIT_LIMIT);
}

// ---------------------------------------------------------------------------
// Sparse form of a tick (tick_form: few axons carry a head on the segments the
// batch's slots use).  The dendrite sum is a wrapping i32 sum, so it may be
// taken from the axons' side in any order:
//   k_sparse_hits    a warp per 64 axons: for every
//                    run of hit segments of an active axon, the entries of the
//                    inverted index (RowIndex: one segment's together) are
//                    spread over the lanes; each adds its slot's weight into
//                    the neuron's acc with an integer atomic
//   k_sparse_neurons GLIF from acc, GSOP of the spikers' movable slots
// At 1.5M quiet neurons (12 % of the axons active, 1 % of the slots hit) the
// dense pass spends its 719 us a tick on 150M mask gathers; the sparse form
// touches the 1.5M hits.
// ---------------------------------------------------------------------------
constexpr uint32_t kSegUnsorted = 0xFFFFu;
constexpr int kHitUnroll = 4;

// The lane that owns item `it` of a warp whose lanes hold consecutive ranges of
// items: the first whose inclusive prefix sum incl exceeds it (31 past the end).
__device__ __forceinline__ uint32_t lane_of_item(uint32_t incl, uint32_t it) {
  uint32_t owner = 0;
#pragma unroll
  for (int stp = 16; stp > 0; stp >>= 1) {
    const uint32_t v = __shfl_sync(kFull, incl, owner + stp - 1);
    if (v <= it) owner += stp;
  }
  return min(owner, 31u);
}

__device__ __forceinline__ uint32_t warp_incl(uint32_t x) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  return x;
}

__global__ void __launch_bounds__(256, 6)
    k_sparse_hits(ShardVramPtrs P, uint32_t A, const uint32_t* __restrict__ rt, const int16_t* __restrict__ rw,
                  const uint2* __restrict__ mask2, const uint32_t* __restrict__ live, const uint32_t* __restrict__ evb,
                  int32_t* __restrict__ acc, ShardCtl* __restrict__ ctl, uint32_t k, const LearnCtl* __restrict__ lc) {
  if (tick_form(ctl, k, A, lc, 1u) != kFormSparse) return;
  const uint32_t* __restrict__ off = ctl->ix_off;
  const uint16_t* __restrict__ seg = ctl->ix_seg;
  const uint32_t* __restrict__ ent = ctl->ix_ent;
  const bool mixed = ctl->mixed_len != 0u;
  const uint32_t pmax = ctl->pmax, seg_max = ctl->seg_max;
  const uint32_t act = seg_max >= 31u ? 0xFFFFFFFFu : ((2u << seg_max) - 1u);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t groups = (A + 63) / 64;
  uint32_t hits = 0;
  for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < groups; g += nwarps) {
    const uint32_t a0 = 64u * g + 2u * lane;   // this lane's two axons
    const uint32_t lw = live[2u * g + (lane >> 4)] >> (2u * (lane & 15u));
    const bool on0 = (lw & 1u) && a0 < A, on1 = (lw & 2u) && a0 + 1u < A;
    uint32_t h0 = 0, h1 = 0;   // hit segments not taken yet (bit 31: "may hit", segments >= 31)
    if (on0) { const uint2 m = __ldg(mask2 + a0); h0 = (m.x | (m.y & 0x7FFFFFFFu)) & act; }
    if (on1) { const uint2 m = __ldg(mask2 + a0 + 1u); h1 = (m.x | (m.y & 0x7FFFFFFFu)) & act; }
    uint32_t o0 = 0, o1 = 0, d0 = 0, d1 = 0;   // first entry and entries of the axon
    if (on0) { o0 = __ldg(off + a0); d0 = __ldg(off + a0 + 1u) - o0; }
    if (on1) { o1 = __ldg(off + a0 + 1u); d1 = __ldg(off + a0 + 2u) - o1; }
    while (__any_sync(kFull, h0 | h1)) {
      // each lane's lowest run of hit segments [s0, s1]
      uint32_t first = 0, count = 0, ax = a0;
      bool test = false;   // the entries' segments are not known to be hit
      if (h0 | h1) {
        const bool second = h0 == 0u;
        uint32_t h = second ? h1 : h0;
        ax = a0 + (second ? 1u : 0u);
        const uint32_t o = second ? o1 : o0, d = second ? d1 : d0;
        const uint16_t* sg = seg + (size_t)ax * 32u;
        if (__ldg(sg) == kSegUnsorted) {
          first = o;
          count = d;
          test = true;
          h = 0;
        } else {
          const uint32_t s0 = (uint32_t)__ffs(h) - 1u;
          const uint32_t run = h >> s0;
          // segment 31's bucket ("may hit") is taken alone: its entries are tested
          const uint32_t len = s0 == 31u ? 1u : min((uint32_t)__ffs(~run) - 1u, 31u - s0);
          const uint32_t s1 = s0 + len;   // one past the run
          const uint32_t e0 = __ldg(sg + s0), e1 = s1 < 32u ? (uint32_t)__ldg(sg + s1) : d;
          first = o + e0;
          count = e1 - e0;
          test = s0 == 31u;
          h &= s1 < 32u ? (0xFFFFFFFFu << s1) : 0u;
        }
        if (second) h1 = h; else h0 = h;
      }
      const uint32_t incl = warp_incl(count);
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      const uint32_t base = first - (incl - count);
      const bool any_test = mixed || __any_sync(kFull, test);
      // 32 x kHitUnroll entries a step: every load of a step is issued before
      // anything waits (entry -> weight is a chain of two cache misses)
      for (uint32_t it0 = 0; it0 < total; it0 += 32u * kHitUnroll) {
        uint32_t r[kHitUnroll], own[kHitUnroll];
#pragma unroll
        for (int u = 0; u < kHitUnroll; u++) {
          const uint32_t it = it0 + 32u * u + lane;
          own[u] = lane_of_item(incl, it);
          const uint32_t b = __shfl_sync(kFull, base, own[u]);
          r[u] = it < total ? __ldg(ent + b + it) : 0xFFFFFFFFu;
        }
        int32_t w[kHitUnroll];
        bool on[kHitUnroll];
#pragma unroll
        for (int u = 0; u < kHitUnroll; u++) {
          w[u] = 0;
          on[u] = false;
          if (r[u] != 0xFFFFFFFFu) {
            const uint32_t n = r[u] / kRowStride;
            w[u] = rw[r[u]];
            on[u] = (__ldg(evb + (n >> 5)) >> (n & 31u)) & 1u;   // else refractory
          }
        }
#pragma unroll
        for (int u = 0; u < kHitUnroll; u++) {
          if (any_test) {   // warp-uniform
            const uint32_t a = __shfl_sync(kFull, ax, own[u]);
            const bool tst = __shfl_sync(kFull, test ? 1u : 0u, own[u]) != 0u;
            if (on[u] && (tst || mixed)) {
              const uint32_t prop = VARIANT_LUT[P.soma_flags[r[u] / kRowStride] >> 4].signal_propagation_length;
              if (tst || prop != pmax)
                on[u] = hit_exact(P.axon_heads, A, a, rt[r[u]] >> AXC_TARGET_SEG_SHIFT, prop);
            }
          }
          if (on[u]) {
            atomicAdd(acc + r[u] / kRowStride, w[u]);
            hits++;
          }
        }
      }
    }
  }
  const uint32_t counts[6] = {0, hits, 0, 0, 0, 0};
  block_counts(counts, ctl->ctr);
}

// ---------------------------------------------------------------------------
// The sparse form's neurons: a warp per 128 consecutive ones, a lane for four
// (16-byte loads of voltage, threshold and acc; which are evaluated comes from
// the prologue's bits, so no list is read: nearly all are).  GLIF from acc
// (physics.cu:209-275), then GSOP of the spikers' movable slots
// (physics.cu:281-373) from the gtab deltas, on the exact path or deferred to
// the fix-up stage, spread over the warp's lanes.  14 us at 393k neurons in a
// quiet brain.
// ---------------------------------------------------------------------------
constexpr int kNeuronBlocks = 5;   // resident 256-thread blocks per SM (48 registers a thread)

// Item `it` of the warp's rows: its neuron (of the warp's 128), row position q
// and the neuron's flags; incl: the lanes' inclusive item counts, per: a lane's
// four counts, a byte each.
__device__ __forceinline__ uint32_t row_item(uint32_t incl, uint32_t per, uint32_t fl4, uint32_t it, uint32_t* q,
                                             uint8_t* flags) {
  const uint32_t own = lane_of_item(incl, it);
  const uint32_t c = __shfl_sync(kFull, per, own), f = __shfl_sync(kFull, fl4, own);
  const uint32_t lane_end = __shfl_sync(kFull, incl, own);
  const uint32_t c0 = c & 0xFFu, c1 = c0 + ((c >> 8) & 0xFFu), c2 = c1 + ((c >> 16) & 0xFFu), c3 = c2 + (c >> 24);
  const uint32_t x = it - (lane_end - c3);
  const uint32_t j = (x >= c0 ? 1u : 0u) + (x >= c1 ? 1u : 0u) + (x >= c2 ? 1u : 0u);
  *q = x - (j == 0u ? 0u : j == 1u ? c0 : j == 2u ? c1 : c2);
  *flags = (uint8_t)(f >> (8u * j));
  return 4u * own + j;
}

__global__ void __launch_bounds__(256, kNeuronBlocks)
    k_sparse_neurons(ShardVramPtrs P, uint32_t N, uint32_t A, const uint32_t* __restrict__ rt, int16_t* __restrict__ rw,
                     const uint16_t* __restrict__ cnt, const uint8_t* __restrict__ lfz,
                     const uint2* __restrict__ mask2, const uint32_t* __restrict__ evb, uint32_t* __restrict__ pend,
                     uint32_t* __restrict__ fix, ShardCtl* __restrict__ ctl, uint32_t k, uint32_t fix_cap,
                     const uint32_t* __restrict__ lit_bits, const LearnCtl* __restrict__ lc,
                     int32_t* __restrict__ acc) {
  if (tick_form(ctl, k, A, lc, 1u) != kFormSparse) return;
  const uint32_t tiles = (N + 127u) / 128u;
  if (blockIdx.x * 8u >= tiles) return;   // no neuron for this block: no table to build
  if (blockIdx.x == 0 && threadIdx.x == 0) count_form(ctl, kFormSparse);
  __shared__ VariantParameters lut[16];
  __shared__ int2 gtab[16][16];
  lut_to_smem(lut);
  const uint32_t pmax = ctl->pmax;
  __syncthreads();
  const int32_t dopamine = (int32_t)(int16_t)ctl->dopamine;
  build_gtab(gtab, lut, dopamine);
  __syncthreads();
  const uint32_t tick = ctl->tick_base + k;
  const uint32_t seg_hi = min(ctl->seg_max, 30u);
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // 16-byte loads where the shard's arrays allow (padded_n a multiple of 16 puts
  // them on 16-byte boundaries of an aligned blob); else a load a neuron
  const bool vec = ((reinterpret_cast<uintptr_t>(P.soma_voltage) | reinterpret_cast<uintptr_t>(P.threshold_offset)) &
                    15u) == 0u &&
                   (reinterpret_cast<uintptr_t>(P.soma_flags) & 3u) == 0u;
  uint32_t ev_slots = 0, nspk = 0, gdone = 0, nev = 0, err = 0;
  for (uint32_t tile = blockIdx.x * 8u + wid; tile < tiles; tile += gridDim.x * 8u) {
    const uint32_t n0 = tile * 128u, nb = n0 + 4u * lane;
    const uint32_t ev = nb < N ? (evb[nb >> 5] >> (nb & 31u)) & 15u : 0u;
    const bool full = vec && nb + 4u <= N;
    int32_t v[4] = {0, 0, 0, 0}, thr[4] = {0, 0, 0, 0}, cur[4] = {0, 0, 0, 0};
    uint32_t cw[4] = {0, 0, 0, 0}, fl4 = 0;
    uint32_t moves = 0;   // movable slots of the spikers, a byte each
    if (ev) {
      if (full) {
        const int4 a = *reinterpret_cast<const int4*>(P.soma_voltage + nb);
        const int4 b = *reinterpret_cast<const int4*>(P.threshold_offset + nb);
        const int4 c = *reinterpret_cast<const int4*>(acc + nb);
        const uint2 d = __ldg(reinterpret_cast<const uint2*>(cnt + nb));
        fl4 = *reinterpret_cast<const uint32_t*>(P.soma_flags + nb);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        thr[0] = b.x; thr[1] = b.y; thr[2] = b.z; thr[3] = b.w;
        cur[0] = c.x; cur[1] = c.y; cur[2] = c.z; cur[3] = c.w;
        cw[0] = d.x & 0xFFFFu; cw[1] = d.x >> 16; cw[2] = d.y & 0xFFFFu; cw[3] = d.y >> 16;
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t n = nb + j;
          if (n >= N) continue;
          v[j] = P.soma_voltage[n];
          thr[j] = P.threshold_offset[n];
          fl4 |= (uint32_t)P.soma_flags[n] << (8 * j);
          cw[j] = cnt[n];
          cur[j] = acc[n];
        }
      }
      uint32_t nf = fl4;
      bool vch = false, tch = false;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (!((ev >> j) & 1u)) continue;
        const uint32_t n = nb + j, flags = (fl4 >> (8 * j)) & 0xFFu, c = cw[j] & 0xFFu;
        const VariantParameters& p = lut[flags >> 4];
        const GlifOut o = glif_step(p, v[j], thr[j], cur[j], tick, n);
        vch |= o.v != v[j];
        tch |= o.thr != thr[j];
        v[j] = o.v;
        thr[j] = o.thr;
        nf = (nf & ~(0xFFu << (8 * j))) | (((flags & 0xF0u) | (o.spike ? 0x05u : 0u)) << (8 * j));
        if (o.glif) P.timers[n] = p.refractory_period;   // an evaluated neuron's timer is 0
        ev_slots += c;
        nev++;
        if (cw[j] & kRowBad) err |= AXC_ERR_TARGET_RANGE;
        if (o.spike) {
          const uint32_t lf = lfz[n], a = P.soma_to_axon[n];
          nspk++;
          gdone += c - lf;   // frozen slots: GSOP leaves them as they are
          moves |= lf << (8 * j);
          if (a < A) atomicAdd(&pend[a], 1u);
          else if (a != AXC_NO_AXON) err |= AXC_ERR_SOMA_AXON;
        }
      }
      if (full) {
        if (vch) *reinterpret_cast<int4*>(P.soma_voltage + nb) = make_int4(v[0], v[1], v[2], v[3]);
        if (tch) *reinterpret_cast<int4*>(P.threshold_offset + nb) = make_int4(thr[0], thr[1], thr[2], thr[3]);
        if (nf != fl4) *reinterpret_cast<uint32_t*>(P.soma_flags + nb) = nf;
        if (cur[0] | cur[1] | cur[2] | cur[3]) *reinterpret_cast<int4*>(acc + nb) = make_int4(0, 0, 0, 0);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          if (!((ev >> j) & 1u)) continue;
          P.soma_voltage[nb + j] = v[j];
          P.threshold_offset[nb + j] = thr[j];
          P.soma_flags[nb + j] = (uint8_t)(nf >> (8 * j));
          acc[nb + j] = 0;
        }
      }
    }
    // GSOP of the spikers' movable slots
    const uint32_t msum = (moves & 0xFFu) + ((moves >> 8) & 0xFFu) + ((moves >> 16) & 0xFFu) + (moves >> 24);
    if (__any_sync(kFull, msum)) {
      const uint32_t incl = warp_incl(msum);
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      for (uint32_t it0 = 0; it0 < total; it0 += 32) {
        const uint32_t it = it0 + lane;
        uint32_t q;
        uint8_t f;
        const uint32_t i = row_item(incl, moves, fl4, it, &q, &f);
        if (it >= total) continue;
        const uint32_t n = n0 + i;
        const uint32_t* t = rt + (size_t)n * kRowStride + q;
        int16_t* w = rw + (size_t)n * kRowStride + q;
        const int16_t w16 = *w;
        const VariantParameters& p = lut[f >> 4];
        const uint32_t prop = p.signal_propagation_length;
        const bool exact = prop == pmax;
        bool fast;
        const bool hit = slot_hit(__ldg(t), exact, exact && prop <= 16u, prop, seg_hi, lit_bits, mask2, P.axon_heads, A,
                                  &fast);
        gdone += gsop_slot<false>(w16, t, w, hit, fast, gtab[f >> 4], P.axon_heads, mask2, A, p, f, dopamine, ctl, fix,
                                  fix_cap, n, q, ColWT{});
      }
    }
  }
  const uint32_t err_any = __reduce_or_sync(kFull, err);
  if (err_any && lane == 0) atomicOr(&ctl->err, err_any);
  const uint32_t counts[6] = {ev_slots, 0, nspk, gdone, nev, 0};
  block_counts(counts, ctl->ctr);
}

// ---------------------------------------------------------------------------
// per tick 2/4, lit-sum form (tick_form: few tested slots, and every axon the row
// layout took as fully lit is fully lit).  An evaluated neuron's input current is
// the row's lit-sum (frozen slots on fully-lit axons with segments 1..30: hits
// whatever the tick, their weights summed once per layout; the dendrite sum is a
// wrapping i32 sum, so the order cannot change a bit), plus the weights of its
// movable lit slots (hits too), plus the hits among its tested slots, tested as
// the 8-lane pass tests them (physics.cu:182-206); GLIF (physics.cu:209-275);
// then GSOP of a spiker's movable slots (physics.cu:281-373): the lit ones take
// their rank's potentiation, the tested ones the gtab deltas, the exact path or
// the fix-up stage.  No target of a lit slot is read.
// A thread per neuron, where few slots need work (a settled brain: 0.5 a
// neuron); where many do (lit_rows) k_rows_update takes 8 lanes a neuron.
// WT: weight changes written through to the columnar blob (per-tick entry point).
// ---------------------------------------------------------------------------
constexpr int kLsumBlocks = 5;   // resident 256-thread blocks per SM (48 registers a thread)

template <bool WT>
__global__ void __launch_bounds__(256, kLsumBlocks)
    k_rows_update_lsum(ShardVramPtrs P, uint32_t A, const uint32_t* __restrict__ rt, int16_t* __restrict__ rw,
                       const uint16_t* __restrict__ cnt, const uint2* __restrict__ mask2,
                       const uint32_t* __restrict__ eval, uint32_t* __restrict__ pend, uint32_t* __restrict__ fix,
                       ShardCtl* __restrict__ ctl, uint32_t k, uint32_t fix_cap, const uint32_t* __restrict__ lit_bits,
                       const int2* __restrict__ rec, ColWT wt, const LearnCtl* __restrict__ lc, uint32_t unit) {
  chain_wait();
  chain_open();
  const PassCtl pc = pass_ctl(ctl, k);
  const uint32_t ecount = ctl_ld32(&ctl->eval_act[k & 1][0]);
  if (tick_form(ctl, k, A, lc, 0u) != kFormLitSum) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->ctr[6] += 1;   // ticks on the lit-sum form
    count_form(ctl, kFormLitSum);
  }
  // neurons per block and pass: fewer than its threads where that spreads a short list over all blocks
  const uint32_t span = min(256u, ((ecount + gridDim.x - 1) / gridDim.x + unit - 1u) / unit * unit);
  if (blockIdx.x * span >= ecount) return;   // no neuron for this block: no table to build
  __shared__ VariantParameters lut[16];
  __shared__ int2 gtab[16][16];
  __shared__ uint32_t s_pmax;
  lut_to_smem(lut);
  __syncthreads();
  const int32_t dopamine = (int32_t)(int16_t)ctl->dopamine;
  pmax_of(&s_pmax, lut);
  build_gtab(gtab, lut, dopamine);
  __syncthreads();
  const uint32_t tick = pc.tick, seg_hi = min(pc.seg_max, 30u), pmax = s_pmax;
  LsumCount kc = {0, 0, 0, 0, 0, 0, 0, 0};
  for (uint32_t i = threadIdx.x < span ? blockIdx.x * span + threadIdx.x : ecount; i < ecount; i += gridDim.x * span) {
    const uint32_t n = eval[i];
    // every load of the neuron at once
    const uint8_t flags = P.soma_flags[n];
    const uint32_t cw = cnt[n];
    const int2 ls = rec[n];
    const int32_t thr0 = P.threshold_offset[n];
    const int32_t v0 = P.soma_voltage[n];
    const uint32_t my_axon = P.soma_to_axon[n];
    const uint32_t c = cw & 0xFFu, y = (uint32_t)ls.y;
    const uint32_t lm = y & 0xFFu, lf = (y >> 8) & 0xFFu, end = (y >> 16) & 0xFFu;
    const uint32_t var = flags >> 4;
    const VariantParameters& p = lut[var];
    const uint32_t prop = p.signal_propagation_length;
    const bool exact = prop == pmax;
    const bool gfast = exact && prop <= 16u;
    if (cw & kRowBad) kc.err |= AXC_ERR_TARGET_RANGE;
    const uint32_t* rt_n = rt + (size_t)n * kRowStride;
    int16_t* rw_n = rw + (size_t)n * kRowStride;
    int32_t i_in = ls.x;
    uint32_t h = c - end;   // the lit-sum slots are hits
    // the tests of row positions 0..31 (the movable slots come first), kept for GSOP
    uint32_t hit_bits = 0, fast_bits = 0;
    for (uint32_t q = 0; q < end; q += 4) {
      const uint4 T4 = *reinterpret_cast<const uint4*>(rt_n + q);
      const uint2 W4 = *reinterpret_cast<const uint2*>(rw_n + q);
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (q + j >= end) break;
        bool fast = true, hit = true;   // movable and lit
        if (q + j >= lm)
          hit = slot_hit(word_of(T4, j), exact, gfast, prop, seg_hi, lit_bits, mask2, P.axon_heads, A, &fast);
        if (hit) {
          i_in = wadd(i_in, (int32_t)half_of(W4, j));
          h++;
        }
        const uint32_t bit = (q + j < 32u) ? (1u << (q + j)) : 0u;
        hit_bits |= hit ? bit : 0u;
        fast_bits |= fast ? bit : 0u;
      }
    }
    kc.ev_slots += c;
    kc.hits += h;
    kc.tested += end - lm;
    kc.nev++;
    const GlifOut o = glif_step(p, v0, thr0, i_in, tick, n);
    neuron_store(P, n, o, flags, p, my_axon, A, pend, kc);
    if (!o.spike) continue;
    // GSOP (physics.cu:281-373) of the movable slots; the frozen ones are left as they are
    kc.gdone += c - lf;
    for (uint32_t q = 0; q < lf; q++) {
      const int16_t w16 = rw_n[q];
      bool fast = true, hit = true;
      if (q < 32u) {   // tested in the loop above (lf <= end)
        hit = (hit_bits >> q) & 1u;
        fast = (fast_bits >> q) & 1u;
      } else if (q >= lm) {
        hit = slot_hit(rt_n[q], exact, gfast, prop, seg_hi, lit_bits, mask2, P.axon_heads, A, &fast);
      }
      kc.gdone += gsop_slot<WT>(w16, rt_n + q, rw_n + q, hit, fast, gtab[var], P.axon_heads, mask2, A, p, flags,
                                dopamine, ctl, fix, fix_cap, n, q, wt);
    }
  }
  const uint32_t err_any = __reduce_or_sync(kFull, kc.err);
  if (err_any && (threadIdx.x & 31) == 0) atomicOr(&ctl->err, err_any);
  const uint32_t counts[6] = {kc.ev_slots, kc.hits, kc.nspk, kc.gdone, kc.nev, kc.tested};
  block_counts(counts, ctl->ctr);
}

// ---------------------------------------------------------------------------
// per tick 2b (learned engine): GSOP (physics.cu:281-373) of the listed
// spikers over the slots of amask only (the others are frozen: GSOP leaves
// them as they are), the (spiker, slot) items of 32 spikers spread over the
// warp's lanes.  Each slot is classified as in the update pass (fully lit,
// else the tick's hit masks; exact path for segments >= 31, other lengths,
// several owners, or a hit that one same-tick push could change) and updated
// from the gtab deltas, on the exact path, or deferred to the fix-up stage.
// Warp w of the listing pass listed its spikers at [beg_w, beg_w + wcnt[w]).
// ---------------------------------------------------------------------------
template <bool LIT>
__global__ void __launch_bounds__(256) k_rows_gsop(ShardVramPtrs P, uint32_t A, const uint32_t* __restrict__ rt,
                                                   int16_t* __restrict__ rw, const uint16_t* __restrict__ cnt,
                                                   const uint2* __restrict__ mask2, const uint32_t* __restrict__ lit_bits,
                                                   const uint4* __restrict__ amask, const uint32_t* __restrict__ gs_n,
                                                   const uint32_t* __restrict__ wcnt, uint32_t nwu,
                                                   uint32_t* __restrict__ fix, ShardCtl* __restrict__ ctl, uint32_t k,
                                                   uint32_t fix_cap, const LearnCtl* __restrict__ lc) {
  // the learned engine lists the spikers of its sparse ticks here; on its dense
  // ticks the update pass applied GSOP itself
  if (lc && tick_form(ctl, k, A, lc, 1u) != kFormScatter) return;
  __shared__ VariantParameters lut[16];
  __shared__ int2 gtab[16][16];
  __shared__ uint32_t s_pmax;
  lut_to_smem(lut);
  __syncthreads();
  const int32_t dopamine = (int32_t)(int16_t)ctl->dopamine;
  pmax_of(&s_pmax, lut);
  build_gtab(gtab, lut, dopamine);
  __syncthreads();
  const uint32_t ecount = ctl->eval_act[k & 1][0];
  const uint32_t per_warp = (((ecount + nwu - 1) / nwu) + 3) & ~3u;
  const uint32_t seg_hi = min(ctl->seg_max, 30u);
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t ngw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long gdone = 0;
  for (uint32_t uw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; uw < nwu; uw += ngw) {
    const uint32_t cntw = wcnt[uw];
    const uint32_t beg = min(uw * per_warp, ecount);
    for (uint32_t e0 = 0; e0 < cntw; e0 += 32) {
      // 32 listed spikers; their movable slots are spread over the lanes
      const bool has = e0 + lane < cntw;
      const uint32_t my_n = has ? gs_n[beg + e0 + lane] : 0u;
      const uint4 my_am = has ? amask[my_n] : make_uint4(0, 0, 0, 0);
      const uint32_t my_k = __popc(my_am.x) + __popc(my_am.y) + __popc(my_am.z) + __popc(my_am.w);
      uint32_t incl = my_k;   // inclusive prefix of the slot counts over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += x;
      }
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      for (uint32_t it0 = 0; it0 < total; it0 += 32) {   // warp-uniform: every lane takes part in the shuffles
        const uint32_t it = it0 + lane;
        // the lane that owns item it: the first whose inclusive prefix exceeds it
        uint32_t owner = 0;
#pragma unroll
        for (int stp = 16; stp > 0; stp >>= 1) {
          const uint32_t v = __shfl_sync(kFull, incl, owner + stp - 1);
          if (v <= it) owner += stp;
        }
        owner = min(owner, 31u);
        const uint32_t n = __shfl_sync(kFull, my_n, owner);
        const uint32_t prev = __shfl_sync(kFull, incl - my_k, owner);
        const uint32_t am0 = __shfl_sync(kFull, my_am.x, owner), am1 = __shfl_sync(kFull, my_am.y, owner);
        const uint32_t am2 = __shfl_sync(kFull, my_am.z, owner), am3 = __shfl_sync(kFull, my_am.w, owner);
        if (it >= total) continue;
        const uint32_t q = nth_bit128(make_uint4(am0, am1, am2, am3), it - prev);
        const uint8_t flags = P.soma_flags[n];
        const uint32_t var = flags >> 4;
        const VariantParameters& p = lut[var];
        const uint32_t prop = p.signal_propagation_length;
        const bool exact = prop == s_pmax;
        const bool gfast = exact && prop <= 16u;
        const size_t r = (size_t)n * kRowStride + q;
        const uint32_t t = __ldg(rt + r);
        const int16_t w16 = rw[r];
        const uint32_t ax = (t & AXC_TARGET_AXON_MASK) - 1u;
        const uint32_t s = t >> AXC_TARGET_SEG_SHIFT;
        bool hit, fast;
        if (LIT && gfast && (s - 1u) < seg_hi && ((__ldg(lit_bits + (ax >> 5)) >> (ax & 31u)) & 1u)) {
          hit = true;
          fast = true;
        } else {
          const uint2 m = __ldg(mask2 + ax);
          const uint32_t sh = min(s, 31u);
          const uint32_t bx = (m.x >> sh) & 1u, by = (m.y >> sh) & 1u;
          hit = (bx | by) != 0u;
          if (hit && (s >= 31u || !exact)) hit = hit_exact(P.axon_heads, A, ax, s, prop);
          fast = gfast && s < 31u && !(m.y >> 31) && (bx || by == (s == 0u));
        }
        int16_t nw = w16;
        if (fast) {
          const int32_t aw = w16 < 0 ? -(int32_t)w16 : (int32_t)w16;
          const int2 d = gtab[var][min((uint32_t)aw >> 11, 15u)];
          int32_t na = aw + (hit ? d.x : -d.y);
          na = min(max(na, 0), 32767);
          nw = (int16_t)(w16 < 0 ? -na : na);
          gdone++;
        } else {
          const int res = gsop_general(P.axon_heads, mask2, A, ax, s, p, flags, dopamine, &nw);
          if (res == 2) continue;
          gdone++;
          if (res == 1) {
            const uint32_t slot = atomicAdd(&ctl->fix_count, 1u);
            if (slot < fix_cap) fix[slot] = (uint32_t)r;
            else ctl->fix_overflow = 1u;
            continue;
          }
        }
        if (nw != w16) rw[r] = nw;
      }
    }
  }
  block_count(gdone, 0, 0, &ctl->ctr[4]);
}

// GSOP of the listed spikers with many slots that may move, 8 lanes per row
// as in the update pass (row_load / row_slots / row_gsop; frozen slots get a
// zero delta).  Warp w of the update pass listed them at [beg_w, beg_w + wcnt[w]).
template <bool LIT>
__global__ void __launch_bounds__(256) k_rows_gsop_rows(ShardVramPtrs P, uint32_t A, const uint32_t* __restrict__ rt,
                                                        int16_t* __restrict__ rw, const uint16_t* __restrict__ cnt,
                                                        const uint2* __restrict__ mask2,
                                                        const uint32_t* __restrict__ lit_bits,
                                                        const uint32_t* __restrict__ gd_n,
                                                        const uint32_t* __restrict__ wcnt, uint32_t nwu,
                                                        uint32_t* __restrict__ fix, ShardCtl* __restrict__ ctl,
                                                        uint32_t k, uint32_t fix_cap, const LearnCtl* __restrict__ lc) {
  if (lc && tick_form(ctl, k, A, lc, 1u) != kFormScatter) return;   // as k_rows_gsop
  __shared__ VariantParameters lut[16];
  __shared__ int2 gtab[16][16];
  __shared__ uint32_t s_pmax;
  lut_to_smem(lut);
  __syncthreads();
  const int32_t dopamine = (int32_t)(int16_t)ctl->dopamine;
  pmax_of(&s_pmax, lut);
  build_gtab(gtab, lut, dopamine);
  __syncthreads();
  const uint32_t ecount = ctl->eval_act[k & 1][0];
  const uint32_t per_warp = (((ecount + nwu - 1) / nwu) + 3) & ~3u;
  const uint32_t smax = ctl->row_smax;
  const RowShape sh = row_shape(smax);
  const uint32_t seg_hi = min(ctl->seg_max, 30u);
  const uint32_t lane = threadIdx.x & 31, g8 = lane & 7, grp = lane >> 3;
  const uint32_t ngw = (gridDim.x * blockDim.x) >> 5;
  unsigned long long gdone = 0;
  uint32_t same = 0;
  for (uint32_t uw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; uw < nwu; uw += ngw) {
    const uint32_t cntw = wcnt[uw];
    const uint32_t beg = min(uw * per_warp, ecount);
    for (uint32_t e = 0; e < cntw; e += 4) {
      const bool valid = e + grp < cntw;
      const uint32_t n = valid ? gd_n[beg + e + grp] : 0u;
      const uint8_t flags = P.soma_flags[n];
      const uint32_t c = valid ? (cnt[n] & 0xFFu) : 0u;
      const uint32_t var = flags >> 4;
      const VariantParameters& p = lut[var];
      const uint32_t prop = p.signal_propagation_length;
      const bool exact = prop == s_pmax;
      const bool gfast = exact && prop <= 16u;
      const uint32_t* rt_n = rt + (size_t)n * kRowStride;
      int16_t* rw_n = rw + (size_t)n * kRowStride;
      uint4 T[4];
      uint2 W[4];
      row_load(T, W, rt_n, rw_n, g8, valid, sh, smax);
      uint32_t hitb, slowb;
      (void)row_slots<LIT>(T, W, c, g8, sh, mask2, lit_bits, seg_hi, exact, gfast, prop, P.axon_heads, A, hitb,
                           slowb);
      if (valid)
        gdone += row_gsop(W, hitb, slowb, c, g8, sh, gtab, var, rt_n, rw_n, P.axon_heads, mask2, A, p, flags,
                          dopamine, ctl, fix, fix_cap, n, same);
    }
  }
  block_count(gdone, 0, 0, &ctl->ctr[4]);
}

// ---------------------------------------------------------------------------
// per tick 3/4: deferred GSOP slots, with the actual push count of the axon
// (pend, before the push stage consumes it) and the original weight.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void fixup_slot(const ShardVramPtrs& P, const VariantParameters* lut, uint32_t A,
                                           const uint32_t* rt, int16_t* rw, const uint32_t* pend,
                                           uint32_t r, int32_t dopamine, const ColWT& wt = ColWT{}) {
  const uint32_t n = r / kRowStride;
  const uint32_t t = rt[r];
  const uint32_t a = (t & AXC_TARGET_AXON_MASK) - 1u;
  const uint32_t s = t >> AXC_TARGET_SEG_SHIFT;
  const uint8_t flags = P.soma_flags[n];
  const VariantParameters& p = lut[flags >> 4];
  uint32_t h[8];
  load_heads(P.axon_heads, a, h);
  push_n(h, pend[a]);
  const uint32_t md = md_of(h, s, p.signal_propagation_length);
  const GsopConsts gc = gsop_consts(flags, p, dopamine);
  const int16_t w0 = rw[r];
  const int16_t w1 = gsop_weight(w0, md, p, gc.bm, gc.raw_pot, gc.final_dep);
  if (w1 != w0) {
    rw[r] = w1;
    if (wt.w) col_write(wt, n, r % kRowStride, w1);
  }
}

// Sparse-form ticks in a row before the index is asked for: building it costs
// what the dense pass loses to the sparse form in ~20 ticks (1.5M neurons).
constexpr uint32_t kIndexStreak = 16;
// Dense ticks in a row after which the gate's plain graphs go without the sparse form's
// kernels (two launches that return at once, 4 us of a saturated tick), longer than the
// bursts of a quiet brain: one whose bursts follow a cycle of 100 ticks lost 8 % when the
// graphs had them only while the last 16 ticks were quiet.
constexpr uint32_t kBusyStreak = 256;

// The next tick's lists (last used two ticks ago).
__device__ __forceinline__ void rows_next_lists(ShardCtl* ctl, uint32_t k) {
  ctl->eval_act[(k + 1) & 1][0] = ctl->eval_act[(k + 1) & 1][1] = 0;
  ctl->dense[(k + 1) & 1] = 0;
}

__device__ __forceinline__ void rows_fixup(const ShardVramPtrs& P, uint32_t N, uint32_t A, const uint32_t* rt,
                                           int16_t* rw, const uint16_t* cnt, const uint2* mask2, const uint32_t* pend,
                                           const uint32_t* eval, const uint32_t* fix, ShardCtl* ctl, uint32_t k,
                                           const uint32_t* ids, uint8_t* out, uint32_t num_outputs, const ColWT& wt,
                                           volatile uint32_t* wish) {
  const uint32_t nfix = ctl->fix_count;
  const uint32_t overflow = ctl->fix_overflow;
  {
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid == 0) {
      // ticks in a row that the sparse form would take: ask for its index
      if (wish) {
        // (the words are read at once: one after another they were the kernel's end)
        const unsigned long long p = ctl_ld64(&ctl->pfx_total), c = ctl_ld64(&ctl->slot_total);
        const uint32_t dark = ctl_ld32(&ctl->dense[k & 1]), was = ctl_ld32(&ctl->streak);
        const uint32_t busy0 = ctl_ld32(&ctl->busy), told = ctl_ld32(&ctl->busy_told);
        const uint32_t eval = ctl_ld32(&ctl->eval_act[k & 1][0]), act = ctl_ld32(&ctl->eval_act[k & 1][1]);
        const bool sparse = !(lit_layout(p, c) && dark == 0u) && sparse_tick(eval, act);
        const uint32_t streak = sparse ? was + 1u : 0u, busy = sparse ? 0u : min(busy0 + 1u, kBusyStreak);
        if (streak != was) ctl->streak = streak;
        if (busy != busy0) ctl->busy = busy;
        if (streak >= kIndexStreak && !index_built(ctl)) wish[0] = 1u;
        if ((busy == kBusyStreak) != (told != 0u)) wish[1] = ctl->busy_told = busy == kBusyStreak;
      }
    }
    // readout of the tick (physics.cu:378-395): flags are final once the update pass is done
    uint32_t err = 0;
    for (uint32_t j = tid; j < num_outputs; j += stride) {
      const uint32_t id = ids[j];
      uint8_t v = 0;
      if (id != AXC_NO_AXON) {
        if (id < N) v = P.soma_flags[id] & 0x01;
        else err = AXC_ERR_READOUT_RANGE;
      }
      out[j] = v;
    }
    if (err) atomicOr(&ctl->err, err);
  }
  if (nfix == 0 && !overflow) return;
  __shared__ VariantParameters lut[16];
  __shared__ uint32_t s_pmax;
  lut_to_smem(lut);
  if (threadIdx.x == 0) s_pmax = lut_pmax();
  __syncthreads();
  const int32_t dopamine = (int32_t)(int16_t)ctl->dopamine;
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (!overflow) {
    for (uint32_t i = tid; i < nfix; i += stride) fixup_slot(P, lut, A, rt, rw, pend, fix[i], dopamine, wt);
    return;
  }
  // the list overflowed: rescan every spiker's slots with the update pass's rule
  const uint32_t ecount = ctl->eval_act[k & 1][0];
  for (uint32_t w = tid; w < ecount * kRowStride; w += stride) {
    const uint32_t n = eval[w / kRowStride], q = w % kRowStride;
    if (!(P.soma_flags[n] & 1) || q >= (cnt[n] & 0xFFu)) continue;
    const uint32_t r = n * kRowStride + q;
    const uint32_t t = rt[r];
    const uint32_t a = (t & AXC_TARGET_AXON_MASK) - 1u;
    if (a >= A) continue;
    const uint32_t s = t >> AXC_TARGET_SEG_SHIFT;
    const VariantParameters& p = lut[P.soma_flags[n] >> 4];
    const uint32_t prop = p.signal_propagation_length;
    const bool gfast = prop == s_pmax && prop <= 16u;
    const uint2 m = mask2[a];
    const uint32_t sh = min(s, 31u);
    const uint32_t bx = (m.x >> sh) & 1u, by = (m.y >> sh) & 1u;
    const bool fast = gfast && s < 31u && !(m.y >> 31) && (bx || by == (s == 0u));
    if (fast) continue;
    uint32_t md0, md1;
    md_pair(P.axon_heads, a, s, prop, &md0, &md1);
    if ((m.y >> 31) || md0 != md1) fixup_slot(P, lut, A, rt, rw, pend, r, dopamine, wt);
  }
}

__global__ void __launch_bounds__(256) k_rows_fixup(ShardVramPtrs P, uint32_t N, uint32_t A,
                                                    const uint32_t* __restrict__ rt, int16_t* __restrict__ rw,
                                                    const uint16_t* __restrict__ cnt,
                                                    const uint2* __restrict__ mask2, const uint32_t* __restrict__ pend,
                                                    const uint32_t* __restrict__ eval,
                                                    const uint32_t* __restrict__ fix, ShardCtl* __restrict__ ctl,
                                                    uint32_t k, const uint32_t* __restrict__ ids,
                                                    uint8_t* __restrict__ out, uint32_t num_outputs, ColWT wt,
                                                    volatile uint32_t* wish) {
  chain_wait();
  chain_open();
  if (blockIdx.x == 0 && threadIdx.x == 0) rows_next_lists(ctl, k);
  rows_fixup(P, N, A, rt, rw, cnt, mask2, pend, eval, fix, ctl, k, ids, out, num_outputs, wt, wish);
}

// per tick 4/4, on a batch's (or learned graph's) last tick: the spikers'
// own-axon pushes (physics.cu:257-261), found in the evaluated list; on the
// other ticks the next prologue applies them.
__device__ __forceinline__ void rows_push(BurstHeads8* heads, const uint32_t* s2a, uint32_t A, uint32_t* pend,
                                          const uint32_t* eval, const uint8_t* flags, ShardCtl* ctl, uint32_t k) {
  const uint32_t ecount = ctl->eval_act[k & 1][0];
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid == 0) {
    rows_next_lists(ctl, k);
    ctl->fix_count = 0;
    ctl->fix_overflow = 0;
  }
  for (uint32_t i = tid; i < ecount; i += stride) {
    const uint32_t n = eval[i];
    if (!(flags[n] & 1)) continue;
    const uint32_t ax = s2a[n];
    if (ax >= A) continue;
    const uint32_t c = atomicExch(&pend[ax], 0u);
    if (!c) continue;
    uint4* p = reinterpret_cast<uint4*>(heads + ax);
    uint4 x = p[0], y = p[1];
    uint32_t h[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
    push_n(h, c);
    p[0] = make_uint4(h[0], h[1], h[2], h[3]);
    p[1] = make_uint4(h[4], h[5], h[6], h[7]);
  }
}

__global__ void __launch_bounds__(256) k_rows_push(BurstHeads8* __restrict__ heads, const uint32_t* __restrict__ s2a,
                                                   uint32_t A, uint32_t* __restrict__ pend,
                                                   const uint32_t* __restrict__ eval, const uint8_t* __restrict__ flags,
                                                   ShardCtl* __restrict__ ctl, uint32_t k) {
  chain_wait();
  chain_open();
  rows_push(heads, s2a, A, pend, eval, flags, ctl, k);
}

__global__ void k_rows_reset_lists(ShardCtl* ctl) {
  ctl->eval_act[0][0] = ctl->eval_act[0][1] = 0;
  ctl->eval_act[1][0] = ctl->eval_act[1][1] = 0;
  ctl->fix_count = 0;
  ctl->fix_overflow = 0;
  ctl->dense[0] = 0;
  ctl->dense[1] = 0;
}


// ---------------------------------------------------------------------------
// per tick 1/4 of the plain engine: k_rows_prologue without the learned
// engine's per-tile accounting, ITEMS axons and neurons per thread (items
// i0 + 256 r).  No barrier before the loads: every thread reads the batch
// constants (seg_max, the LUT's largest length, set at batch start) itself,
// next to its own loads.  The evaluated neurons are appended with one atomic
// per block.
// ---------------------------------------------------------------------------
// push_n for the common counts 0 and 1 without the general shift network
__device__ __forceinline__ void push_few(uint32_t h[8], uint32_t c) {
  if (c == 1u) {
#pragma unroll
    for (int q = 7; q > 0; q--) h[q] = h[q - 1];
    h[0] = 0u;
  } else if (c > 1u) {
    push_n(h, c);
  }
}

// INDEX: also the active axons' count and, where live is given, the live axons' and
// evaluated neurons' bits, for the sparse form (the learned engine's plain graph).
// The flags that a refractory neuron's tick clears (physics.cu:168-174): stored here,
// or with SMALL (one item) returned with bit 8 set for the caller to store; the listed
// neurons stay in s_list, their count and place in the tick's list in s_place.
template <int ITEMS, bool INDEX, int THREADS, bool SMALL>
__device__ __forceinline__ uint32_t rows_prologue(uint32_t i0, BurstHeads8* heads, uint32_t A, uint32_t v_seg,
                                                  const uint32_t* bitmask, uint32_t voff, uint32_t nv,
                                                  uint32_t* incoming, const uint32_t* batch_counts, uint32_t k,
                                                  uint2* mask2, const uint32_t* axw, uint8_t* flags, uint8_t* timers,
                                                  uint32_t N, uint32_t* eval, ShardCtl* ctl, uint32_t raise_err,
                                                  uint32_t* lit_bits, uint32_t* pend_apply, uint32_t inc_direct,
                                                  uint32_t set_tick, uint32_t tick_base, int32_t dopamine,
                                                  const uint32_t* xlit, uint32_t* live, uint32_t* evb, uint32_t* alit,
                                                  uint32_t alit_new, uint32_t* s_list, uint32_t* s_place) {
  __shared__ uint32_t s_base;
  __shared__ uint32_t s_warp[ITEMS][THREADS / 32];   // evaluated neurons | active axons << 16

  // all loads first: heads, owners, pending pushes, input bits, timers, constants,
  // and the axons the row layout took as fully lit (xlit, 32 per warp)
  uint4 hx[ITEMS], hy[ITEMS];
  uint32_t own[ITEMS], npush[ITEMS], xw[ITEMS];
  uint8_t tm[ITEMS], fl[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    const uint32_t i = i0 + (uint32_t)THREADS * r;
    npush[r] = 0;
    own[r] = 0;
    tm[r] = 0;
    fl[r] = 0;
    xw[r] = (xlit && i < A) ? __ldg(xlit + (i >> 5)) : 0u;
    if (i < A) {
      const uint4* p = reinterpret_cast<const uint4*>(heads + i);
      hx[r] = p[0];
      hy[r] = p[1];
      own[r] = __ldg(axw + i);
      if (pend_apply) npush[r] = pend_apply[i];   // the previous tick's soma pushes
      if (bitmask) {
        const uint32_t v = i - voff;
        if (v < nv) npush[r] += (__ldg(bitmask + (v >> 5)) >> (v & 31u)) & 1u;
      }
    }
    if (i < N) {
      tm[r] = timers[i];
      fl[r] = flags[i];
    }
  }
  const uint32_t seg_max = ctl->seg_max, pmax = ctl->pmax;
  // network pushes this tick: per-tick calls say so directly, batches by the tick's count
  const bool inc = inc_direct || (batch_counts && batch_counts[k] > 0);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->ctr[0] += 1;
    if (raise_err) atomicOr(&ctl->err, raise_err);
    ctl->fix_count = 0;      // the previous tick's fix-up is done
    ctl->fix_overflow = 0;
    if (set_tick) {          // per-tick calls: the tick number and dopamine the later stages read
      ctl->tick_base = tick_base;
      ctl->dopamine = dopamine;
    }
  }
  // segments the batch's slots use: 0..seg_max (bit 31: any segment >= 31)
  const uint32_t act = seg_max >= 31u ? 0xFFFFFFFFu : ((2u << seg_max) - 1u);
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t ebal[ITEMS], clear = 0;
#pragma unroll
  for (int r = 0; r < ITEMS; r++) {
    const uint32_t i = i0 + (uint32_t)THREADS * r;
    bool lit = false, on = false;
    if (i < A) {
      uint32_t c = npush[r];
      if (pend_apply && c) pend_apply[i] = 0;
      if (inc) {
        const uint32_t ci = incoming[i];
        if (ci) { c += ci; incoming[i] = 0; }
      }
      uint32_t h[8] = {hx[r].x, hx[r].y, hx[r].z, hx[r].w, hy[r].x, hy[r].y, hy[r].z, hy[r].w};
      push_few(h, c);
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (h[j] != AXC_AXON_SENTINEL) h[j] += v_seg;
      uint4* p = reinterpret_cast<uint4*>(heads + i);
      p[0] = make_uint4(h[0], h[1], h[2], h[3]);
      p[1] = make_uint4(h[4], h[5], h[6], h[7]);
      const uint2 m = split_masks(h, pmax, ax_owners(own[r]));
      mask2[i] = m;
      // fully lit: heads 0..6 hit every segment 1..30 the axon's slots use and at
      // most one soma owns the axon (for those segments the hit is 1 and one
      // push cannot change it)
      lit = (m.x & own[r] & kAxSegs) == (own[r] & kAxSegs) && !(m.y >> 31);
      if (INDEX) on = ((m.x | (m.y & 0x7FFFFFFFu)) & act) != 0u;
    }
    const uint32_t lb = __ballot_sync(kFull, lit), onb = INDEX ? __ballot_sync(kFull, on) : 0u;
    if (lane == 0 && i < A) {
      lit_bits[i >> 5] = lb;
      always_lit(alit + (i >> 5), lb, alit_new);
      if (INDEX && live) live[i >> 5] = onb;
      // an axon the row layout summed as fully lit is not: this tick takes the full pass
      if (xw[r] & ~lb) atomicAdd(&ctl->dense[k & 1], (uint32_t)__popc(xw[r] & ~lb));
    }
    bool ev = false;
    if (i < N) {
      if (tm[r] > 0) {                              // physics.cu:168-174 after the burst reset
        timers[i] = (uint8_t)(tm[r] - 1);
        if (fl[r] & 0x0Fu) {
          if (SMALL)
            clear = 0x100u | (fl[r] & 0xF0u);
          else
            flags[i] = fl[r] & 0xF0u;
        }
      } else {
        ev = true;
      }
    }
    ebal[r] = __ballot_sync(kFull, ev);
    if (lane == 0) {
      if (INDEX && live && i < N) evb[i >> 5] = ebal[r];
      s_warp[r][w] = __popc(ebal[r]) | (INDEX ? __popc(onb) << 16 : 0);
    }
  }
  __syncthreads();
  if (w == 0) {   // exclusive scan of the warps' counts, then the block's place in the list
    constexpr uint32_t E = ITEMS * (THREADS / 32), PER = (E + 31) / 32;
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
      c[q] = lane * PER + q < E ? (&s_warp[0][0])[lane * PER + q] : 0u;
      sum += c[q];
    }
    const uint32_t incl = warp_incl(sum);
    uint32_t run = incl - sum;
#pragma unroll
    for (uint32_t q = 0; q < PER; q++) {
      if (lane * PER + q < E) (&s_warp[0][0])[lane * PER + q] = INDEX ? run & 0xFFFFu : run;
      run += c[q];
    }
    if (lane == 31) {
      if (INDEX)
        s_base = append_count(ctl, k, incl & 0xFFFFu, incl >> 16);
      else if (SMALL)
        s_place[0] = incl;
      else
        s_base = incl ? atomicAdd(&ctl->eval_act[k & 1][0], incl) : 0u;
    }
  }
  __syncthreads();
  if (SMALL) {   // the block's own list; its place in the tick's list (for the fix-up and the push) arrives later
    if (w == 1 && lane == 0) s_place[1] = s_place[0] ? atomicAdd(&ctl->eval_act[k & 1][0], s_place[0]) : 0u;
    if ((ebal[0] >> lane) & 1u) s_list[s_warp[0][w] + __popc(ebal[0] & ((1u << lane) - 1u))] = i0;
    return clear;
  }
#pragma unroll
  for (int r = 0; r < ITEMS; r++)
    if ((ebal[r] >> lane) & 1u)
      eval[s_base + s_warp[r][w] + __popc(ebal[r] & ((1u << lane) - 1u))] = i0 + (uint32_t)THREADS * r;
  return clear;
}

template <int ITEMS, bool INDEX>
__global__ void __launch_bounds__(256) k_rows_prologue_plain(BurstHeads8* __restrict__ heads, uint32_t A,
                                                             uint32_t v_seg, const uint32_t* __restrict__ bitmask,
                                                             uint32_t voff, uint32_t nv,
                                                             uint32_t* __restrict__ incoming,
                                                             const uint32_t* __restrict__ batch_counts, uint32_t k,
                                                             uint2* __restrict__ mask2,
                                                             const uint32_t* __restrict__ axw,
                                                             uint8_t* __restrict__ flags,
                                                             uint8_t* __restrict__ timers, uint32_t N,
                                                             uint32_t* __restrict__ eval, ShardCtl* __restrict__ ctl,
                                                             uint32_t raise_err, uint32_t* __restrict__ lit_bits,
                                                             uint32_t* __restrict__ pend_apply, uint32_t inc_direct,
                                                             uint32_t set_tick, uint32_t tick_base, int32_t dopamine,
                                                             const uint32_t* __restrict__ xlit,
                                                             uint32_t* __restrict__ live,
                                                             uint32_t* __restrict__ evb, uint32_t* __restrict__ alit,
                                                             uint32_t alit_new) {
  chain_wait();
  chain_open();
  rows_prologue<ITEMS, INDEX, 256, false>(blockIdx.x * (256u * ITEMS) + threadIdx.x, heads, A, v_seg, bitmask, voff,
      nv, incoming, batch_counts, k, mask2, axw, flags, timers, N, eval, ctl, raise_err, lit_bits, pend_apply,
      inc_direct, set_tick, tick_base, dopamine, xlit, live, evb, alit, alit_new, nullptr, nullptr);
}
// Items (an axon and a neuron each) per thread of k_rows_prologue_plain: two
// halve the blocks, and with them the list-append atomics on one counter and
// the per-block barriers (1.5M neurons: 18,162 against 17,733 ticks/s; four
// are slower, 16,717), where the grid at one item has at least kProWide
// blocks (four waves of 8 blocks per SM on 152 SMs); a smaller brain keeps one
// item per thread and twice the blocks (16k neurons: 66,644 ticks/s with one
// item and 64 blocks, 60,629 with two and 32).
constexpr uint32_t kProWide = 4864;

// ---------------------------------------------------------------------------
// small brains: a batch's ticks (or a per-tick call) in one launch
// ---------------------------------------------------------------------------
// A tick of a small brain is launches and latency: four kernels of 2 to 8 us, most
// of it their start, their tables and one chain of dependent loads each.  Here the
// stages of all ticks run in one grid of resident blocks with two barriers a tick
// (a third where a GSOP slot was deferred or network spikes follow), the tables are
// built once, a block keeps the neurons it lists, and a graph has one node for its
// ticks.  16,384 neurons: 14.8 -> 9.6 us per tick of a batch; 2,048: 20.4 -> 18.8 us
// per call of the per-tick entry point.
struct SmallArgs {
  ShardVramPtrs P;
  uint32_t N, A, v_seg;
  const uint32_t* bitmask;   // words per tick; null without input
  uint32_t words, voff, nv, raise;
  const uint32_t* spikes;    // network spikes, spike_cap per tick; null without
  uint32_t spike_cap, spike_count;   // spike_count: without counts
  const uint32_t* counts;
  uint32_t* incoming;
  uint32_t *rt, *eval, *pend, *fix, *lit, *alit, *xlit;
  int16_t* rw;
  const uint16_t* cnt;
  const uint8_t* lfz;
  const int2* rec;
  const uint32_t* axw;
  uint2* mask2;
  ShardCtl* ctl;
  const uint32_t* ids;       // readout; outputs 0 without
  uint8_t* out;
  uint32_t outputs, fix_cap;
  uint32_t ticks, k0, lit_tick;   // lit_tick: the tick that starts alit anew, or ticks
  uint32_t set_tick, tick_base;   // set_tick: a per-tick call (tick_base, dopamine from here)
  int32_t dopamine;
  ColWT wt;
};

// Tries of a barrier of the resident grid: about 3 s (axc_row_engine_barrier_limit;
// tests set 0 to take the give-up path).
constexpr uint32_t kGridWaitLimit = 1u << 22;
__device__ uint32_t g_barrier_limit = kGridWaitLimit;

// All threads of the grid.  CLUSTER: the cluster's hardware barrier.  Else a counter
// that every block adds to (zeroed before each launch), with a bounded wait (tries):
// false once a block gave up, on which the grid's blocks all return.  The pushes that
// are then left in pend and incoming are dropped by the write-back behind (gave_up).
template <bool CLUSTER>
__device__ __forceinline__ bool small_barrier(ShardCtl* ctl, uint32_t& target, uint32_t tries, uint32_t* s_ok) {
  if (CLUSTER) {
    asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
    return true;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->barrier) : "memory");
    bool ok = false;
    for (uint32_t it = 0; it < tries && !ok; it++) {
      uint32_t seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&ctl->barrier) : "memory");
      ok = (int32_t)(seen - target) >= 0;
    }
    if (!ok) {
      atomicOr(&ctl->err, AXC_ERR_WAIT_LIMIT);
      ctl->gave_up = 1u;
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

__device__ __forceinline__ uint32_t small_spikes(const SmallArgs& b, uint32_t t) {
  if (!b.spikes) return 0u;
  return b.counts ? min(b.counts[t], b.spike_cap) : b.spike_count;
}

__device__ __forceinline__ void small_incoming(const SmallArgs& b, uint32_t t) {
  const uint32_t n = small_spikes(b, t);
  const uint32_t* ids = b.spikes + (size_t)t * b.spike_cap;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    if (ids[i] < b.A) atomicAdd(&b.incoming[ids[i]], 1u);
}

template <bool CLUSTER, bool WT>
__global__ void __launch_bounds__(1024, 1) k_rows_small(const __grid_constant__ SmallArgs b) {
  __shared__ VariantParameters lut[16];
  __shared__ int2 gtab[16][16];
  __shared__ uint32_t ptab[16][17];
  __shared__ uint32_t s_pmax, s_ok, s_place[2];
  __shared__ uint32_t s_list[1024];     // the block's evaluated neurons of the tick
  __shared__ uint32_t s_cnt[8][32];     // each warp's counts
  __shared__ uint64_t s_bar;
  extern __shared__ __align__(128) uint32_t s_lit[];
  ShardCtl* ctl = b.ctl;
  if (threadIdx.x == 0) mbar_init(&s_bar, 1);
  if (threadIdx.x < 256) (&s_cnt[0][0])[threadIdx.x] = 0;
  lut_to_smem(lut);
  __syncthreads();
  pmax_of(&s_pmax, lut);
  const int32_t dopamine = (int32_t)(int16_t)(b.set_tick ? b.dopamine : ctl->dopamine);
  build_gtab(gtab, lut, dopamine);
  __syncthreads();
  const bool packed = build_ptab(ptab, gtab);
  // axons and list entries go to the blocks warp by warp: few of them use every SM
  const uint32_t wid = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const uint32_t tries = CLUSTER ? 0u : g_barrier_limit;
  uint32_t target = 0, parity = 0;
  bool staging = true;
  const uint32_t smax = ctl->row_smax, seg_max = ctl->seg_max;
  const uint32_t tick0 = (b.set_tick ? b.tick_base : ctl->tick_base) + b.k0;
  if (small_spikes(b, 0)) {
    small_incoming(b, 0);
    if (!small_barrier<CLUSTER>(ctl, target, tries, &s_ok)) return;
  }
  for (uint32_t t = 0; t < b.ticks; t++) {
    const uint32_t k = b.k0 + t;
    const uint32_t item = wid * 32u + (threadIdx.x & 31u);
    const uint32_t clear = rows_prologue<1, false, 1024, true>(item, b.P.axon_heads, b.A, b.v_seg,
                                  b.bitmask ? b.bitmask + (size_t)t * b.words : nullptr, b.voff, b.nv, b.incoming,
                                  nullptr, k, b.mask2, b.axw, b.P.soma_flags, b.P.timers, b.N, b.eval, ctl, b.raise,
                                  b.lit, t ? b.pend : nullptr, small_spikes(b, t) != 0u, b.set_tick, b.tick_base,
                                  b.dopamine, b.xlit, nullptr, nullptr, b.alit, t == b.lit_tick ? 1u : 0u, s_list,
                                  s_place);
    if (!small_barrier<CLUSTER>(ctl, target, tries, &s_ok)) return;
    const TickForm form = tick_form(ctl, k, b.A, nullptr, 0u);
    const uint32_t ecount = s_place[0];
    if (threadIdx.x < ecount) b.eval[s_place[1] + threadIdx.x] = s_list[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x == 0) rows_next_lists(ctl, k);
    if (clear) b.P.soma_flags[item] = (uint8_t)clear;   // after the readout of the tick before
    // The lit-sum form's ticks take the 8-lane pass over the same rows: with a thread
    // per neuron each neuron's slots are a serial chain, and there are few neurons.
    const bool lit_rows = form == kFormLitSum || form == kFormLitRows;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      count_form(ctl, lit_rows ? kFormLitRows : form);
      count_form(ctl, kCountSmall);
    }
    // Else the fully-lit bitmap: other blocks' plain stores, then a bulk copy, over
    // what this block's threads read in an earlier tick.
    const bool stage = staging && !lit_rows;
    bool lit_on = staging;
    if (stage) {
      if (threadIdx.x == 0) {
        asm volatile("fence.proxy.async;" ::: "memory");
        bulk_to_smem(s_lit, b.lit, lit_smem_bytes(b.A), &s_bar);
      }
      lit_on = __syncthreads_and(mbar_wait_bounded(&s_bar, parity, g_first_wait_limit));
    }
    uint32_t counts[8];
    rows_update<WT>(lit_rows ? kFormLitRows : form, threadIdx.x >> 5, 32u, PassCtl{tick0 + t, smax, seg_max}, b.P, b.A,
                    b.rt, b.rw, b.cnt, b.mask2, s_list, ecount, b.pend, b.fix, ctl, b.fix_cap, b.lfz, b.wt, b.rec, lut,
                    gtab, form != kFormDense && packed ? ptab : nullptr, s_pmax, dopamine, s_lit, lit_on, counts);
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const uint32_t x = __reduce_add_sync(kFull, counts[c]);
      if ((threadIdx.x & 31u) == 0) s_cnt[c][threadIdx.x >> 5] += x;
    }
    if ((t & 255u) == 255u || t + 1 == b.ticks) {   // before 32 bits could overflow
      __syncwarp();
      uint32_t mine[8];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        mine[c] = (threadIdx.x & 31u) == 0 ? s_cnt[c][threadIdx.x >> 5] : 0u;
        if ((threadIdx.x & 31u) == 0) s_cnt[c][threadIdx.x >> 5] = 0;
      }
      block_counts(mine, ctl->ctr, ctl->gsop_same);
    }
    if (stage) {
      // a wait that gave up: the copy must land before the next one
      if (!lit_on) staging = __syncthreads_and(mbar_wait_bounded(&s_bar, parity));
      parity ^= 1u;
    }
    if (!small_barrier<CLUSTER>(ctl, target, tries, &s_ok)) return;
    const uint32_t nfix = ctl->fix_count | ctl->fix_overflow;
    rows_fixup(b.P, b.N, b.A, b.rt, b.rw, b.cnt, b.mask2, b.pend, b.eval, b.fix, ctl, k, b.ids,
               b.out + (size_t)t * b.outputs, b.outputs, b.wt, nullptr);
    const bool spikes = t + 1 < b.ticks && small_spikes(b, t + 1) != 0u;
    if (spikes) small_incoming(b, t + 1);
    // What comes next writes what the fix-up reads (heads, pending pushes) and reads
    // the network spikes' counts, but leaves the readout's flags: no barrier without them.
    if ((nfix || spikes) && !small_barrier<CLUSTER>(ctl, target, tries, &s_ok)) return;
  }
  // the last tick's soma pushes
  rows_push(b.P.axon_heads, b.P.soma_to_axon, b.A, b.pend, b.eval, b.P.soma_flags, ctl, b.k0 + b.ticks - 1u);
}

}  // namespace

uint32_t set_first_wait_limit(uint32_t tries) {
  static uint32_t current = kWaitLimit;
  const uint32_t prev = current;
  if (cudaMemcpyToSymbol(g_first_wait_limit, &tries, sizeof(tries)) == cudaSuccess) current = tries;
  return prev;
}

uint32_t set_barrier_limit(uint32_t tries) {
  static uint32_t current = kGridWaitLimit;
  const uint32_t prev = current;
  if (cudaMemcpyToSymbol(g_barrier_limit, &tries, sizeof(tries)) == cudaSuccess) current = tries;
  return prev;
}

cudaError_t rows_wish_alloc(ShardScratch& s) {
  if (s.h_counts_pinned) return cudaSuccess;
  const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&s.h_counts_pinned), 64, cudaHostAllocDefault);
  if (e == cudaSuccess) s.h_counts_pinned[0] = s.h_counts_pinned[1] = 0u;
  return e;
}

cudaError_t rows_alloc(ShardScratch& s, uint32_t N, uint32_t A, bool with_fix, cudaStream_t stream) {
  if (s.rows && s.rows->N >= N && s.rows->A >= A && (s.rows->fix || !with_fix)) return cudaSuccess;
  graph_cache_drop(&s);   // captured graphs hold the old buffers' addresses
  rows_touched(s);
  rows_free(s);
  auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
  size_t off = 0;
  const size_t o_rt = off; off = al(off + (size_t)N * kRowStride * 4);
  const size_t o_rw = off; off = al(off + (size_t)N * kRowStride * 2);
  const size_t o_cnt = off; off = al(off + (size_t)N * 2);
  const size_t o_m2 = off; off = al(off + ((size_t)A + 1) * 8);
  const size_t o_axw = off; off = al(off + (size_t)A * 4);
  const size_t o_eval = off; off = al(off + (size_t)N * 4 + 4);
  const size_t o_fix = off; off = al(off + (with_fix ? (size_t)kFixCap * 4 : 0));
  const size_t o_lit = off; off = al(off + ((size_t)std::max(A, N) / 32 + 2) * 4 + 16);
  const size_t o_live = off; off = al(off + ((size_t)A / 64 + 1) * 8);
  const size_t o_evb = off; off = al(off + ((size_t)N / 32 + 1) * 4);
  const size_t o_acc = off; off = al(off + (size_t)N * 4 + 4);
  const size_t o_gsn = off; off = al(off + (size_t)N * 4 + 4);
  const size_t o_gdn = off; off = al(off + (size_t)N * 4 + 4);
  const size_t o_am = off; off = al(off + (size_t)N * 16 + 16);
  const size_t o_lfz = off; off = al(off + (size_t)N + 4);
  const size_t o_om = off; off = al(off + (size_t)N * 16 + 16);
  const size_t o_wcnt = off; off = al(off + (size_t)kMaxUpdateWarps * 8);
  const size_t o_lsum = off; off = al(off + (size_t)N * 8 + 8);
  const size_t o_lm = off; off = al(off + (size_t)N * 16 + 16);
  const size_t o_alit = off; off = al(off + ((size_t)std::max(A, N) / 32 + 2) * 4 + 16);
  const size_t o_xlit = off; off = al(off + ((size_t)A / 32 + 2) * 4 + 16);
  void* base = nullptr;
  cudaError_t e = cudaMalloc(&base, off);
  if (e != cudaSuccess) return e;
  // zeroed in the order of the caller's stream: a blocking memset would go on
  // the legacy stream, which a non-blocking stream does not wait for (work
  // queued there before it, another shard's graph say, would delay the zeroing
  // into this shard's first batch)
  e = cudaMemsetAsync(base, 0, off, stream);
  if (e == cudaSuccess && stream == nullptr) e = cudaStreamSynchronize(nullptr);
  if (e == cudaSuccess) e = cudaMemsetAsync(&s.ctl->idx_ok, 0, 4, stream);   // an index went with the old rows
  if (e != cudaSuccess) { cudaFree(base); return e; }
  RowCache* r = new RowCache();
  char* b = static_cast<char*>(base);
  r->N = N;
  r->A = A;
  r->base = base;
  r->rt = reinterpret_cast<uint32_t*>(b + o_rt);
  r->rw = reinterpret_cast<int16_t*>(b + o_rw);
  r->cnt = reinterpret_cast<uint16_t*>(b + o_cnt);
  r->mask2 = reinterpret_cast<uint2*>(b + o_m2);
  r->axw = reinterpret_cast<uint32_t*>(b + o_axw);
  r->eval = reinterpret_cast<uint32_t*>(b + o_eval);
  r->fix = with_fix ? reinterpret_cast<uint32_t*>(b + o_fix) : nullptr;
  r->lit = reinterpret_cast<uint32_t*>(b + o_lit);
  r->live = reinterpret_cast<uint32_t*>(b + o_live);
  r->evb = reinterpret_cast<uint32_t*>(b + o_evb);
  r->acc = reinterpret_cast<int32_t*>(b + o_acc);
  r->gs_n = reinterpret_cast<uint32_t*>(b + o_gsn);
  r->gd_n = reinterpret_cast<uint32_t*>(b + o_gdn);
  r->amask = reinterpret_cast<uint4*>(b + o_am);
  r->lfz = reinterpret_cast<uint8_t*>(b + o_lfz);
  r->omask = reinterpret_cast<uint4*>(b + o_om);
  r->wcnt = reinterpret_cast<uint32_t*>(b + o_wcnt);
  r->rec = reinterpret_cast<int2*>(b + o_lsum);
  r->lmask = reinterpret_cast<uint4*>(b + o_lm);
  r->alit = reinterpret_cast<uint32_t*>(b + o_alit);
  r->xlit = reinterpret_cast<uint32_t*>(b + o_xlit);
  s.rows = r;
  return cudaSuccess;
}

cudaError_t rows_posmap(ShardScratch& s, cudaStream_t stream) {
  if (!s.rows) return cudaErrorInvalidValue;
  if (s.rows->posmap) return cudaSuccess;
  const size_t bytes = (size_t)s.rows->N * kRowStride;
  cudaError_t e = cudaMalloc(&s.rows->posmap, bytes ? bytes : 1);
  if (e == cudaSuccess) e = cudaMemsetAsync(s.rows->posmap, 0, bytes, stream);
  if (e == cudaSuccess) graph_cache_drop(&s);   // graphs captured without the map do not write it
  return e;
}

void rows_free(ShardScratch& s) {
  if (!s.rows) return;
  if (s.rows->posmap) cudaFree(s.rows->posmap);
  if (s.rows->ix.base) cudaFree(s.rows->ix.base);
  cudaFree(s.rows->base);
  delete s.rows;
  s.rows = nullptr;
}

namespace {
__global__ void __launch_bounds__(512) k_rows_decide(ShardCtl* ctl, uint32_t force, uint32_t ticks,
                                                    const uint32_t* lit, uint32_t A) {
  layout_decide(ctl, force, ticks, lit, A, false);
}
}  // namespace

cudaError_t launch_rows_decide(ShardScratch& s, uint32_t A, bool force, uint32_t ticks, cudaStream_t stream) {
  k_rows_decide<<<1, 512, 0, stream>>>(s.ctl, force ? 1u : 0u, ticks, s.rows->alit, A);
  return cudaGetLastError();
}

cudaError_t launch_rows_begin(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, cudaStream_t stream,
                              bool row_sum, bool permute, bool with_posmap, bool conditional) {
  RowCache& r = *s.rows;
  const uint32_t cond = conditional ? 1u : 0u;
  k_rows_reset_lists<<<1, 1, 0, stream>>>(s.ctl);
  if (A) k_rows_prep<<<std::min((A + 255) / 256, 4u * (uint32_t)sm_count()), 256, 0, stream>>>(
             s.ctl, r.axw, A, r.alit, permute ? r.xlit : nullptr, cond);
  if (N) {
    k_rows_mult<<<(N + 255) / 256, 256, 0, stream>>>(v.soma_to_axon, N, A, r.axw, r.mask2, s.ctl, cond);
    const uint32_t tiles = (N + 31) / 32, wave = kBuildBlocks * (uint32_t)sm_count();
    const uint32_t per = std::min(kBuildTiles, (tiles + wave - 1) / wave);
    k_rows_build<<<(tiles + per - 1) / per, 256, 0, stream>>>(v.dendrite_targets, v.dendrite_weights, v.soma_flags, N, r.rt,
                                                    r.rw, r.cnt, r.amask, r.omask, r.lfz, s.ctl, A,
                                                    row_sum ? 1u : 0u, permute ? 1u : 0u,
                                                    permute ? r.xlit : nullptr, permute ? r.rec : nullptr, r.lmask,
                                                    with_posmap ? r.posmap : nullptr, r.axw, cond, per);
  }
  return cudaGetLastError();
}

// Largest fully-lit bitmap the update kernel stages in shared memory (the
// 1024-thread variant also uses ~3.4 KB of static shared memory).
static size_t lit_smem_limit() {
  static PerDevice<size_t> limit;
  const int dev = current_device();
  return limit.get(dev, [dev] {
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    size_t lim = optin > 8192 ? (size_t)optin - 8192 : 0;
    if (cudaFuncSetAttribute(k_rows_update<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_rows_update<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lim) !=
            cudaSuccess) {
      cudaGetLastError();
      lim = 0;
    }
    return lim;
  });
}

// The update pass (with the fully-lit bitmap in shared memory when it fits).
// lc: the learned engine's control block (the pass returns at once on its
// sparse ticks), or null.
static bool rows_lit(uint32_t A) { return (size_t)lit_smem_bytes(A) <= lit_smem_limit(); }

// pdl: launched into the tick's kernel chain (launch_chain).
static void launch_rows_update(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, uint32_t k,
                               uint32_t fix_cap, const LearnCtl* lc, cudaStream_t stream, ColWT wt = ColWT{},
                               bool pdl = false, bool index = false, bool shared_gpu = false) {
  RowCache& r = *s.rows;
  const int sms = sm_count();
  const bool lit = rows_lit(A);
  const dim3 grid(lit ? sms : 4 * sms), block(lit ? 1024 : 256);
  const size_t smem = lit ? lit_smem_bytes(A) : 0;
  auto go = [&](auto kern) {
    launch_chain(kern, grid, block, smem, stream, pdl, v, A, r.rt, r.rw, r.cnt, r.mask2, r.eval, s.pend, r.fix, s.ctl,
                 k, fix_cap, r.lit, lc, r.lfz, wt, index ? 1u : 0u, r.rec, shared_gpu ? block.x / 8u : 4u);
  };
  if (wt.w) {   // the per-tick entry point: weight changes written through
    if (lit)
      go(k_rows_update<true, true>);
    else
      go(k_rows_update<false, true>);
  } else if (lit) {
    go(k_rows_update<true, false>);
  } else {
    go(k_rows_update<false, false>);
  }
}

// The lit-sum form's pass.
static void launch_rows_lsum(const ShardVramPtrs& v, ShardScratch& s, uint32_t A, uint32_t k, uint32_t fix_cap,
                             const LearnCtl* lc, cudaStream_t stream, ColWT wt = ColWT{}, bool pdl = false,
                             bool shared_gpu = false) {
  RowCache& r = *s.rows;
  launch_chain(wt.w ? k_rows_update_lsum<true> : k_rows_update_lsum<false>, dim3(kLsumBlocks * sm_count()), dim3(256),
               0, stream, pdl, v, A, r.rt, r.rw, r.cnt, r.mask2, r.eval, s.pend, r.fix, s.ctl, k, fix_cap, r.lit,
               r.rec, wt, lc, shared_gpu ? 256u : 32u);
}

// The sparse form (the learned engine's graphs): hits, then neurons, persistent warps.
static void launch_rows_sparse(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, uint32_t k,
                               uint32_t fix_cap, const LearnCtl* lc, cudaStream_t stream) {
  RowCache& r = *s.rows;
  k_sparse_hits<<<6 * sm_count(), 256, 0, stream>>>(v, A, r.rt, r.rw, r.mask2, r.live, r.evb, r.acc, s.ctl, k, lc);
  const uint32_t blocks = max(1u, min((N + 1023) / 1024, (uint32_t)(kNeuronBlocks * sm_count())));
  k_sparse_neurons<<<blocks, 256, 0, stream>>>(v, N, A, r.rt, r.rw, r.cnt, r.lfz, r.mask2, r.evb, s.pend, r.fix, s.ctl,
                                               k, fix_cap, r.lit, lc, r.acc);
}

// The GSOP passes over the spikers the tick's update pass listed (32 warps per
// SM, each with its slice of the evaluated list; a GSOP warp per slice).
static void launch_rows_gsop(const ShardVramPtrs& v, ShardScratch& s, uint32_t A, uint32_t k, uint32_t fix_cap,
                             cudaStream_t stream, const LearnCtl* lc = nullptr) {
  RowCache& r = *s.rows;
  const uint32_t nwu = (uint32_t)sm_count() * 32u;
  if (rows_lit(A)) {
    k_rows_gsop<true><<<nwu / 8, 256, 0, stream>>>(v, A, r.rt, r.rw, r.cnt, r.mask2, r.lit, r.amask, r.gs_n, r.wcnt,
                                                   nwu, r.fix, s.ctl, k, fix_cap, lc);
    k_rows_gsop_rows<true><<<nwu / 8, 256, 0, stream>>>(v, A, r.rt, r.rw, r.cnt, r.mask2, r.lit, r.gd_n,
                                                        r.wcnt + kMaxUpdateWarps, nwu, r.fix, s.ctl, k, fix_cap, lc);
  } else {
    k_rows_gsop<false><<<nwu / 8, 256, 0, stream>>>(v, A, r.rt, r.rw, r.cnt, r.mask2, r.lit, r.amask, r.gs_n, r.wcnt,
                                                    nwu, r.fix, s.ctl, k, fix_cap, lc);
    k_rows_gsop_rows<false><<<nwu / 8, 256, 0, stream>>>(v, A, r.rt, r.rw, r.cnt, r.mask2, r.lit, r.gd_n,
                                                         r.wcnt + kMaxUpdateWarps, nwu, r.fix, s.ctl, k, fix_cap, lc);
  }
}

// One tick of the row engine: prologue, update (+GSOP), fix-up, push.  In a
// batch (a.batch) the tick number, dopamine and network spike count come from
// the control block and the soma pushes may be deferred to the next tick's
// prologue; a per-tick call (cu_step_day_phase) passes them to the prologue,
// applies its pushes before it returns, and writes GSOP's weight changes
// through to the columnar blob (its row cache outlives the call).  ev
// (optional) gets the stage boundaries 2..5 recorded: after the prologue,
// after the 8-lane pass, after the lit-sum pass, after fix-up and push (GSOP
// is part of the update passes).
cudaError_t launch_tick_rows(const ShardVramPtrs& v, ShardScratch& s, const TickArgs& a, cudaStream_t stream,
                             cudaEvent_t* ev, bool have_incoming) {
  RowCache& r = *s.rows;
  const uint32_t N = a.padded_n, A = a.total_axons;
  const int sms = sm_count();
  const uint32_t* bitmask = (a.num_virtual > 0) ? a.input_bitmask : nullptr;
  uint32_t raise = 0;
  if (bitmask && ((uint64_t)a.virtual_offset + a.num_virtual > A)) raise |= AXC_ERR_VIRTUAL_RANGE;
  const uint32_t G = max(A, N);
  const bool per_tick = !a.batch;
  // The per-tick entry point launches the kernels after the prologue into the
  // kernel chain (launch_chain), which overlaps each stream launch with the
  // kernel before it: 4,841 against 4,617 calls/s at 1.5M neurons.  A batch's
  // captured graph gains nothing from it (16,955 against 17,073 ticks/s) and
  // keeps plain edges.  Never while stage events are recorded.
  const bool pdl = per_tick && ev == nullptr;
  if (G) {
    const bool wide = (G + 255) / 256 >= kProWide;
    launch_chain(wide ? (a.index ? k_rows_prologue_plain<2, true> : k_rows_prologue_plain<2, false>)
                      : (a.index ? k_rows_prologue_plain<1, true> : k_rows_prologue_plain<1, false>),
                 dim3(wide ? (G + 511) / 512 : (G + 255) / 256), dim3(256), 0, stream, false, v.axon_heads, A,
                 a.v_seg, bitmask, a.virtual_offset, a.num_virtual, s.incoming,
                 (have_incoming && !per_tick) ? s.batch_counts : nullptr, a.k, r.mask2, r.axw, v.soma_flags,
                 v.timers, N, r.eval, s.ctl, raise, r.lit, (a.k > 0 && !per_tick) ? s.pend : nullptr,
                 (have_incoming && per_tick) ? 1u : 0u, per_tick ? 1u : 0u, a.tick - a.k, (int32_t)a.dopamine,
                 r.xlit, a.sparse ? r.live : nullptr, r.evb, r.alit, a.lit_new ? 1u : 0u);
  }
  if (ev) cudaEventRecord(ev[2], stream);
  ColWT wt{};
  if (per_tick) {
    wt.w = v.dendrite_weights;
    wt.om = r.omask;
    wt.lm = r.lmask;
    wt.N = N;
  }
  // stages: ev[2]..ev[3] the 8-lane pass, ev[3]..ev[4] the lit-sum pass (both
  // with GSOP; both are launched and each returns at once on the other's
  // ticks), ev[4]..ev[5] fix-up and push.
  const uint32_t fix_cap = min(a.fix_cap, kFixCap);
  launch_rows_update(v, s, N, A, a.k, fix_cap, nullptr, stream, wt, pdl && G, a.sparse, a.shared_gpu);
  if (ev) cudaEventRecord(ev[3], stream);
  launch_rows_lsum(v, s, A, a.k, fix_cap, nullptr, stream, wt, pdl, a.shared_gpu);
  if (a.sparse) launch_rows_sparse(v, s, N, A, a.k, fix_cap, nullptr, stream);
  if (ev) cudaEventRecord(ev[4], stream);
  const bool readout = a.num_outputs > 0 && a.mapped_soma_ids && a.output_history;
  launch_chain(k_rows_fixup, dim3(2 * sms), dim3(256), 0, stream, pdl, v, N, A, r.rt, r.rw, r.cnt, r.mask2, s.pend,
               r.eval, r.fix, s.ctl, a.k, a.mapped_soma_ids, a.output_history, readout ? a.num_outputs : 0, wt,
               (volatile uint32_t*)(a.index ? s.h_counts_pinned : nullptr));
  // the soma pushes: by the next tick's prologue within a batch, here on its last tick
  if (!a.defer_push)
    launch_chain(k_rows_push, dim3(8 * sms), dim3(256), 0, stream, pdl, v.axon_heads, v.soma_to_axon, A, s.pend,
                 r.eval, v.soma_flags, s.ctl, a.k);
  if (ev) cudaEventRecord(ev[5], stream);
  return cudaGetLastError();
}

// Rows that run in one cluster / in one resident grid (k_rows_small), by the larger
// of neurons and axons.  A cluster's barrier takes 0.7 us and the grid's 1.2, but its
// 16 SMs take longer over 4,000 plastic rows (45 us a per-tick call) than the
// kernel chain (39); the grid is even with the chain at 100,000 axons (saturated
// rows: 370 us per 20 ticks on both) and behind it at 150,000 (432 against 400).
constexpr uint32_t kSmallCluster = 4096, kSmallTick = 3072;   // the latter: per-tick calls
constexpr uint32_t kSmallBlocks = 640;   // a resident grid: neurons or axons per SM

// Blocks of k_rows_small's cluster here, 0 where none fits.
static uint32_t small_cluster() {
  static PerDevice<uint32_t> size;
  return size.get(current_device(), [] {
    for (const uint32_t c : {16u, 8u}) {
      int n = 0, m = 0;
      auto fits = [&](auto kern, int* out) {
        if (c > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
          return false;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c);
        cfg.blockDim = dim3(1024);
        cfg.dynamicSmemBytes = lit_smem_bytes(kSmallCluster);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = c;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        return cudaOccupancyMaxActiveClusters(out, kern, &cfg) == cudaSuccess && *out > 0;
      };
      if (fits(k_rows_small<true, false>, &n) && fits(k_rows_small<true, true>, &m)) return c;
      cudaGetLastError();
    }
    return 0u;
  });
}

// Blocks of k_rows_small's resident grid here, 0 where it does not fit.
static uint32_t small_grid() {
  static PerDevice<uint32_t> size;
  return size.get(current_device(), [] {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_rows_small<false, false>, 1024,
                                                      lit_smem_bytes(kSmallBlocks * sm_count())) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    return n > 0 ? (uint32_t)sm_count() : 0u;
  });
}

bool rows_small(uint32_t N, uint32_t A, bool whole_gpu, bool batch) {
  const uint32_t G = max(N, A);
  if (G <= (batch ? kSmallCluster : kSmallTick) && small_cluster()) return true;
  return whole_gpu && G <= kSmallBlocks * (uint32_t)sm_count() && small_grid();
}

cudaError_t launch_rows_small(const ShardVramPtrs& v, ShardScratch& s, const TickArgs& a, uint32_t ticks,
                              uint32_t words, cudaStream_t stream) {
  RowCache& r = *s.rows;
  SmallArgs b{};
  b.P = v;
  b.N = a.padded_n;
  b.A = a.total_axons;
  b.v_seg = a.v_seg;
  b.bitmask = a.num_virtual > 0 ? a.input_bitmask : nullptr;
  b.words = words;
  b.voff = a.virtual_offset;
  b.nv = a.num_virtual;
  b.raise = b.bitmask && (uint64_t)a.virtual_offset + a.num_virtual > b.A ? AXC_ERR_VIRTUAL_RANGE : 0u;
  b.spikes = a.batch || a.num_incoming > 0 ? a.incoming_spikes : nullptr;
  b.spike_cap = a.max_incoming;
  b.spike_count = a.num_incoming;
  b.counts = a.batch ? s.batch_counts : nullptr;
  b.incoming = s.incoming;
  b.rt = r.rt;
  b.eval = r.eval;
  b.pend = s.pend;
  b.fix = r.fix;
  b.lit = r.lit;
  b.alit = r.alit;
  b.xlit = r.xlit;
  b.rw = r.rw;
  b.cnt = r.cnt;
  b.lfz = r.lfz;
  b.rec = r.rec;
  b.axw = r.axw;
  b.mask2 = r.mask2;
  b.ctl = s.ctl;
  if (a.num_outputs > 0 && a.mapped_soma_ids && a.output_history) {
    b.ids = a.mapped_soma_ids;
    b.out = a.output_history;
    b.outputs = a.num_outputs;
  }
  b.fix_cap = min(a.fix_cap, kFixCap);
  b.ticks = ticks;
  b.k0 = a.k;
  b.lit_tick = a.batch ? (ticks > kLitWindow ? ticks - kLitWindow : 0u) : a.lit_new ? 0u : ticks;
  b.set_tick = a.batch ? 0u : 1u;
  b.tick_base = a.tick - a.k;
  b.dopamine = a.dopamine;
  if (!a.batch) {
    b.wt.w = v.dendrite_weights;
    b.wt.om = r.omask;
    b.wt.lm = r.lmask;
    b.wt.N = b.N;
  }
  const bool cluster = max(b.N, b.A) <= kSmallCluster && small_cluster();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cluster ? small_cluster() : small_grid());
  cfg.blockDim = dim3(1024);
  cfg.dynamicSmemBytes = lit_smem_bytes(b.A);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  if (cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cfg.gridDim.x;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg,
                            !cluster ? k_rows_small<false, false> : a.batch ? k_rows_small<true, false>
                                                                            : k_rows_small<true, true>,
                            b);
}

// Index of the current rows.  Entries are counted per axon, placed through a
// cursor (any order), then sorted by segment within the axon, a warp per axon.
namespace {
__global__ void __launch_bounds__(256) k_ix_count(const uint32_t* __restrict__ rt, const uint16_t* __restrict__ cnt,
                                                  uint32_t N, uint32_t A, uint32_t* __restrict__ deg) {
  const size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (size_t)N * kRowStride) return;
  const uint32_t n = (uint32_t)(r / kRowStride), q = (uint32_t)(r % kRowStride);
  if (q >= (cnt[n] & 0xFFu)) return;
  const uint32_t a = (rt[r] & AXC_TARGET_AXON_MASK) - 1u;
  if (a < A) atomicAdd(deg + a, 1u);   // invalid targets (redirected to A) never hit
}

__global__ void __launch_bounds__(256) k_ix_fill(const uint32_t* __restrict__ rt, const uint16_t* __restrict__ cnt,
                                                 uint32_t N, uint32_t A, uint32_t* __restrict__ cursor,
                                                 uint32_t* __restrict__ ent) {
  const size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= (size_t)N * kRowStride) return;
  const uint32_t n = (uint32_t)(r / kRowStride), q = (uint32_t)(r % kRowStride);
  if (q >= (cnt[n] & 0xFFu)) return;
  const uint32_t a = (rt[r] & AXC_TARGET_AXON_MASK) - 1u;
  if (a < A) ent[atomicAdd(cursor + a, 1u)] = (uint32_t)r;
}

// Entries of an axon sorted in registers: up to kIxPer a lane.
constexpr uint32_t kIxPer = 16;

__global__ void __launch_bounds__(256) k_ix_sort(const uint32_t* __restrict__ rt, const uint32_t* __restrict__ off,
                                                 uint32_t A, uint32_t* __restrict__ ent, uint16_t* __restrict__ seg) {
  __shared__ uint32_t s_cnt[8][32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t a = blockIdx.x * 8u + w;
  if (a >= A) return;
  const uint32_t o = off[a], d = off[a + 1] - o;
  if (d > 32u * kIxPer) {
    if (lane == 0) seg[(size_t)a * 32u] = (uint16_t)kSegUnsorted;
    return;
  }
  s_cnt[w][lane] = 0;
  __syncwarp();
  uint32_t e[kIxPer], b[kIxPer];   // entry, bucket | rank within the bucket << 8
#pragma unroll
  for (uint32_t i = 0; i < kIxPer; i++) {
    const uint32_t x = lane + 32u * i;
    b[i] = 0;
    e[i] = 0;
    if (x < d) {
      e[i] = ent[o + x];
      const uint32_t s = min(__ldg(rt + e[i]) >> AXC_TARGET_SEG_SHIFT, 31u);
      b[i] = s | (atomicAdd(&s_cnt[w][s], 1u) << 8);
    }
  }
  __syncwarp();
  const uint32_t mine = s_cnt[w][lane];
  uint32_t incl = mine;
#pragma unroll
  for (int st = 1; st < 32; st <<= 1) {
    const uint32_t x = __shfl_up_sync(kFull, incl, st);
    if (lane >= (uint32_t)st) incl += x;
  }
  __syncwarp();
  s_cnt[w][lane] = incl - mine;
  seg[(size_t)a * 32u + lane] = (uint16_t)(incl - mine);
  __syncwarp();
#pragma unroll
  for (uint32_t i = 0; i < kIxPer; i++)
    if (lane + 32u * i < d) ent[o + s_cnt[w][b[i] & 0xFFu] + (b[i] >> 8)] = e[i];
}

// Exclusive scan of in[0..n) (also kept in cur) into out[0..n]: blocks of 4096
// values, then one block over the block sums, then their addition.
__global__ void __launch_bounds__(1024) k_ix_scan(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                  uint32_t n, uint32_t* __restrict__ bsum) {
  __shared__ uint32_t s[32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t base = blockIdx.x * 4096u + threadIdx.x * 4u;
  uint32_t v[4], t = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    v[i] = base + i < n ? in[base + i] : 0u;
    t += v[i];
  }
  uint32_t incl = t;
#pragma unroll
  for (int st = 1; st < 32; st <<= 1) {
    const uint32_t x = __shfl_up_sync(kFull, incl, st);
    if (lane >= (uint32_t)st) incl += x;
  }
  if (lane == 31) s[w] = incl;
  __syncthreads();
  if (w == 0) {
    uint32_t x = s[lane];
#pragma unroll
    for (int st = 1; st < 32; st <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, st);
      if (lane >= (uint32_t)st) x += y;
    }
    s[lane] = x;
  }
  __syncthreads();
  uint32_t run = incl - t + (w ? s[w - 1] : 0u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
  if (threadIdx.x == 1023 && bsum) bsum[blockIdx.x] = run;
}

__global__ void __launch_bounds__(256) k_ix_add(uint32_t* __restrict__ off, uint32_t* __restrict__ cur, uint32_t n,
                                                const uint32_t* __restrict__ bsum) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t x = off[i] + bsum[i / 4096u];
  if (i + 1u == n) off[n] = x + cur[i];
  off[i] = x;
  cur[i] = x;
}

__global__ void k_ix_done(ShardCtl* ctl, RowIndex ix) {
  ctl->ix_off = ix.off;
  ctl->ix_seg = ix.seg;
  ctl->ix_ent = ix.ent;
  ctl->idx_ok = 1u;
  ctl->idx_sum = ctl->lay_sum;
  ctl->lay_now = 0u;   // laid out above: the batch's own layout kernels return at once
}
}  // namespace

cudaError_t rows_index_wish(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, uint32_t A, cudaStream_t stream,
                            bool row_sum, bool with_posmap) {
  volatile uint32_t* wish = s.h_counts_pinned;
  if (!wish || !*wish || !s.rows || N == 0 || A == 0) return cudaSuccess;
  *wish = 0u;
  RowCache& r = *s.rows;
  // 4096 blocks of 4096 axons in the scan, 32-bit entries
  if (r.ix_failed || A > (1u << 24) || (size_t)r.N * kRowStride > 0xFFFFFFFFull) return cudaSuccess;
  RowIndex& ix = r.ix;
  if (!ix.base) {
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    size_t off = 0;
    const size_t o_off = off; off = al(off + ((size_t)r.A + 2) * 4);
    const size_t o_cur = off; off = al(off + (size_t)r.A * 4);
    const size_t o_bsum = off; off = al(off + 4097 * 4);
    const size_t o_seg = off; off = al(off + (size_t)r.A * 64);
    const size_t o_ent = off; off = al(off + (size_t)r.N * kRowStride * 4);
    if (cudaMalloc(&ix.base, off) != cudaSuccess) {
      cudaGetLastError();   // no room: the dense pass goes on
      ix.base = nullptr;
      r.ix_failed = true;
      return cudaSuccess;
    }
    char* b = static_cast<char*>(ix.base);
    ix.off = reinterpret_cast<uint32_t*>(b + o_off);
    ix.cur = reinterpret_cast<uint32_t*>(b + o_cur);
    ix.bsum = reinterpret_cast<uint32_t*>(b + o_bsum);
    ix.seg = reinterpret_cast<uint16_t*>(b + o_seg);
    ix.ent = reinterpret_cast<uint32_t*>(b + o_ent);
  }
  cudaError_t e = launch_rows_begin(v, s, N, A, stream, row_sum, true, with_posmap, true);
  if (e == cudaSuccess) e = cudaMemsetAsync(ix.cur, 0, (size_t)A * 4, stream);
  if (e != cudaSuccess) return e;
  const uint32_t gb = (uint32_t)(((size_t)N * kRowStride + 255) / 256), nb = (A + 4095) / 4096;
  k_ix_count<<<gb, 256, 0, stream>>>(r.rt, r.cnt, N, A, ix.cur);
  k_ix_scan<<<nb, 1024, 0, stream>>>(ix.cur, ix.off, A, ix.bsum);
  k_ix_scan<<<1, 1024, 0, stream>>>(ix.bsum, ix.bsum, nb, nullptr);
  k_ix_add<<<(A + 255) / 256, 256, 0, stream>>>(ix.off, ix.cur, A, ix.bsum);
  k_ix_fill<<<gb, 256, 0, stream>>>(r.rt, r.cnt, N, A, ix.cur, ix.ent);
  k_ix_sort<<<(A + 7) / 8, 256, 0, stream>>>(r.rt, ix.off, A, ix.ent, ix.seg);
  k_ix_done<<<1, 1, 0, stream>>>(s.ctl, ix);
  return cudaGetLastError();
}

cudaError_t launch_rows_end(const ShardVramPtrs& v, ShardScratch& s, uint32_t N, cudaStream_t stream) {
  RowCache& r = *s.rows;
  const uint32_t blocks = std::max(1u, (N + 255) / 256), tiles = std::max(1u, (N + 31) / 32);
  k_rows_writeback<<<blocks, 256, 0, stream>>>(v.dendrite_weights, N, r.rw, r.cnt, r.omask, r.lmask, s.ctl, s.pend,
                                               s.incoming, s.total_axons);
  k_rows_writeback_tiles<<<std::min(tiles, 4u * (uint32_t)sm_count()), 256, 0, stream>>>(v.dendrite_weights, N, r.rw,
                                                                                         r.omask, r.lmask, s.ctl);
  return cudaGetLastError();
}

}  // namespace axc
