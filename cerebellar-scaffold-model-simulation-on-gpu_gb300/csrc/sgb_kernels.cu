// Step kernels of the scaffold simulation hot path (sm_103a).
//
// One exchange step t consists of two grid-wide phases:
//   update   every cell, one warp per 32-cell word: INPUT cells draw their
//            Philox Poisson / periodic stimulus (reference InputStimulation,
//            UserInputFunctions.cu:86-120); LIF cells consume ring slot t and
//            integrate `substeps` Euler substeps (reference update_lif_ch,
//            Simulation_header.cu:305-381).  Spikes leave as a bitmap word
//            per warp (ballot), a compacted active list (ballot + popc + one
//            atomic per warp) and per-segment counts.
//   deliver  event-driven push: one warp per spiking cell walks the cell's
//            row of the push table and adds fixed-point weights into ring
//            slot t + delay of each target; dense pull for projections in ELL
//            mode: each post cell gathers the spike bits of its in-row from the
//            bitmap of step t + 1 - delay and adds the sum into ring slot t + 1
//            (the reference's pull, Simulation_header.cu:83-139, with the delay
//            applied on read as at GPUScaffoldSimulation.cu:735).
// Two drivers run these phases: per-step kernels (replayed from a CUDA graph;
// kernel boundaries order the phases) and one persistent cooperative kernel
// per chunk of steps (a bounded grid barrier orders them).  The persistent
// kernel comes in three forms: fused (every word resident in one warp, every
// projection event-driven: update and push share one phase, one barrier a
// step, push rows in shared memory, long rows delivered by their targets'
// blocks; with one substep a step it
// publishes each step's spikes one step early, as soon as the potential that
// decides them is known, and makes a step's writes after its barrier
// arrival -- the late-push timeline, optionally with a split barrier),
// resident (words resident, some dense pulls: one barrier a step with one
// substep, else two) and general (more words than warps; one
// barrier a step with the pushes in each block's shared memory when every
// projection is event-driven, else two with a global item list).  With
// plastic projections a plasticity phase runs before the deliveries.  The
// ring holds int32 fixed-point sums, so push and pull delivery, any launch
// order and any number of instances give bit-identical conductances.
#include <stdint.h>

#include <algorithm>

#include "sgb_device.h"
#include "sgb_philox.h"
#include "../../include/scaffold_gb300.h"

namespace sgb {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// Step indices shared by every phase of one step.
struct StepIdx {
  unsigned long long t;
  uint32_t slot;  // t % ring_slots
  uint32_t hrow;  // t % hist_rows
  uint32_t srow;  // t % (hist_rows + 1): spike-summary row
  uint32_t rel;   // step index within the chunk
  // Element offsets of the step's rows, computed once per step (all fit 32
  // bits: ring_slots * n_pad < 2^31, 2 * hist_rows * n_words <= 2^28).
  uint32_t roff;   // ring slot: slot * n_pad (int2 elements)
  uint32_t hoff;   // history row of step t: (hist_rows - 1 - hrow) * n_words
  uint32_t hoff2;  // its second copy, hist_rows rows further
  bool keep;       // general kernel, two cells per lane: write the history row
};

template <bool BF16>
__device__ __forceinline__ float load_weight(const void* w, uint32_t q) {
  if (BF16) return __uint_as_float(((uint32_t)__ldg((const unsigned short*)w + q)) << 16);
  return __ldg((const float*)w + q);
}

__device__ __forceinline__ bool window_on(const SrcDev& s, int64_t k) {
  if (s.win_end <= s.win_start) return true;
  int64_t kk = k;
  if (s.win_period > 0) {
    if ((uint64_t)k <= 0xFFFFFFFFull && (uint64_t)s.win_period <= 0xFFFFFFFFull) {
      kk = (int64_t)((uint32_t)k % (uint32_t)s.win_period);  // same value, 32-bit divide
    } else {
      kk = k % s.win_period;
      if (kk < 0) kk += s.win_period;
    }
  }
  return kk >= s.win_start && kk < s.win_end;
}

// PeriodicFiring (UserInputFunctions.cu:8-10): fires in the substep where the
// cycle count floor((t - start) * f / 1000) increments.
__device__ __forceinline__ bool periodic_fire(const SrcDev& s, int64_t k) {
  const double x1 = __dmul_rn((double)(k - s.k_phase), s.cyc);
  const double x0 = __dmul_rn((double)(k - s.k_phase - 1), s.cyc);
  return floor(x1) != floor(x0);
}

__device__ __forceinline__ bool input_fire(const StepArgs& a, const SrcDev* srcs, const SegDev& sd,
                                           uint32_t local, uint32_t mask, unsigned long long t) {
  const int substeps = a.substeps;
  bool fire = false;
  U4 r{};
#pragma unroll 1
  for (int s = 0; s < substeps; ++s) {
    if ((s & 3) == 0) r = philox_draw(sd.seed, sd.key_base + local, t, kTagInput, (uint32_t)(s >> 2));
    const uint32_t x = u4_get(r, s & 3);
    const int64_t k = (int64_t)t * substeps + s;
    uint32_t m = mask;
    while (m) {
      const int b = __ffs(m) - 1;
      m &= m - 1;
      const SrcDev src = srcs[sd.src_first + b];
      if (!window_on(src, k)) continue;
      if (src.kind == SGB_INPUT_POISSON)
        fire |= (uint64_t)x < src.thresh;
      else
        fire |= periodic_fire(src, k);
    }
  }
  return fire;
}
// Conductance-based LIF, `substeps` explicit Euler steps.  Statement order is
// the reference's (Simulation_header.cu:338-370): synaptic current from the
// old conductances, conductance decay plus the step's increment on substep 0
// only, spike test on the old potential, refractory count, reset.  Every
// operation is a single IEEE-rounded FP32 op so a CPU restatement reproduces
// it bit for bit.
// The LIF constants of a segment, fetched as four 16-byte groups (plus the
// refractory length): a word's update issues 5 loads for them, not 17.
struct LifK {
  float El, Vr, Vth, Ie, neg_gL, dt_cm, keep0, keep1, gw0, gw1, E0, E1, inv0, inv1;
  uint32_t sel0, sel1;
  int32_t ref_steps;
};
__device__ __forceinline__ LifK lif_k(const SegDev& sd) {
  const float4* p = reinterpret_cast<const float4*>(&sd.El);
  const float4 a = p[0], b = p[1], c = p[2], d = p[3];
  LifK k;
  k.El = a.x; k.Vr = a.y; k.Vth = a.z; k.Ie = a.w;
  k.neg_gL = b.x; k.dt_cm = b.y; k.keep0 = b.z; k.keep1 = b.w;
  k.gw0 = c.x; k.gw1 = c.y; k.E0 = c.z; k.E1 = c.w;
  k.inv0 = d.x; k.inv1 = d.y; k.sel0 = __float_as_uint(d.z); k.sel1 = __float_as_uint(d.w);
  k.ref_steps = sd.ref_steps;
  return k;
}

// SUB = 1: the single-substep form of the same operations (the benchmark
// configurations); SUB = 0: `substeps` substeps.
template <int SUB>
__device__ __forceinline__ bool lif_update(const LifK& k, int substeps, float4& st, int2 acc) {
  float u = st.x, g0 = st.y, g1 = st.z;
  int ref = __float_as_int(st.w);
  const float dge = __fmul_rn(__int2float_rn(acc.x), k.inv0);
  const float dgi = __fmul_rn(__int2float_rn(acc.y), k.inv1);
  const float in0 = k.sel0 ? dgi : dge;
  const float in1 = k.sel1 ? dgi : dge;
  bool spk = false;
  const int n = SUB == 1 ? 1 : substeps;
  for (int s = 0; s < n; ++s) {
    const float isyn = __fmaf_rn(g1, __fsub_rn(u, k.E1), __fmul_rn(g0, __fsub_rn(u, k.E0)));
    const float cur = __fsub_rn(__fmaf_rn(k.neg_gL, __fsub_rn(u, k.El), k.Ie), isyn);
    const float du = __fmul_rn(k.dt_cm, cur);
    if (s == 0) {
      g0 = __fmaf_rn(g0, k.keep0, __fmul_rn(k.gw0, in0));
      g1 = __fmaf_rn(g1, k.keep1, __fmul_rn(k.gw1, in1));
    } else {
      g0 = __fmul_rn(g0, k.keep0);
      g1 = __fmul_rn(g1, k.keep1);
    }
    const bool above = u > k.Vth;
    spk |= above;
    ref = above ? k.ref_steps : (ref > 0 ? ref - 1 : 0);
    u = ref ? k.Vr : __fadd_rn(u, du);
  }
  st = make_float4(u, g0, g1, __int_as_float(ref));
  return spk;
}

__device__ __forceinline__ bool lif_step(const LifK& k, int substeps, float4& st, int2 acc) {
  return substeps == 1 ? lif_update<1>(k, 1, st, acc) : lif_update<0>(k, substeps, st, acc);
}

// ---- phase 1: one warp updates the 32 cells of word w --------------------------
// Cross-block data (ring slots written by other SMs' atomics, counters, push
// items) is accessed with ld/st.global.cg so a persistent kernel never sees a
// stale L1 line.

// Push items carry the step that produced them; a consumer clears each item
// it delivers, so the delivery phase finds the end of the list without
// reading the item count.
__device__ __forceinline__ uint32_t item_tag(unsigned long long t) {
  return ((uint32_t)t & 0x3FFFFFu) | 0x400000u;  // never 0 (cleared)
}

// Spike bits of word w at step t: both copies of the history row, and, when
// any cell of the word spiked, the word's bit in the step's summary row.
__device__ __forceinline__ void put_hist(const StepArgs& a, const StepIdx& ix, uint32_t w,
                                         uint32_t bits) {
  __stcg(a.hist + (ix.hoff + w), bits);  // rows in decreasing step order
  __stcg(a.hist + (ix.hoff2 + w), bits);
  if (bits) atomicOr(a.hsum + (size_t)ix.srow * a.n_swords + (w >> 5), 1u << (w & 31u));
}

// The summary row of step t + 1 is free during step t (the oldest row a pull
// of step t reads is that of t + 1 - H); threads gtid, gtid + gthreads, ...
// clear it.
__device__ __forceinline__ void clear_next_summary(const StepArgs& a, const StepIdx& ix,
                                                   uint32_t gtid, uint32_t gthreads) {
  const uint32_t row = ix.srow == a.hist_rows ? 0u : ix.srow + 1u;
  for (uint32_t j = gtid; j < a.n_swords; j += gthreads)
    __stcg(a.hsum + (size_t)row * a.n_swords + j, 0u);
}

// One cell's step; state and constants in registers, ring slot consumed.
__device__ __forceinline__ bool cell_fire(const StepArgs& a, const SegDev& sd, uint32_t i,
                                          uint32_t local, bool valid, float4& st, uint32_t mask,
                                          const StepIdx& ix) {
  if (!valid) return false;
  if (sd.kind == kSegInput) return mask ? input_fire(a, a.srcs, sd, local, mask, ix.t) : false;
  int2* rp = reinterpret_cast<int2*>(a.ring) + (ix.roff + i);
  const int2 acc = __ldcg(rp);
  if (acc.x | acc.y) __stcg(rp, make_int2(0, 0));
  return lif_step(lif_k(sd), a.substeps, st, acc);
}

template <bool BF16>
__device__ __forceinline__ uint32_t push_item(const StepArgs& a, uint2 it, uint32_t slot0);

// A block's own push-item list (general persistent kernel with one grid
// barrier per step): items in shared memory, the step's count.
constexpr uint32_t kGenItems = 1024;  // items per block and step (8 KiB)
struct BlockItems {
  uint2* items;
  uint32_t* count;
};

// Spike bookkeeping of one word: bitmap word, per-segment count, event count,
// raster entries, and the spiking cells' push rows cut into kPushChunk items
// laid out by a warp-inclusive scan (one atomic reserves the warp's items):
// in the step's global list, or with LOCAL in the block's list, where the
// warp itself pushes the items past its capacity (their slots t + d, d >= 1,
// are read after the step's barrier).  Returns the synapses pushed here.
template <bool BF16 = false, bool LOCAL = false>
__device__ __forceinline__ uint32_t publish_word(const StepArgs& a, uint32_t w, uint32_t seg,
                                                 uint32_t i, bool fired, uint32_t r0, uint32_t r1,
                                                 uint32_t outdeg, const StepIdx& ix,
                                                 BlockItems bi = {nullptr, nullptr}) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t ballot = __ballot_sync(kFull, fired);
  if (lane == 0) put_hist(a, ix, w, ballot);
  if (ballot == 0) return 0;
  const uint32_t n = __popc(ballot);
  const uint32_t rank = __popc(ballot & ((1u << lane) - 1u));
  const uint32_t ev = __reduce_add_sync(kFull, fired ? outdeg : 0u);
  const uint32_t nit = fired ? (r1 - r0 + kPushChunk - 1) / kPushChunk : 0u;
  uint32_t incl = nit;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  const uint32_t tot_items = __shfl_sync(kFull, incl, 31);
  uint32_t off = 0, roff = 0;
  Ctl* ctl = a.ctl;
  if (lane == 0) {
    if (tot_items) off = LOCAL ? atomicAdd(bi.count, tot_items)
                               : atomicAdd(&ctl->active_count[ix.t & 1], tot_items);
    atomicAdd(&a.counts[(size_t)ix.rel * a.n_segs + seg], n);
    if (ev) atomicAdd(&ctl->events, (unsigned long long)ev);
    if (a.raster_cap) roff = atomicAdd(&ctl->raster_count, n);
  }
  off = __shfl_sync(kFull, off, 0) + incl - nit;
  uint32_t walked = 0;
  if (LOCAL) {
    for (uint32_t k = 0; k < nit && off + k < kGenItems; ++k) {
      const uint32_t q0 = r0 + k * kPushChunk;
      bi.items[off + k] = make_uint2(q0, min(kPushChunk, r1 - q0) << 23);
    }
    uint32_t spill = __ballot_sync(kFull, off + nit > kGenItems);
    while (spill) {
      const int src = __ffs(spill) - 1;
      spill &= spill - 1;
      const uint32_t o = __shfl_sync(kFull, off, src), c = __shfl_sync(kFull, nit, src);
      const uint32_t b0 = __shfl_sync(kFull, r0, src), b1 = __shfl_sync(kFull, r1, src);
      for (uint32_t k = o < kGenItems ? kGenItems - o : 0u; k < c; ++k) {
        const uint32_t q0 = b0 + k * kPushChunk;
        walked += push_item<BF16>(a, make_uint2(q0, min(kPushChunk, b1 - q0) << 23), ix.slot);
      }
    }
  } else {
    uint2* items = a.items + (size_t)(ix.t & 1) * a.item_cap;
    const uint32_t tag = item_tag(ix.t);
    for (uint32_t k = 0; k < nit; ++k) {
      const uint32_t q0 = r0 + k * kPushChunk;
      const uint32_t len = min(kPushChunk, r1 - q0);
      __stcg(items + off + k, make_uint2(q0, (len << 23) | tag));
    }
  }
  if (a.raster_cap) {
    roff = __shfl_sync(kFull, roff, 0);
    if (fired) {
      if (roff + rank < a.raster_cap)
        a.raster[roff + rank] = i;
      else
        atomicOr(&ctl->error, kErrRasterOverflow);
    }
  }
  return walked;
}

// General form, everything from global memory.  The word's state and ring
// slot are loaded first (their addresses depend only on the word index), the
// segment descriptor next; push-row bounds and out-degrees only for spiking
// cells.  Callers may issue load_word for the next word before finishing the
// current one (the two touch different cells).
struct WordIn {
  float u;
  float2 g;
  int2 acc;
  uint32_t seg;
};

__device__ __forceinline__ WordIn load_word(const StepArgs& a, uint32_t w, const StepIdx& ix) {
  const uint32_t i = (w << 5) + (threadIdx.x & 31u);
  WordIn in;
  in.seg = __ldg(a.seg_of_word + w);
  in.acc = __ldcg(reinterpret_cast<const int2*>(a.ring) + (ix.roff + i));
  // State streams through L2 only: no L1 allocation for the largest stream,
  // which would evict the segment descriptors every word reads.
  in.u = __ldcg(a.su + i);
  in.g = __ldcg(a.sg + i);
  return in;
}

// Register state {u, g0, g1, ref bits} from / to the stored fields.
__device__ __forceinline__ float4 state_in(float u, float2 g, float vr) {
  const int32_t ref = unpack_ref(u);
  return make_float4(ref ? vr : u, g.x, g.y, __int_as_float(ref));
}
__device__ __forceinline__ void state_out(const StepArgs& a, uint32_t i, const float4& st) {
  __stcg(a.su + i, pack_u(st.x, __float_as_int(st.w)));
  __stcg(a.sg + i, make_float2(st.y, st.z));
}

// RECENT: the handle may keep per-cell spike registers (plastic
// projections); the general persistent kernel takes the RECENT = false form
// when it has none, so the update of a network without plasticity carries
// no trace of them.
// SEGSMEM: the segment descriptors and stimulus sources are in the general
// persistent kernel's dynamic shared memory (g_dyn: descriptors, then
// sources) rather than read from global memory.
extern __shared__ __align__(16) unsigned char g_dyn[];
__host__ __device__ __forceinline__ size_t seg_table_bytes(uint32_t n_segs) {
  return ((size_t)n_segs * sizeof(SegDev) + 15) & ~(size_t)15;
}

template <bool RECENT = true, bool SEGSMEM = false, bool BF16 = false, bool LOCAL = false>
__device__ __forceinline__ uint32_t finish_word(const StepArgs& a, uint32_t w, const WordIn& in,
                                                const StepIdx& ix,
                                                BlockItems bi = {nullptr, nullptr}) {
  if (in.seg == 0xFFFFu) return 0;  // padding between segments (warp-uniform)
  const uint32_t lane = threadIdx.x & 31u;
  const SegDev& sd = SEGSMEM ? reinterpret_cast<const SegDev*>(g_dyn)[in.seg] : a.segs[in.seg];
  const uint4 hd = *reinterpret_cast<const uint4*>(&sd);  // base, count, key_base, kind
  const uint32_t i = (w << 5) + lane;
  const uint32_t local = i - hd.x;
  const bool valid = local < hd.y;
  bool fired = false;
  if (hd.w == kSegInput) {  // warp-uniform
    if (valid) {
      const uint32_t mask = __ldg(a.src_mask + i);
      const SrcDev* srcs =
          SEGSMEM ? reinterpret_cast<const SrcDev*>(g_dyn + seg_table_bytes(a.n_segs)) : a.srcs;
      if (mask) fired = input_fire(a, srcs, sd, local, mask, ix.t);
    }
  } else {
    // Every lane of a LIF word runs the update: a padding lane past the
    // segment's end integrates its own (never read) padding state and is
    // masked out of the spikes, so no lane diverges here.
    if (in.acc.x | in.acc.y)
      __stcg(reinterpret_cast<int2*>(a.ring) + (ix.roff + i), make_int2(0, 0));
    const LifK k = lif_k(sd);
    float4 st = state_in(in.u, in.g, k.Vr);
    fired = lif_step(k, a.substeps, st, in.acc) && valid;
    state_out(a, i, st);
  }
  // Handles with plastic projections: each cell's last 64 steps of spikes,
  // bit j = step t - j, for the pairing windows.
  if (RECENT && a.recent && valid)
    a.recent[(ix.t & 1ull) * a.n_pad + i] =
        (__ldcg(a.recent + ((ix.t + 1ull) & 1ull) * a.n_pad + i) << 1) | (fired ? 1ull : 0ull);
  uint32_t r0 = 0, r1 = 0, od = 0;
  if (fired) {
    od = __ldg(a.outdeg + i);
    if (a.any_push) {
      r0 = __ldg(a.push_row + i);
      r1 = __ldg(a.push_row + i + 1);
    }
  }
  return publish_word<BF16, LOCAL>(a, w, in.seg, i, fired, r0, r1, od, ix, bi);
}

__device__ __forceinline__ void update_word(const StepArgs& a, uint32_t w, const StepIdx& ix) {
  finish_word(a, w, load_word(a, w, ix), ix);
}

// Words gw, gw + nw, ... with the next word's loads in flight while the
// current one is computed.  Returns the synapses pushed on the way.
template <bool RECENT, bool SEGSMEM, bool BF16, bool LOCAL>
__device__ __forceinline__ uint32_t update_words(const StepArgs& a, uint32_t gw, uint32_t nw,
                                                 const StepIdx& ix, BlockItems bi) {
  uint32_t w = gw, walked = 0;
  if (w >= a.n_words) return 0;
  WordIn cur = load_word(a, w, ix);
  while (true) {
    const uint32_t wn = w + nw;
    WordIn nxt;
    if (wn < a.n_words) nxt = load_word(a, wn, ix);
    walked += finish_word<RECENT, SEGSMEM, BF16, LOCAL>(a, w, cur, ix, bi);
    if (wn >= a.n_words) break;
    w = wn;
    cur = nxt;
  }
  return walked;
}

// ---- two cells per lane (general persistent kernel, one-barrier form) ----------
// A pair is two consecutive words, cells 64p .. 64p + 63; lane L takes cells
// 64p + 2L and 64p + 2L + 1, both in word 2p + (L >> 4), so a lane's two cells
// share a segment (segments start on 32-cell boundaries).  A lane moves its
// cells' ring entries, potentials and conductances as one int4, float2 and
// float4 each, and the per-word work -- segment header, LIF constants, bitmap
// words, counts, push items -- is shared by twice the cells.  Each cell's
// arithmetic is exactly the one-cell form's.
struct PairIn {
  int4 acc;      // {exc, inh} of the lane's two cells
  float4 g;      // {g0, g1} of the two cells
  float2 u;      // stored potential fields of the two cells
  uint32_t seg;  // segment of the lane's word
};

__device__ __forceinline__ PairIn load_pair(const StepArgs& a, uint32_t p, const StepIdx& ix) {
  const uint32_t c = (p << 6) + 2u * (threadIdx.x & 31u);
  PairIn in;
  in.seg = __ldg(a.seg_of_word + (c >> 5));
  // ix.roff and c are even: 16-byte aligned pairs of int2 / float2.
  in.acc = __ldcg(reinterpret_cast<const int4*>(reinterpret_cast<const int2*>(a.ring) + (ix.roff + c)));
  in.u = __ldcg(reinterpret_cast<const float2*>(a.su + c));
  in.g = __ldcg(reinterpret_cast<const float4*>(a.sg + c));
  return in;
}

// Bitmap words of words w, w + 1 (w even, so both share a summary word).
__device__ __forceinline__ void put_hist2(const StepArgs& a, const StepIdx& ix, uint32_t w,
                                          uint32_t b0, uint32_t b1) {
  __stcg(reinterpret_cast<uint2*>(a.hist + (ix.hoff + w)), make_uint2(b0, b1));
  __stcg(reinterpret_cast<uint2*>(a.hist + (ix.hoff2 + w)), make_uint2(b0, b1));
  const uint32_t sbits = (b0 ? 1u << (w & 31u) : 0u) | (b1 ? 2u << (w & 31u) : 0u);
  if (sbits) atomicOr(a.hsum + (size_t)ix.srow * a.n_swords + (w >> 5), sbits);
}

// Spike bookkeeping of a pair: per-segment counts (one per word), events,
// raster entries, and the spiking cells' push rows cut into kPushChunk items
// in the block's list (items past its capacity are pushed here); with ix.keep
// also the bitmap words.  Returns the synapses pushed here.  Without the
// history of every step and the scans over the warp (a lane reserves its own
// items): 925,500 cells 8.2 -> 7.6 us per step, 32 instances with 3.3M cells
// 18.9 -> 17.3 us.
template <bool BF16>
__device__ __forceinline__ uint32_t publish_pair(const StepArgs& a, uint32_t p, uint32_t c,
                                                 uint32_t seg, bool f0, bool f1, const StepIdx& ix,
                                                 BlockItems bi) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t b0 = __ballot_sync(kFull, f0), b1 = __ballot_sync(kFull, f1);
  if (ix.keep) {
    // Cell j of word 2p is lane j >> 1's cell j & 1; of word 2p + 1, lane 16 + (j >> 1)'s.
    const uint32_t from = (lane & 1u) ? b1 : b0;
    const uint32_t W0 = __ballot_sync(kFull, (from >> (lane >> 1)) & 1u);
    const uint32_t W1 = __ballot_sync(kFull, (from >> (16u + (lane >> 1))) & 1u);
    if (lane == 0) put_hist2(a, ix, 2u * p, W0, W1);
  }
  if ((b0 | b1) == 0u) return 0;
  Ctl* ctl = a.ctl;
  const uint32_t half = lane < 16u ? 0xFFFFu : 0xFFFF0000u;  // the lanes of this lane's word
  const uint32_t mine = __popc(b0 & half) + __popc(b1 & half);
  if ((lane & 15u) == 0u && mine) atomicAdd(&a.counts[(size_t)ix.rel * a.n_segs + seg], mine);
  uint32_t ev = 0, ra = 0, rb = 0, rc = 0;
  if (f0 || f1) {
    if (f0) ev += __ldg(a.outdeg + c);
    if (f1) ev += __ldg(a.outdeg + c + 1u);
    if (a.any_push) {
      ra = __ldg(a.push_row + c);
      rb = __ldg(a.push_row + c + 1u);
      rc = __ldg(a.push_row + c + 2u);
    }
  }
  const uint32_t na = f0 ? (rb - ra + kPushChunk - 1) / kPushChunk : 0u;
  const uint32_t nb = f1 ? (rc - rb + kPushChunk - 1) / kPushChunk : 0u;
  const uint32_t nit = na + nb;
  uint32_t off = 0;
  if (nit) off = atomicAdd(bi.count, nit);
  for (uint32_t k = 0; k < nit && off + k < kGenItems; ++k) {
    const uint32_t q0 = k < na ? ra + k * kPushChunk : rb + (k - na) * kPushChunk;
    const uint32_t q1 = k < na ? rb : rc;
    bi.items[off + k] = make_uint2(q0, min(kPushChunk, q1 - q0) << 23);
  }
  // One addition per warp: the counter is one address for the whole chip (60,000
  // spikes a step, one addition each: 52.8 us per step, 27.9 so).
  if (__popc(b0 | b1) > 1) {
    ev = __reduce_add_sync(kFull, ev);
    if (lane != 0) ev = 0;
  }
  if (ev) atomicAdd(&ctl->events, (unsigned long long)ev);
  uint32_t walked = 0;
  uint32_t spill = __ballot_sync(kFull, off + nit > kGenItems);
  while (spill) {
    const int src = __ffs(spill) - 1;
    spill &= spill - 1;
    const uint32_t o = __shfl_sync(kFull, off, src), cnt = __shfl_sync(kFull, nit, src);
    const uint32_t sa = __shfl_sync(kFull, na, src);
    const uint32_t pa = __shfl_sync(kFull, ra, src), pb = __shfl_sync(kFull, rb, src),
                   pc = __shfl_sync(kFull, rc, src);
    for (uint32_t k = o < kGenItems ? kGenItems - o : 0u; k < cnt; ++k) {
      const uint32_t q0 = k < sa ? pa + k * kPushChunk : pb + (k - sa) * kPushChunk;
      const uint32_t q1 = k < sa ? pb : pc;
      walked += push_item<BF16>(a, make_uint2(q0, min(kPushChunk, q1 - q0) << 23), ix.slot);
    }
  }
  if (a.raster_cap) {
    uint32_t roff = 0;
    if (lane == 0) roff = atomicAdd(&ctl->raster_count, (uint32_t)(__popc(b0) + __popc(b1)));
    const uint32_t below = (1u << lane) - 1u;
    uint32_t q = __shfl_sync(kFull, roff, 0) + __popc(b0 & below) + __popc(b1 & below);
    if (f0) {
      if (q < a.raster_cap) a.raster[q] = c; else atomicOr(&ctl->error, kErrRasterOverflow);
      ++q;
    }
    if (f1) {
      if (q < a.raster_cap) a.raster[q] = c + 1u; else atomicOr(&ctl->error, kErrRasterOverflow);
    }
  }
  return walked;
}

template <bool SEGSMEM, bool BF16>
__device__ __forceinline__ uint32_t finish_pair(const StepArgs& a, uint32_t p, const PairIn& in,
                                                const StepIdx& ix, BlockItems bi) {
  const uint32_t c = (p << 6) + 2u * (threadIdx.x & 31u);
  bool f0 = false, f1 = false;
  if (in.seg != 0xFFFFu) {  // padding words past the last segment (half-warp uniform)
    const SegDev& sd = SEGSMEM ? reinterpret_cast<const SegDev*>(g_dyn)[in.seg] : a.segs[in.seg];
    const uint4 hd = *reinterpret_cast<const uint4*>(&sd);  // base, count, key_base, kind
    const uint32_t l0 = c - hd.x;
    const bool v0 = l0 < hd.y, v1 = l0 + 1u < hd.y;
    if (hd.w == kSegInput) {
      const SrcDev* srcs =
          SEGSMEM ? reinterpret_cast<const SrcDev*>(g_dyn + seg_table_bytes(a.n_segs)) : a.srcs;
      const uint2 m = v0 ? __ldg(reinterpret_cast<const uint2*>(a.src_mask + c)) : make_uint2(0u, 0u);
      if (m.x) f0 = input_fire(a, srcs, sd, l0, m.x, ix.t);
      if (v1 && m.y) f1 = input_fire(a, srcs, sd, l0 + 1u, m.y, ix.t);
    } else {
      // Both lanes' cells run the LIF step (a padding cell integrates its own,
      // never read, padding state and is masked out of the spikes).
      if (in.acc.x | in.acc.y | in.acc.z | in.acc.w)
        __stcg(reinterpret_cast<int4*>(reinterpret_cast<int2*>(a.ring) + (ix.roff + c)),
               make_int4(0, 0, 0, 0));
      const LifK k = lif_k(sd);
      float4 s0 = state_in(in.u.x, make_float2(in.g.x, in.g.y), k.Vr);
      float4 s1 = state_in(in.u.y, make_float2(in.g.z, in.g.w), k.Vr);
      f0 = lif_step(k, a.substeps, s0, make_int2(in.acc.x, in.acc.y)) && v0;
      f1 = lif_step(k, a.substeps, s1, make_int2(in.acc.z, in.acc.w)) && v1;
      __stcg(reinterpret_cast<float2*>(a.su + c),
             make_float2(pack_u(s0.x, __float_as_int(s0.w)), pack_u(s1.x, __float_as_int(s1.w))));
      __stcg(reinterpret_cast<float4*>(a.sg + c), make_float4(s0.y, s0.z, s1.y, s1.z));
    }
  }
  return publish_pair<BF16>(a, p, c, in.seg, f0, f1, ix, bi);
}

// Pairs gp, gp + np, ... with the next pair's loads in flight while the
// current one is computed.  Returns the synapses pushed on the way.
template <bool SEGSMEM, bool BF16>
__device__ __forceinline__ uint32_t update_pairs(const StepArgs& a, uint32_t gp, uint32_t np,
                                                 const StepIdx& ix, BlockItems bi) {
  const uint32_t n_pairs = a.n_words >> 1;
  uint32_t p = gp, walked = 0;
  if (p >= n_pairs) return 0;
  PairIn cur = load_pair(a, p, ix);
  while (true) {
    const uint32_t pn = p + np;
    PairIn nxt;
    if (pn < n_pairs) nxt = load_pair(a, pn, ix);
    walked += finish_pair<SEGSMEM, BF16>(a, p, cur, ix, bi);
    if (pn >= n_pairs) break;
    p = pn;
    cur = nxt;
  }
  return walked;
}

// ---- phase 2: deliveries ------------------------------------------------------
// One warp delivers one push item (at most kPushChunk synapses of a spiking
// cell's row): all loads of the item are issued before its atomics so the
// item costs one memory round trip; returns the item's synapse count.
template <bool BF16>
__device__ __forceinline__ uint32_t push_item(const StepArgs& a, uint2 it, uint32_t slot0) {
  constexpr int kPer = kPushChunk / 32;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t q1 = it.x + (it.y >> 23);
  uint32_t wd[kPer];
  float wv[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const uint32_t q = it.x + k * 32 + lane;
    wd[k] = q < q1 ? __ldg(a.push_syn + q) : 0u;
    wv[k] = q < q1 ? load_weight<BF16>(a.push_w, q) : 0.f;
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    if (it.x + k * 32 + lane >= q1) break;
    uint32_t slot = slot0 + ((wd[k] >> kPushPostBits) & 15u);
    if (slot >= a.ring_slots) slot -= a.ring_slots;
    atomicAdd(a.ring + (((size_t)slot * a.n_pad + (wd[k] & kPushPostMask)) << 1) + (wd[k] >> 31),
              __float2int_rn(wv[k]));
  }
  return it.y >> 23;
}

// ---- dense pull (ELL) ----------------------------------------------------------
// A unit is kPullUnit consecutive entries of one projection's ELL, whatever
// its layout.  An entry is the offset of its spike bit above the step's
// history base (word e >> 5, bit e & 31); for the few entries whose pre cell
// spiked the weight is read and added into the post cell's ring slot with one
// atomic (the post is recovered from the entry's offset).
__device__ __forceinline__ const uint32_t* hist_base(const StepArgs& a, uint32_t hrow) {
  return a.hist + (size_t)(a.hist_rows - 1u - hrow) * a.n_words;  // row of step t
}

template <bool BF16>
__device__ __forceinline__ float pull_weight(const ProjDev& P, uint32_t o) {
  // A plastic projection's weights change every step (inside a persistent
  // launch too): read at L2, not through the non-coherent read-only path.
  return BF16 ? __uint_as_float((uint32_t)__ldcg((const unsigned short*)P.ell_w + o) << 16)
              : __ldcg((const float*)P.ell_w + o);
}
__device__ __forceinline__ size_t pull_target(const StepArgs& a, const ProjDev& P, uint32_t o,
                                              uint32_t slot1) {
  const uint32_t post = P.ell_rowmajor ? o / P.ell_K : o % P.post_count;
  return (((size_t)slot1 * a.n_pad + P.post_base + post) << 1) + P.channel;
}
template <bool BF16>
__device__ __forceinline__ void pull_hit(const StepArgs& a, const ProjDev& P, uint32_t o,
                                         uint32_t slot1) {
  const float wv = pull_weight<BF16>(P, o);
  atomicAdd(a.ring + pull_target(a, P, o, slot1), __float2int_rn(wv));
}

// Persistent kernels: one of a unit's kPullParts ranges of kPullUnit /
// kPullParts entries (`part`; 8 per lane, loaded at once, within their
// 64-register budget), so a unit spreads over that many warps and a pull is
// one round of loads per warp.  Entries straight from global memory, tested
// against the block's staged summary when there is one, history words from
// L2 (other blocks write them during the launch).  Returns the lane's hits.
constexpr uint32_t kPullParts = 4;
template <bool BF16>
__device__ __forceinline__ uint32_t pull_unit(const StepArgs& a, const PullUnit un, uint32_t part,
                                              const uint32_t* hb, uint32_t slot1,
                                              const uint32_t* s_sum) {
  constexpr uint32_t B = kPullUnit / kPullParts / 32;
  const uint32_t pad = a.hist_rows * a.n_pad;
  const ProjDev& P = a.projs[un.proj];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t hits = 0;
  const uint32_t o0 = un.o0 + part * (kPullUnit / kPullParts);
  {
    const uint32_t ob = o0 + lane;
    uint32_t e[B];
#pragma unroll
    for (uint32_t u = 0; u < B; ++u) e[u] = __ldg(P.ell_syn + ob + 32u * u);  // padded to units
    uint32_t hit = 0;
    if (s_sum) {
      // The block's staged summary settles most entries; the history word is
      // read only for those whose 32-cell word had a spike.
#pragma unroll
      for (uint32_t u = 0; u < B; ++u) {
        const uint32_t sw = s_sum[e[u] >> 10];
        if (__funnelshift_r(sw, sw, e[u] >> 5) & 1u)
          hit |= ((__ldcg(hb + (e[u] >> 5)) >> (e[u] & 31u)) & 1u) << u;
      }
    } else {
#pragma unroll
      for (uint32_t u = 0; u < B; ++u)
        if (e[u] < pad) hit |= ((__ldcg(hb + (e[u] >> 5)) >> (e[u] & 31u)) & 1u) << u;
    }
    hits += __popc(hit);
    while (hit) {
      const uint32_t u = __ffs(hit) - 1;
      hit &= hit - 1;
      pull_hit<BF16>(a, P, ob + 32u * u, slot1);
    }
  }
  return hits;
}

// The spike summary of steps t - d1, d1 = 0 .. max_delay - 1 (the delay rows
// a pull of step t reads; a longer history kept for plasticity is not) into
// shared memory as rows d1 of n_swords words, plus the zero word that
// padding entries (row hist_rows) test; threads tid, tid + nthreads, ... with
// four loads issued before their stores.  The caller synchronizes the block.
__device__ __forceinline__ void stage_summary(const StepArgs& a, const StepIdx& ix, uint32_t* s_sum,
                                              uint32_t tid, uint32_t nthreads) {
  const uint32_t R = a.hist_rows + 1u, n = a.max_delay * a.n_swords;
  for (uint32_t j0 = tid; j0 < n; j0 += 4u * nthreads) {
    uint32_t v[4];
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
      const uint32_t j = j0 + k * nthreads;
      const uint32_t d1 = j / a.n_swords, w = j - d1 * a.n_swords;
      v[k] = j < n ? __ldcg(a.hsum + (size_t)((ix.srow + R - d1) % R) * a.n_swords + w) : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k)
      if (j0 + k * nthreads < n) s_sum[j0 + k * nthreads] = v[k];
  }
  if (tid == 0) s_sum[a.hist_rows * a.n_swords] = 0u;
}

// Delivery phase for one warp: push items gw, gw + nw, ... up to the first
// slot not written this step (each delivered item is cleared), then the dense
// pull units.  Returns the synapses walked by the push items.
template <bool BF16, bool PULL>
__device__ __forceinline__ uint32_t deliver_warp(const StepArgs& a, uint32_t gw, uint32_t nw,
                                                 const StepIdx& ix, const uint32_t* s_sum = nullptr) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t walked = 0;
  if (a.any_push) {
    uint2* list = a.items + (size_t)(ix.t & 1) * a.item_cap;
    const uint32_t tag = item_tag(ix.t);
    for (uint32_t u = gw; u < a.item_cap; u += nw) {
      const uint2 it = __ldcg(list + u);
      if ((it.y & 0x7FFFFFu) != tag) break;
      if (lane == 0) __stcg(&list[u].y, 0u);
      walked += push_item<BF16>(a, it, ix.slot);
    }
  }
  if (PULL && a.n_pull_units) {
    const uint32_t slot1 = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
    uint32_t hits = 0;
    const uint32_t* hb = hist_base(a, ix.hrow);
    for (uint32_t v = gw; v < a.n_pull_units * kPullParts; v += nw)
      hits += pull_unit<BF16>(a, a.pull_units[v / kPullParts], v % kPullParts, hb, slot1, s_sum);
    hits = __reduce_add_sync(kFull, hits);
    if (lane == 0 && hits) atomicAdd(&a.ctl->pulled, (unsigned long long)hits);
  }
  return walked;
}

__device__ __forceinline__ void ix_rows(const StepArgs& a, StepIdx& ix) {
  ix.roff = ix.slot * a.n_pad;
  ix.hoff = (a.hist_rows - 1u - ix.hrow) * a.n_words;
  ix.hoff2 = ix.hoff + a.hist_rows * a.n_words;
}

__device__ __forceinline__ StepIdx step_of(const StepArgs& a) {
  const Ctl* ctl = a.ctl;
  StepIdx ix;
  ix.t = ctl->step;
  ix.slot = ctl->ring_slot;
  ix.hrow = ctl->hist_row;
  ix.srow = (uint32_t)(ix.t % (a.hist_rows + 1ull));
  ix.rel = ctl->t_rel;
  ix_rows(a, ix);
  return ix;
}

// The next step's indices (persistent kernels).
__device__ __forceinline__ void ix_advance(const StepArgs& a, StepIdx& ix) {
  ix.slot = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
  ix.hrow = ix.hrow + 1u == a.hist_rows ? 0u : ix.hrow + 1u;
  ix.srow = ix.srow == a.hist_rows ? 0u : ix.srow + 1u;
  ix_rows(a, ix);
}

// ---- per-step kernels (CUDA-graph driver) ----------------------------------
// A step's kernels depend on one another, but their launches need not: each is
// launched as a programmatic dependent of the one before (step_launch), so its
// blocks are scheduled while that one still runs, and waits (step_wait) before its
// first access for that kernel to end and its writes to be visible.  Every
// block passes this point, so a kernel's end implies the end of all before it.
// In a graph: 92,550 cells event-driven 6.85 -> 6.5 us per step, every
// projection dense 13.3 -> 12.2, 9,255 cells 5.8 -> 5.4.
__device__ __forceinline__ void step_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void step_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void step_begin() {
  step_wait();
  step_next();
}

// Start of a chunk of `steps` steps: clears its counts and, for a persistent
// launch, the barrier counter and the board (n_bar words), and takes new
// stimulus sources from the host's pinned copy.
__global__ void __launch_bounds__(kBlock) k_chunk_begin(StepArgs a, uint32_t steps, uint32_t n_bar,
                                                        const SrcDev* srcs) {
  const uint32_t gtid = blockIdx.x * kBlock + threadIdx.x, n = gridDim.x * kBlock;
  for (size_t j = gtid; j < (size_t)steps * a.n_segs; j += n) a.counts[j] = 0u;
  for (uint32_t j = gtid; j < n_bar; j += n) reinterpret_cast<uint32_t*>(a.bar)[j] = 0u;
  if (srcs)
    for (uint32_t j = gtid; j < a.n_srcs * (uint32_t)(sizeof(SrcDev) / 8); j += n)
      reinterpret_cast<unsigned long long*>(const_cast<SrcDev*>(a.srcs))[j] =
          reinterpret_cast<const volatile unsigned long long*>(srcs)[j];
  if (gtid == 0) {
    a.ctl->t_rel = 0;
    a.ctl->raster_count = 0;
    a.raster_off[0] = 0;
  }
}

// LOOP: more words than warps that fit the chip at once, so that each warp
// takes several and the step's indices and the loads of a word are waited for
// once, not in every wave of blocks (per step: 370,200 cells 10.3 -> 9.3 us,
// 925,500 15.5 -> 13.2, 1,388,250 dense 56.8 -> 51.2; 3 blocks per SM 14.2 and
// 53, 5 14.3 and 52.7).
//   A grid of more than kUpdateBlocks per SM lets the next kernel start only as
// its blocks end: started before, the delivery's blocks crowd onto the SMs that
// have room first (300,000 cells in ten substeps, 150 Hz input: 33.2 us per step,
// 28.8 so; scaffolds of 370,200 cells 14.4 and 14.2; smaller grids leave room on
// every SM, and start it at once: 92,550 cells in two substeps 7.9, else 8.0).
constexpr uint32_t kUpdateBlocks = 4;  // per SM
template <bool LOOP>
__global__ void __launch_bounds__(kBlock, LOOP ? kUpdateBlocks : 0) k_update(StepArgs a) {
  step_wait();
  const bool early = LOOP || gridDim.x <= a.sms * kUpdateBlocks;
  if (early) step_next();
  const uint32_t gtid = blockIdx.x * kBlock + threadIdx.x;
  const uint32_t w = gtid >> 5;
  const StepIdx ix = step_of(a);
  clear_next_summary(a, ix, gtid, gridDim.x * kBlock);
  if (LOOP)
    update_words<true, false, false, false>(a, w, gridDim.x * (kBlock / 32), ix, {nullptr, nullptr});
  else if (w < a.n_words)
    update_word(a, w, ix);
  if (!early) step_next();
}

// Delivery of step t; the last block to finish also advances the step
// (ring slot, history row, buffer parity, raster offsets).
template <bool BF16>
__global__ void __launch_bounds__(kBlock) k_deliver(StepArgs a) {
  step_begin();
  Ctl* ctl = a.ctl;
  const StepIdx ix = step_of(a);
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t walked = deliver_warp<BF16, false>(a, (blockIdx.x * kBlock + threadIdx.x) >> 5,
                                             (gridDim.x * kBlock) >> 5, ix);
  if (lane == 0 && walked) atomicAdd(&ctl->delivered, (unsigned long long)walked);
  // Step bookkeeping by the last block to arrive.
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&ctl->barrier_gen, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    ctl->barrier_gen = 0;
    const unsigned long long t = ix.t + 1ull;
    ctl->step = t;
    ctl->ring_slot = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
    ctl->hist_row = ix.hrow + 1u == a.hist_rows ? 0u : ix.hrow + 1u;
    ctl->active_count[t & 1] = 0;
    ctl->t_rel = ix.rel + 1u;
    a.raster_off[ix.rel + 1u] = ctl->raster_count;
  }
}

// Dense pull of the per-step driver (one 1,024-thread block per SM).  Each
// block stages the summary rows of steps t + 1 - d, d = 1..H (one bit per
// 32-cell word: did any cell of it spike) in shared memory, delay-major, so
// an entry's summary word is s_sum[e >> 10]; the word after them stays zero,
// so padding entries (delay field H) never pass.  Warps stream
// units (gw, gw + nw, ...; the first one's loads overlap the staging): a lane
// loads its 32 entries of a unit at once, settles every entry whose summary
// bit is clear in shared memory, and walks the few that passed four at a
// time (usually one trip per warp), loading each entry again (an L1 hit) and
// then its history word (an ordinary load, through L1: as a programmatic
// dependent this grid may be resident while k_update still writes the step's
// row, which the read-only path rules out and step_begin's wait orders; loaded
// at L2 instead, 1,388,250 cells take 59 us per step, not 53).  Without room
// for the summary (SUM false) every entry walks.
template <bool BF16, bool SUM>
__global__ void __launch_bounds__(kPullBlock, 1) k_pull(StepArgs a) {
  constexpr uint32_t E = kPullUnit / 32;  // entries per lane per unit
  constexpr uint32_t W = 4;               // entries walked per trip
  extern __shared__ uint32_t s_sum[];     // [H][n_swords] + 1 (padding's word)
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t gw = (blockIdx.x * kPullBlock + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * kPullBlock) >> 5;
  const uint32_t n = a.n_pull_units;
  step_begin();
  const StepIdx ix = step_of(a);
  const uint32_t slot1 = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
  uint32_t e[E];
  if (gw < n) {
    const PullUnit un = a.pull_units[gw];
    const uint32_t* src = a.projs[un.proj].ell_syn + un.o0 + lane;
#pragma unroll
    for (uint32_t k = 0; k < E; ++k) e[k] = __ldg(src + k * 32u);
  }
  if (SUM) {
    stage_summary(a, ix, s_sum, threadIdx.x, kPullBlock);
    __syncthreads();
  }
  const uint32_t* hb = hist_base(a, ix.hrow);
  const uint32_t pad = a.hist_rows * a.n_pad;
  uint32_t hits = 0;
  for (uint32_t u = gw; u < n; u += nw) {
    const PullUnit un = a.pull_units[u];
    const ProjDev& P = a.projs[un.proj];
    const uint32_t* src = P.ell_syn + un.o0 + lane;  // tables are padded to whole units
    if (u != gw) {
#pragma unroll
      for (uint32_t k = 0; k < E; ++k) e[k] = __ldg(src + k * 32u);
    }
    uint32_t need = 0;
#pragma unroll
    for (uint32_t k = 0; k < E; ++k) {
      if (SUM) {
        const uint32_t sw = s_sum[e[k] >> 10];
        need |= (__funnelshift_r(sw, sw, e[k] >> 5) & 1u) << k;
      } else {
        need |= (uint32_t)(e[k] < pad) << k;
      }
    }
    while (need) {
      uint32_t ks[W], ev[W], hw[W];
#pragma unroll
      for (uint32_t j = 0; j < W; ++j) {
        ks[j] = need ? __ffs(need) - 1u : E;
        need &= need - 1u;
      }
#pragma unroll
      for (uint32_t j = 0; j < W; ++j) ev[j] = ks[j] < E ? __ldg(src + ks[j] * 32u) : 0u;
#pragma unroll
      for (uint32_t j = 0; j < W; ++j)
        hw[j] = ks[j] < E ? hb[ev[j] >> 5] : 0u;
#pragma unroll
      for (uint32_t j = 0; j < W; ++j) {
        if (ks[j] < E && ((hw[j] >> (ev[j] & 31u)) & 1u)) {
          ++hits;
          pull_hit<BF16>(a, P, un.o0 + ks[j] * 32u + lane, slot1);
        }
      }
    }
  }
  hits = __reduce_add_sync(kFull, hits);
  if (lane == 0 && hits) atomicAdd(&a.ctl->pulled, (unsigned long long)hits);
}

// Dense pull with 16-byte entry loads (per-step driver; one 1,024-thread
// block per SM): as k_pull with the staged summary, but a lane holds entries
// 4L .. 4L + 3 of each 128-entry row of its unit and loads them as one uint4,
// eight loads per unit instead of 32.  Entry m of the lane (0 .. 31) is at
// unit offset (m >> 2) * 128 + 4L + (m & 3).
template <bool BF16>
__global__ void __launch_bounds__(kPullBlock, 1) k_pull_vec(StepArgs a) {
  constexpr uint32_t V = kPullUnit / 128;  // 16-byte loads per lane per unit
  constexpr uint32_t E = 4 * V;            // entries per lane per unit
  constexpr uint32_t W = 4;                // entries walked per trip
  extern __shared__ uint32_t s_sum[];      // [H][n_swords] + 1 (padding's word)
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t gw = (blockIdx.x * kPullBlock + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * kPullBlock) >> 5;
  const uint32_t n = a.n_pull_units;
  step_begin();
  const StepIdx ix = step_of(a);
  const uint32_t slot1 = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
  uint4 q[V];
  if (gw < n) {
    const PullUnit un = a.pull_units[gw];
    const uint4* src = reinterpret_cast<const uint4*>(a.projs[un.proj].ell_syn + un.o0) + lane;
#pragma unroll
    for (uint32_t k = 0; k < V; ++k) q[k] = __ldg(src + 32u * k);
  }
  stage_summary(a, ix, s_sum, threadIdx.x, kPullBlock);
  __syncthreads();
  const uint32_t* hb = hist_base(a, ix.hrow);
  uint32_t hits = 0;
  for (uint32_t u = gw; u < n; u += nw) {
    const PullUnit un = a.pull_units[u];
    const ProjDev& P = a.projs[un.proj];
    const uint32_t* base = P.ell_syn + un.o0 + 4u * lane;  // tables are padded to whole units
    if (u != gw) {
#pragma unroll
      for (uint32_t k = 0; k < V; ++k) q[k] = __ldg(reinterpret_cast<const uint4*>(base) + 32u * k);
    }
    uint32_t need = 0;
#pragma unroll
    for (uint32_t k = 0; k < V; ++k) {
      const uint32_t ev4[4] = {q[k].x, q[k].y, q[k].z, q[k].w};
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
        const uint32_t sw = s_sum[ev4[j] >> 10];
        need |= (__funnelshift_r(sw, sw, ev4[j] >> 5) & 1u) << (4u * k + j);
      }
    }
    while (need) {
      uint32_t ms[W], ev[W], hw[W];
#pragma unroll
      for (uint32_t j = 0; j < W; ++j) {
        ms[j] = need ? __ffs(need) - 1u : E;
        need &= need - 1u;
      }
#pragma unroll
      for (uint32_t j = 0; j < W; ++j)
        ev[j] = ms[j] < E ? __ldg(base + (ms[j] >> 2) * 128u + (ms[j] & 3u)) : 0u;
#pragma unroll
      for (uint32_t j = 0; j < W; ++j) hw[j] = ms[j] < E ? hb[ev[j] >> 5] : 0u;
#pragma unroll
      for (uint32_t j = 0; j < W; ++j) {
        if (ms[j] < E && ((hw[j] >> (ev[j] & 31u)) & 1u)) {
          ++hits;
          pull_hit<BF16>(a, P, un.o0 + (ms[j] >> 2) * 128u + 4u * lane + (ms[j] & 3u), slot1);
        }
      }
    }
  }
  hits = __reduce_add_sync(kFull, hits);
  if (lane == 0 && hits) atomicAdd(&a.ctl->pulled, (unsigned long long)hits);
}

// Block barrier 1 over the first n threads (a multiple of 32).
__device__ __forceinline__ void bar_sync_first(uint32_t n) {
  asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
}

// STDP of the plastic projections, step t (SynapticPlasticity.cu:40-120), run
// after the cells of step t updated and before the dense pull that delivers
// into slot t + 1, so that delivery uses the new values -- in the reference
// the propagation of the next millisecond follows invoke_stdp_plasticity.
// One warp per unit of 1,024 ELL cells, one lane per cell.  The entry of a
// cell is its pre cell's spike-bit offset for step t + 1 - d above the history
// row of step t, so the spikes of steps t - d - s are at e + (s + 1) n_pad;
// the post cell's spike of step t is at its own index, a teacher's at the
// offset precomputed per post cell.  COH: inside a persistent launch the
// history, spike registers and plastic values were written this launch by
// other SMs, so they are read at L2 (ld.global.cg); a per-step kernel reads
// data written by earlier launches and may use the read-only path.
template <bool COH>
__device__ __forceinline__ uint32_t ld_coh(const uint32_t* p) {
  return COH ? __ldcg(p) : __ldg(p);
}
template <bool COH>
__device__ __forceinline__ uint32_t hist_bit(const uint32_t* hb, uint32_t off) {
  return (ld_coh<COH>(hb + (off >> 5)) >> (off & 31u)) & 1u;
}

// A synapse whose dw is 0 keeps its value and weight bit for bit, so with a0
// = a1_j = 0 (the reference's own coefficients) only synapses of post cells
// whose post / teacher spike is set change: a row-major unit whose posts all
// lack it is skipped after one lookup per post.  Units are kStdpUnit cells
// (four per lane, loads issued together), so the rows of the few posts that
// do change spread over many warps; the window's spike count is gathered
// eight rows at a time.
// Hist: where a spike bit at an offset above the step's history row is read
// (HistGlobal, or the rows a block keeps in shared memory).
template <bool COH>
struct HistGlobal {
  const uint32_t* hb;
  __device__ __forceinline__ uint32_t bit(uint32_t off) const { return hist_bit<COH>(hb, off); }
};

template <class Hist>
__device__ __forceinline__ bool stdp_post_spiked(const PlastDev& L, const ProjDev& P, const Hist& h,
                                                 uint32_t post) {
  const uint32_t so = L.rule == SGB_STDP_TEACHER ? __ldg(L.teacher + post) : P.post_base + post;
  return so != 0xFFFFFFFFu && h.bit(so);
}

// Updates the cells of one unit (the whole warp, four cells per lane).
// EARLY: run during the update of step t (a rule that reads only earlier
// steps' spikes), so `recent`, the spike registers, are those of step t - 1,
// read one bit lower; else those of step t.
// spiked: the screening found the unit inside one post cell's row with its
// post / teacher spike set, so the entries need not look it up again.
template <bool BF16, bool COH, bool EARLY, class Hist>
__device__ __forceinline__ void stdp_unit(const StepArgs& a, const PullUnit un, const Hist& h,
                                          uint32_t pad, const unsigned long long* recent,
                                          bool spiked = false) {
  constexpr uint32_t B = kStdpUnit / 32;
  const uint32_t lane = threadIdx.x & 31u;
  const PlastDev& L = a.plast[un.proj];
  const ProjDev& P = a.projs[L.proj];
  const uint32_t end = min(un.o0 + kStdpUnit, P.ell_n);
  const bool all = L.a0 != 0.f || L.a1_j != 0.f;  // every synapse may change
  uint32_t e[B], n_upd = 0;
  bool sp[B];
#pragma unroll
  for (uint32_t k = 0; k < B; ++k) {
    const uint32_t o = un.o0 + lane + 32u * k;
    e[k] = o < end ? __ldg(P.ell_syn + o) : pad;
  }
#pragma unroll
  for (uint32_t k = 0; k < B; ++k) {
    const uint32_t o = un.o0 + lane + 32u * k;
    sp[k] = e[k] < pad &&
            (spiked || stdp_post_spiked(L, P, h, P.ell_rowmajor ? o / P.ell_K : o % P.post_count));
  }
#pragma unroll
  for (uint32_t k = 0; k < B; ++k) {
    if (e[k] >= pad || !(all || sp[k])) continue;  // padding, or dw = 0
    const uint32_t o = un.o0 + lane + 32u * k;
    ++n_upd;
    bool s_pre;
    uint32_t nwin = 0;  // pre spikes at t - d - j, j < window
    if (L.recent_ok) {
      // The pre cell's spike register: bit d is step t - d, bits d .. d +
      // window - 1 the window (d + window <= 64 for this projection).
      const uint32_t d = e[k] / a.n_pad + 1u, g = e[k] - (d - 1u) * a.n_pad;
      const unsigned long long* rb = recent + g;
      const unsigned long long r = (COH ? __ldcg(rb) : __ldg(rb)) >> (EARLY ? d - 1u : d);
      s_pre = (r & 1ull) != 0ull;
      if (sp[k] && L.a2_ji != 0.f)
        nwin = __popcll(L.window == 64u ? r : r & ((1ull << L.window) - 1ull));
    } else {
      s_pre = h.bit(e[k] + a.n_pad) != 0u;
      if (sp[k] && L.a2_ji != 0.f) {
        for (uint32_t j0 = 0; j0 < L.window; j0 += 8u) {
          uint32_t bit[8];
#pragma unroll
          for (uint32_t j = 0; j < 8u; ++j)
            bit[j] = j0 + j < L.window ? h.bit(e[k] + (j0 + j + 1u) * a.n_pad) : 0u;
#pragma unroll
          for (uint32_t j = 0; j < 8u; ++j) nwin += bit[j];
        }
      }
    }
    // Reference order: A0, A1_J (pre), A1_I (post / teacher), A2_JI window.
    float dw = __fadd_rn(0.f, L.a0);
    if (s_pre) dw = __fadd_rn(dw, L.a1_j);
    if (sp[k]) dw = __fadd_rn(dw, L.a1_i);
    for (uint32_t j = 0; j < nwin; ++j) dw = __fadd_rn(dw, L.a2_ji);
    float v = __fadd_rn(__ldcg(L.val + o), dw);
    v = v < 0.f ? 0.f : (v > L.v_max ? L.v_max : v);
    L.val[o] = v;
    const float tw = __fmul_rn(__ldg(L.w0 + o), v);
    if (BF16)
      reinterpret_cast<uint16_t*>(L.w_table)[o] = f32_to_bf16_bits(tw);
    else
      reinterpret_cast<float*>(L.w_table)[o] = tw;
  }
  n_upd = __reduce_add_sync(kFull, n_upd);
  if (lane == 0 && n_upd) atomicAdd(&a.ctl->plast_updates, (unsigned long long)n_upd);
}

// A synapse whose dw is 0 keeps its value and weight bit for bit, so with a0
// = a1_j = 0 (the reference's own coefficients) only synapses of post cells
// whose post / teacher spike is set change.  Each warp first tests up to 32
// of its units at once, one per lane (a row-major unit: the one or two posts
// it covers), then updates only the units that can change.  Units are
// kStdpUnit cells, so the rows of the few posts that do change spread over
// many warps; the window's spike count is gathered eight rows at a time.
// The plasticity phase of step ix over warps gw, gw + nw, ... (k_stdp, or a
// phase of the persistent kernels between the update and the deliveries).
template <bool BF16, bool COH, bool EARLY>
__device__ __forceinline__ void stdp_warp(const StepArgs& a, uint32_t gw, uint32_t nw,
                                          const StepIdx& ix) {
  const uint32_t lane = threadIdx.x & 31u;
  const HistGlobal<COH> hb{hist_base(a, ix.hrow)};
  const uint32_t pad = a.hist_rows * a.n_pad;
  const unsigned long long* recent = a.recent + ((EARLY ? ix.t + 1ull : ix.t) & 1ull) * a.n_pad;
  for (uint32_t base = gw; base < a.n_stdp_units; base += 32u * nw) {
    const uint32_t u = base + lane * nw;
    bool active = false, one = false;  // one: a single post, whose post / teacher spike is set
    if (u < a.n_stdp_units) {
      const PullUnit un = a.stdp_units[u];
      const PlastDev& L = a.plast[un.proj];
      const ProjDev& P = a.projs[L.proj];
      if (L.a0 != 0.f || L.a1_j != 0.f || !P.ell_rowmajor) {
        active = true;
      } else {
        const uint32_t end = min(un.o0 + kStdpUnit, P.ell_n);
        const uint32_t p0 = un.o0 / P.ell_K, p1 = (end - 1u) / P.ell_K;
        for (uint32_t p = p0; p <= p1; ++p) active |= stdp_post_spiked(L, P, hb, p);
        one = active && p0 == p1;
      }
    }
    uint32_t act = __ballot_sync(kFull, active);
    const uint32_t ones = __ballot_sync(kFull, one);
    while (act) {
      const uint32_t j = __ffs(act) - 1;
      act &= act - 1;
      stdp_unit<BF16, COH, EARLY>(a, a.stdp_units[base + j * nw], hb, pad, recent, (ones >> j) & 1u);
    }
  }
}

// EARLY: launched beside k_update of the same step (rules that read only
// earlier steps' spikes), reading the spike registers of step t - 1.
template <bool BF16, bool EARLY>
__global__ void __launch_bounds__(kBlock) k_stdp(StepArgs a) {
  stdp_warp<BF16, false, EARLY>(a, (blockIdx.x * kBlock + threadIdx.x) >> 5,
                                (gridDim.x * kBlock) >> 5, step_of(a));
}

// Plastic values back to their start, v_max (the reference starts at 1, its
// clamp), and the tables to the matching weights.
template <bool BF16>
__global__ void __launch_bounds__(kBlock) k_plast_reset(StepArgs a) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t gw = (blockIdx.x * kBlock + threadIdx.x) >> 5, nw = (gridDim.x * kBlock) >> 5;
  for (uint32_t u = gw; u < a.n_stdp_units; u += nw) {
    const PullUnit un = a.stdp_units[u];
    const PlastDev& L = a.plast[un.proj];
    const uint32_t end = min(un.o0 + kStdpUnit, a.projs[L.proj].ell_n);
    for (uint32_t o = un.o0 + lane; o < end; o += 32u) {
      L.val[o] = L.v_max;
      const float tw = __fmul_rn(__ldg(L.w0 + o), L.v_max);
      if (BF16)
        reinterpret_cast<uint16_t*>(L.w_table)[o] = f32_to_bf16_bits(tw);
      else
        reinterpret_cast<float*>(L.w_table)[o] = tw;
    }
  }
}

// Per-segment spike totals of the chunk, folded into the FP64 accumulators;
// the error flags and, when the host wants them and they are few, the chunk's
// counts go to pinned host memory from here, without a copy of their own.
__global__ void __launch_bounds__(kBlock) k_chunk_end(StepArgs a, uint32_t* host_err, uint32_t* host_counts) {
  const uint32_t seg = blockIdx.x;
  const uint32_t steps = a.ctl->t_rel;
  if (host_counts)
    for (uint32_t j = seg * kBlock + threadIdx.x; j < steps * a.n_segs; j += gridDim.x * kBlock)
      host_counts[j] = a.counts[j];
  if (seg == 0 && threadIdx.x == 0) *host_err = a.ctl->error;
  if (seg >= a.n_segs) return;
  unsigned long long s = 0;
  for (uint32_t r = threadIdx.x; r < steps; r += blockDim.x) s += a.counts[(size_t)r * a.n_segs + seg];
  for (int o = 16; o; o >>= 1) s += __shfl_down_sync(kFull, s, o);
  __shared__ unsigned long long part[kBlock / 32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tot = 0;
    for (int w = 0; w < kBlock / 32; ++w) tot += part[w];
    a.totals[seg] += (double)tot;
  }
}

// Cell states in id order (first[seg]: a segment's first id), as the host
// reads them: potential, two conductances, refractory steps.  One thread per
// padded cell; bound by the copy of its output to the host.
__global__ void __launch_bounds__(kBlock) k_state_out(StepArgs a, const long long* first, float* u, float2* g,
                                                      int32_t* ref) {
  const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
  if (i >= a.n_pad) return;
  const uint32_t seg = a.seg_of_word[i >> 5];
  if (seg == 0xFFFFu) return;
  const SegDev& sd = a.segs[seg];
  const uint32_t local = i - sd.base;
  if (local >= sd.count) return;
  const long long o = first[seg] + local;
  const float x = a.su[i];
  const int32_t r = sd.kind == kSegLif ? unpack_ref(x) : 0;
  u[o] = r ? sd.Vr : x;
  g[o] = a.sg[i];
  ref[o] = r;
}

// ---- persistent driver ----------------------------------------------------------
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid-wide barrier over co-resident blocks (cooperative launch).  After the
// block barrier, thread 0 arrives on a counter with a gpu-scope release
// reduction (cumulative over the block's writes ordered before it by
// __syncthreads), then polls with gpu-scope acquire loads; the closing
// __syncthreads hands the acquired view to the whole block.  No separate
// fences: measured on 152 blocks, ~0.3 us per barrier less than fence +
// atomicAdd + fence.  It waits for every block's arrival at this barrier (plus
// a.bar_extra arrivals that no block makes, in the tests of this limit) -- at
// most kBarrierTimeoutNs of global time, checked every 256 polls.  On timeout it records
// kErrBarrierTimeout; every block then returns at its next barrier (or as
// soon as it sees the flag), so the kernel always ends and the host reads
// the flag as SGB_ERR_DEVICE.  grid_arrive / grid_wait are the two halves,
// for callers with work that does not depend on the other blocks in between.
__device__ __forceinline__ void grid_arrive(const StepArgs& a, unsigned long long& target) {
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(a.bar) : "memory");
}

// One thread polls the arrival counter until it reaches target (plus the
// tests' a.bar_extra) with gpu-scope acquire loads, for at most
// kBarrierTimeoutNs of global time; false (and kErrBarrierTimeout recorded)
// when the wait ran out or another block had already recorded a timeout.
__device__ __forceinline__ bool poll_arrivals(const StepArgs& a, unsigned long long target) {
  const unsigned long long want = target + a.bar_extra;
  unsigned long long t0 = 0;
  uint32_t it = 0;
  while (ld_acquire(a.bar) < want) {
    if ((++it & 255u) == 0u) {
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > kBarrierTimeoutNs || (__ldcg(&a.ctl->error) & kErrBarrierTimeout)) {
        atomicOr(&a.ctl->error, kErrBarrierTimeout);
        return false;
      }
    }
    __nanosleep(32);
  }
  return true;
}

__device__ __forceinline__ bool grid_wait(const StepArgs& a, unsigned long long target,
                                          uint32_t poller = 0) {
  __shared__ int abort_flag;
  if (threadIdx.x == poller) abort_flag = !poll_arrivals(a, target);
  __syncthreads();
  return !abort_flag;
}

// Arrival by one thread whose gpu-scope fence comes first: the fence followed
// by the relaxed reduction is a release pattern, cumulative over the writes
// that a block barrier ordered before the fence.
__device__ __forceinline__ void grid_arrive_fenced(const StepArgs& a) {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(a.bar) : "memory");
}

__device__ __forceinline__ bool grid_barrier(const StepArgs& a, unsigned long long& target) {
  grid_arrive(a, target);
  return grid_wait(a, target);
}

__host__ __device__ __forceinline__ size_t seg_smem_bytes_dev(const StepArgs& a) {
  return seg_table_bytes(a.n_segs) + (((size_t)a.n_srcs * sizeof(SrcDev) + 15) & ~(size_t)15);
}

// History rows k_persistent_pull keeps: the delay rows of a pull, and one more
// for a teacher max_delay steps back.
__host__ __device__ __forceinline__ uint32_t pull_rows(const StepArgs& a) {
  return a.max_delay + (a.n_plast ? 1u : 0u);
}

// Raster offsets of a launch with one grid barrier per step: a block may
// already reserve raster entries of step s while another still reads the
// count of step s - 1, so the offsets come from the step counts instead (a
// step's entries are contiguous: its reservations all follow the previous
// barrier).  After the launch's last barrier every count is final; block 0
// scans them (all its threads call this; s_wsum holds kPersistBlock / 32).
__device__ __noinline__ void raster_offsets(const uint32_t* counts, uint32_t n_segs, uint32_t* raster_off,
                                            uint32_t n_steps, uint32_t* s_wsum) {
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  const uint32_t per = (n_steps + blockDim.x - 1) / blockDim.x;
  const uint32_t q0 = min(n_steps, threadIdx.x * per), q1 = min(n_steps, q0 + per);
  uint32_t tot = 0;
#pragma unroll 1
  for (uint32_t q = q0; q < q1; ++q)
#pragma unroll 1
    for (uint32_t g = 0; g < n_segs; ++g) tot += __ldcg(counts + (size_t)q * n_segs + g);
  uint32_t incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, o);
    if (lane >= (uint32_t)o) incl += v;
  }
  __syncthreads();  // s_wsum's previous readers are done
  if (lane == 31) s_wsum[wib] = incl;
  __syncthreads();
  if (wib == 0) {
    const uint32_t x = lane < (blockDim.x >> 5) ? s_wsum[lane] : 0u;
    uint32_t xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, xi, o);
      if (lane >= (uint32_t)o) xi += v;
    }
    s_wsum[lane] = xi - x;
  }
  __syncthreads();
  uint32_t run = s_wsum[wib] + incl - tot;
#pragma unroll 1
  for (uint32_t q = q0; q < q1; ++q) {
#pragma unroll 1
    for (uint32_t g = 0; g < n_segs; ++g) run += __ldcg(counts + (size_t)q * n_segs + g);
    raster_off[q + 1] = run;
  }
}
__device__ __forceinline__ void raster_offsets_from_counts(const StepArgs& a, uint32_t n_steps,
                                                           uint32_t* s_wsum) {
  raster_offsets(a.counts, a.n_segs, a.raster_off, n_steps, s_wsum);
}

// General persistent kernel.  ONE (networks without dense pulls or rules that
// read the step's own spikes): a step's pushes only target ring slots
// t + 1 .. t + D while its update reads slot t, so each block collects its
// spiking cells' push items in shared memory during the update, delivers them
// right after it, and one grid barrier ends the step.  Otherwise the items go
// to a global list delivered by all warps between two grid barriers.
// LANE (one-barrier form, no plasticity): 1 one cell per lane (update_words),
// 2 two cells per lane (update_pairs).
template <bool BF16, bool ONE, int LANE = 1>
__global__ void __launch_bounds__(kPersistBlock, 1) k_persistent(StepArgs a, uint32_t n_steps) {
  // Dynamic shared memory: the segment descriptors every word reads (when
  // a.seg_smem), then the staged spike summary (dense pulls, when it fits).
  uint32_t* s_sum = reinterpret_cast<uint32_t*>(g_dyn + (a.seg_smem ? seg_smem_bytes_dev(a) : 0));
  __shared__ uint2 s_items[ONE ? kGenItems : 1];
  __shared__ uint32_t s_icnt[2];  // item count of step parity p; the other one is reset
  __shared__ uint32_t s_wsum[kPersistBlock / 32];
  if (threadIdx.x == 0) s_icnt[0] = s_icnt[1] = 0;
  if (a.seg_smem) {
    const uint4* src = reinterpret_cast<const uint4*>(a.segs);
    uint4* dst = reinterpret_cast<uint4*>(g_dyn);
    for (uint32_t j = threadIdx.x; j < a.n_segs * (uint32_t)(sizeof(SegDev) / 16); j += kPersistBlock)
      dst[j] = src[j];
    const uint2* ss = reinterpret_cast<const uint2*>(a.srcs);
    uint2* sd = reinterpret_cast<uint2*>(g_dyn + seg_table_bytes(a.n_segs));
    for (uint32_t j = threadIdx.x; j < a.n_srcs * (uint32_t)(sizeof(SrcDev) / 8); j += kPersistBlock)
      sd[j] = ss[j];
  }
  __syncthreads();
  Ctl* ctl = a.ctl;
  StepIdx ix = step_of(a);
  const unsigned long long t0 = ix.t;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t gw = (blockIdx.x * kPersistBlock + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * kPersistBlock) >> 5;
  // One-barrier form: update words are dealt warp-major over the blocks
  // (slot = warp x blocks + block), so consecutive words -- a stimulated input
  // segment, say -- spread over all blocks; each row of nw words is still
  // swept together.
  const uint32_t uw = ONE ? (threadIdx.x >> 5) * gridDim.x + blockIdx.x : gw;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  unsigned long long target = 0;
  uint32_t walked = 0;
  for (uint32_t s = 0; s < n_steps; ++s) {
    ix.t = t0 + s;
    ix.rel = s;
    // Item counter of step t + 1: its last user was the update of step t - 1
    // (kept zero in ONE launches too, for launches of the other form).
    if (leader) __stcg(&ctl->active_count[(ix.t + 1) & 1], 0u);
    // Without dense pulls and plasticity no one reads the history during the
    // launch: it writes the rows of its last hist_rows steps, for the other
    // kernels and the host, and clears their summary rows and the next one's.
    const bool all_rows = LANE != 2;
    ix.keep = all_rows || s + a.hist_rows >= n_steps;
    if (all_rows || s + 1u + a.hist_rows >= n_steps)
      clear_next_summary(a, ix, blockIdx.x * kPersistBlock + threadIdx.x, gridDim.x * kPersistBlock);
    const BlockItems bi{s_items, &s_icnt[s & 1u]};
    if (a.n_plast)
      walked += a.seg_smem ? update_words<true, true, BF16, ONE>(a, uw, nw, ix, bi)
                           : update_words<true, false, BF16, ONE>(a, uw, nw, ix, bi);
    else if (LANE == 2)
      walked += a.seg_smem ? update_pairs<true, BF16>(a, uw, nw, ix, bi)
                           : update_pairs<false, BF16>(a, uw, nw, ix, bi);
    else
      walked += a.seg_smem ? update_words<false, true, BF16, ONE>(a, uw, nw, ix, bi)
                           : update_words<false, false, BF16, ONE>(a, uw, nw, ix, bi);
    // Plastic values of step t before its dense deliveries: with rules that
    // read only earlier steps' spikes, in the update phase itself.
    if (a.n_plast && a.stdp_early) stdp_warp<BF16, true, true>(a, gw, nw, ix);
    if (ONE) {
      __syncthreads();
      const uint32_t n_items = min(s_icnt[s & 1u], kGenItems);
      // The other parity's count was last read before the previous barrier.
      if (threadIdx.x == 0) s_icnt[(s & 1u) ^ 1u] = 0;
      for (uint32_t u = threadIdx.x >> 5; u < n_items; u += kPersistBlock / 32)
        walked += push_item<BF16>(a, s_items[u], ix.slot);
      if (!grid_barrier(a, target)) return;
      ix_advance(a, ix);
      continue;
    }
    if (!grid_barrier(a, target)) return;
    if (a.raster_cap && leader) a.raster_off[s + 1] = __ldcg(&ctl->raster_count);
    if (a.n_plast && !a.stdp_early) {
      stdp_warp<BF16, true, false>(a, gw, nw, ix);
      if (!grid_barrier(a, target)) return;
    }
    const uint32_t* sum = nullptr;
    if (a.n_pull_units && a.pull_sum) {
      stage_summary(a, ix, s_sum, threadIdx.x, kPersistBlock);
      __syncthreads();
      sum = s_sum;
    }
    walked += deliver_warp<BF16, true>(a, gw, nw, ix, sum);
    if (!grid_barrier(a, target)) return;
    ix_advance(a, ix);
  }
  if (ONE && a.raster_cap && blockIdx.x == 0) raster_offsets_from_counts(a, n_steps, s_wsum);
  if (lane == 0 && walked) atomicAdd(&ctl->delivered, (unsigned long long)walked);
  if (leader) {
    ctl->step = t0 + n_steps;
    ctl->ring_slot = ix.slot;
    ctl->hist_row = ix.hrow;
    ctl->t_rel = n_steps;
  }
}

// Resident form for networks with at most one 32-cell word per warp: each warp
// keeps its cells' state, source masks, out-degrees and push-row bounds in
// registers for the whole chunk and writes the state back at the end, so a
// step's critical path is the ring read, the cell update and the deliveries.
template <bool BF16>
__global__ void __launch_bounds__(kPersistBlock, 1) k_persistent_resident(StepArgs a,
                                                                          uint32_t n_steps) {
  // Dynamic shared memory as in the general kernel: segment descriptors and
  // sources (when a.seg_smem), then the staged spike summary.
  uint32_t* s_sum = reinterpret_cast<uint32_t*>(g_dyn + (a.seg_smem ? seg_smem_bytes_dev(a) : 0));
  if (a.seg_smem) {
    const uint4* src = reinterpret_cast<const uint4*>(a.segs);
    uint4* dst = reinterpret_cast<uint4*>(g_dyn);
    for (uint32_t j = threadIdx.x; j < a.n_segs * (uint32_t)(sizeof(SegDev) / 16); j += kPersistBlock)
      dst[j] = src[j];
    const uint2* ss = reinterpret_cast<const uint2*>(a.srcs);
    uint2* sd = reinterpret_cast<uint2*>(g_dyn + seg_table_bytes(a.n_segs));
    for (uint32_t j = threadIdx.x; j < a.n_srcs * (uint32_t)(sizeof(SrcDev) / 8); j += kPersistBlock)
      sd[j] = ss[j];
    __syncthreads();
  }
  const SegDev* segs = a.seg_smem ? reinterpret_cast<const SegDev*>(g_dyn) : a.segs;
  Ctl* ctl = a.ctl;
  StepIdx ix = step_of(a);
  const unsigned long long t0 = ix.t;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t gw = (blockIdx.x * kPersistBlock + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * kPersistBlock) >> 5;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  // Words are dealt round-robin over the blocks (word slot = warp x blocks +
  // block), so every SM holds about the same number of cells and spikes.
  const uint32_t ws = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  const bool has = ws < a.n_upd_words;
  uint32_t w = 0, seg = 0, i = 0, local = 0, mask = 0, r0 = 0, r1 = 0, od = 0;
  bool valid = false, lif = false;
  float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
  if (has) {
    w = __ldg(a.upd_words + ws);
    seg = __ldg(a.seg_of_word + w);
    i = (w << 5) + lane;
    const SegDev& sd = a.segs[seg];
    local = i - sd.base;
    valid = local < sd.count;
    lif = sd.kind == kSegLif;
    if (valid) {
      if (lif) st = state_in(a.su[i], a.sg[i], sd.Vr); else mask = __ldg(a.src_mask + i);
      od = __ldg(a.outdeg + i);
      if (a.any_push) {
        r0 = __ldg(a.push_row + i);
        r1 = __ldg(a.push_row + i + 1);
      }
    }
  }
  unsigned long long target = 0;
  uint32_t walked = 0;
  for (uint32_t s = 0; s < n_steps; ++s) {
    ix.t = t0 + s;
    ix.rel = s;
    if (leader) __stcg(&ctl->active_count[(ix.t + 1) & 1], 0u);
    clear_next_summary(a, ix, blockIdx.x * kPersistBlock + threadIdx.x, gridDim.x * kPersistBlock);
    if (has) {
      const bool fired = cell_fire(a, segs[seg], i, local, valid, st, mask, ix);
      if (a.recent && valid)
        a.recent[(ix.t & 1ull) * a.n_pad + i] =
            (__ldcg(a.recent + ((ix.t + 1ull) & 1ull) * a.n_pad + i) << 1) | (fired ? 1ull : 0ull);
      publish_word(a, w, seg, i, fired, r0, r1, od, ix);
    }
    // Plastic values of step t before its dense deliveries: with rules that
    // read only earlier steps' spikes, in the update phase itself, on the
    // warps without a word (word slots past the last word) when there are
    // some, so that updates and plasticity run side by side.
    if (a.n_plast && a.stdp_early) {
      const uint32_t n_idle = nw > a.n_upd_words ? nw - a.n_upd_words : 0u;
      if (n_idle == 0u)
        stdp_warp<BF16, true, true>(a, gw, nw, ix);
      else if (!has)
        stdp_warp<BF16, true, true>(a, ws - a.n_upd_words, n_idle, ix);
    }
    if (!grid_barrier(a, target)) break;
    if (a.raster_cap && leader) a.raster_off[s + 1] = __ldcg(&ctl->raster_count);
    if (a.n_plast && !a.stdp_early) {
      stdp_warp<BF16, true, false>(a, gw, nw, ix);
      if (!grid_barrier(a, target)) break;
    }
    const uint32_t* sum = nullptr;
    if (a.n_pull_units && a.pull_sum) {
      stage_summary(a, ix, s_sum, threadIdx.x, kPersistBlock);
      __syncthreads();
      sum = s_sum;
    }
    walked += deliver_warp<BF16, true>(a, gw, nw, ix, sum);
    if (!grid_barrier(a, target)) break;
    ix_advance(a, ix);
  }
  if (valid && lif) state_out(a, i, st);
  if (__ldcg(&ctl->error) & kErrBarrierTimeout) return;
  if (lane == 0 && walked) atomicAdd(&ctl->delivered, (unsigned long long)walked);
  if (leader) {
    ctl->step = t0 + n_steps;
    ctl->ring_slot = ix.slot;
    ctl->hist_row = ix.hrow;
    ctl->t_rel = n_steps;
  }
}

// Resident form with dense pulls, one substep a step: one grid barrier a step.
// The reference tests a spike on the potential before the step's integration,
// so the spikes of step t + 1 are known when step t's update ends.  Iteration t
// publishes them (as the fused kernel's late-push timelines do) and, in the
// same phase, pulls into slot t + 1 from the spikes of steps <= t, which the
// previous barrier completed: nothing in an iteration waits for another
// block's work of the same iteration.
//   The pull reads no table from global memory: a block keeps the entries of
// its units (unit u belongs to block u mod blocks) in shared memory for the
// whole launch, as many as fit, beside the D history rows a pull reads; an
// iteration loads only the row of step t (n_words words) and tests every entry
// on its own bit, so only deliveries leave the SM: their weight and one
// reduction.  The rows also free the writers of row t + 1 from readers of
// row t + 1 - H.
//   A unit's entries come sorted by spike bit (k_pull_sort), each with its place
// in the unit.  32 consecutive ones cover a few words, so a lane settles a
// group of 32 with one look at the rows' summary bits, and only the groups
// that pass (one in five to ten) are tested entry by entry: 70 warp
// instructions per 128 entries without this made the test, at five warps per
// scheduler, the longest part of the step.  Sorted, the delay-1 entries are a
// prefix of the unit.  Only
// those wait for the spikes of step t; the others' deliveries into slot t + 2
// come from spikes of steps <= t as well, so they are made behind iteration t's
// barrier arrival, in the time the barrier takes (the launch's first step
// finds those into its slot made by the prologue, the last one makes none, so
// a launch ends as with the other kernels).
//   Plastic projections: the block that pulls a unit also updates its weights,
// so a block barrier orders the two.  Rules that read only earlier steps'
// spikes (stdp_early) make the update of step t + 1 behind iteration t's
// barrier arrival, the others that of step t before its pulls (and all of
// them then).  The spike registers stay in their owners' registers and are
// published in three buffers (step mod 3): behind the arrival, faster blocks
// already write those of step t + 2 while step t's are read.
//   What bounds it is latency: history row and ring slot (one L2 round trip),
// the test of the delay-1 entries, weight, reduction, barrier.  92,550 cells:
// every projection dense, 16-bit weights, 9.0 us per step with two barriers
// and the entries read from L2 -> 4.1 us; Teacher rule on 1.75M synapses
// 10.2 -> 5.1 us (one barrier alone, every entry tested: 4.5 and 6.0 us).
struct HistRows {     // rows of the last steps, newest at word `base`, in decreasing step order
  const uint32_t* s;
  uint32_t base, total;  // total: words of all rows (the rows are a ring)
  __device__ __forceinline__ uint32_t word(uint32_t w) const {
    const uint32_t x = base + w;
    return s[min(x, x - total)];
  }
  __device__ __forceinline__ uint32_t bit(uint32_t off) const {
    return (word(off >> 5) >> (off & 31u)) & 1u;
  }
};

// A unit's entries in k_persistent_pull's form: the spike bit's word above the
// step's row << 15 | place in the unit << 5 | bit in the word, ascending;
// padding (word pull_rows * n_words, which the ring of rows maps to row 0)
// last.  A group is 32 consecutive ones, one per lane.
constexpr uint32_t kWordShift = 15;
static_assert(kPullUnit == 1u << (kWordShift - 5), "place of an entry in its unit");
constexpr uint32_t kGroup = 32, kGroups = kPullUnit / kGroup;

// Units of a block and what each needs besides its entries.
struct PullInfo {
  uint32_t proj, o0;
  uint32_t n1, n;  // delay-1 entries, entries (without padding)
};
static_assert(sizeof(PullInfo) == 16, "PullInfo copied as uint4");

// Sorts the entries of unit blockIdx.x (bitonic, two entries per thread).
__global__ void __launch_bounds__(kPullUnit / 2) k_pull_sort(StepArgs a, uint32_t* out, uint4* info) {
  __shared__ uint32_t s[kPullUnit];
  const PullUnit un = a.pull_units[blockIdx.x];
  const uint32_t* src = a.projs[un.proj].ell_syn + un.o0;
  const uint32_t pad = pull_rows(a) * a.n_pad;
  uint32_t n1 = 0, n = 0;
  for (uint32_t p = threadIdx.x; p < kPullUnit; p += kPullUnit / 2) {
    const uint32_t e = min(src[p], pad);
    s[p] = ((e >> 5) << kWordShift) | (p << 5) | (e & 31u);
    n1 += (uint32_t)__syncthreads_count(e < a.n_pad);
    n += (uint32_t)__syncthreads_count(e < pad);
  }
  for (uint32_t k = 2; k <= kPullUnit; k <<= 1)
    for (uint32_t d = k >> 1; d; d >>= 1) {
      __syncthreads();
      const uint32_t x = ((threadIdx.x & ~(d - 1u)) << 1) | (threadIdx.x & (d - 1u)), y = x | d;
      const uint32_t u = s[x], v = s[y];
      if ((u > v) == ((x & k) == 0u)) {
        s[x] = v;
        s[y] = u;
      }
    }
  __syncthreads();
  for (uint32_t p = threadIdx.x; p < kPullUnit; p += kPullUnit / 2)
    out[blockIdx.x * kPullUnit + p] = s[p];
  if (threadIdx.x == 0) info[blockIdx.x] = make_uint4(un.proj, un.o0, n1, n);
}

// Units of the calling block, and the dynamic shared memory of k_persistent_pull:
// segment descriptors and sources, projections, the history rows and a summary
// bit per word of them, then per held unit its entries, its PullInfo, with
// plastic projections where each sub-unit's post / teacher spikes are, its
// groups' words and its groups in the two work lists.
__host__ __device__ __forceinline__ size_t pull_proj_bytes(const StepArgs& a) {
  return ((size_t)a.n_projs * sizeof(ProjDev) + 15) & ~(size_t)15;
}
__host__ __device__ __forceinline__ uint32_t pull_sum_words(const StepArgs& a) {
  return (pull_rows(a) * a.n_swords + 1u + 3u) & ~3u;  // and one that a group's look may run into
}
__host__ __device__ __forceinline__ size_t pull_fixed_bytes(const StepArgs& a) {
  return seg_smem_bytes_dev(a) + pull_proj_bytes(a) + (size_t)pull_rows(a) * a.n_words * 4 +
         (size_t)pull_sum_words(a) * 4;
}
constexpr uint32_t kSub = kPullUnit / kStdpUnit;  // plasticity sub-units per pull unit
__host__ __device__ __forceinline__ size_t pull_unit_bytes(const StepArgs& a) {
  return kPullUnit * 4 + sizeof(PullInfo) + kGroups * (4 + 2 * 2) + (a.n_plast ? kSub * sizeof(uint2) : 0);
}

// Sub-unit x of the block (kStdpUnit ELL cells from *o0 of plastic projection
// *k): where the spikes of its one or two posts (or their teachers) are above
// the step's history row (.y kNever: one post), or kAlways in .y when every
// cell may change or it covers more posts; kNever in .x: no spike, or not
// plastic.
constexpr uint32_t kAlways = 0xFFFFFFFEu, kNever = 0xFFFFFFFFu;
__device__ __forceinline__ uint2 stdp_sub(const StepArgs& a, uint32_t x, uint32_t* k, uint32_t* o0) {
  const PullUnit pu = a.pull_units[blockIdx.x + (x / kSub) * gridDim.x];
  *o0 = pu.o0 + (x % kSub) * kStdpUnit;
  for (*k = 0; *k < a.n_plast; ++*k) {
    const PlastDev& L = a.plast[*k];
    const ProjDev& P = a.projs[L.proj];
    if (L.proj != pu.proj || *o0 >= P.ell_n) continue;
    if (L.a0 != 0.f || L.a1_j != 0.f || !P.ell_rowmajor) return make_uint2(kAlways, kAlways);
    const uint32_t p0 = *o0 / P.ell_K, p1 = (min(*o0 + kStdpUnit, P.ell_n) - 1u) / P.ell_K;
    if (p1 > p0 + 1u) return make_uint2(kAlways, kAlways);
    const bool te = L.rule == SGB_STDP_TEACHER;
    const uint32_t s0 = te ? __ldg(L.teacher + p0) : P.post_base + p0;
    if (p1 == p0) return make_uint2(s0, kNever);
    const uint32_t s1 = te ? __ldg(L.teacher + p1) : P.post_base + p1;
    return make_uint2(s0, s1 == kNever ? s0 : s1);  // a post without a teacher never changes
  }
  return make_uint2(kNever, kNever);
}

// The plasticity of a step on the block's own units (h and recent as the step
// sees them): threads screen sub-units, then warps update those that can
// change.  s_sub: the held sub-units' stdp_sub, or NULL.  Run by the block's
// first n_thr threads, which meet on block barrier 1 (0 when all run it);
// every round but a last one without updates ends with that barrier.  s_n[2]
// counts the active sub-units of alternate rounds, par the next round's.
template <bool BF16, bool EARLY>
__device__ __forceinline__ void stdp_own(const StepArgs& a, const HistRows& h,
                                         const unsigned long long* recent, const uint2* s_sub,
                                         uint32_t* s_list, uint32_t* s_n, uint32_t& par, uint32_t n_thr) {
  auto sync = [n_thr] {
    if (n_thr == blockDim.x) __syncthreads(); else bar_sync_first(n_thr);
  };
  const uint32_t pad = a.hist_rows * a.n_pad;
  const uint32_t n_sub = (a.n_pull_units + gridDim.x - 1u - blockIdx.x) / gridDim.x * kSub;
  for (uint32_t b = 0; b < n_sub; b += n_thr, par ^= 1u) {
    const uint32_t x = b + threadIdx.x;
    if (x < n_sub) {
      uint32_t k, o0;
      const uint2 so = s_sub ? s_sub[x] : stdp_sub(a, x, &k, &o0);
      bool active = so.y == kAlways;
      if (!active) active = (so.x != kNever && h.bit(so.x)) || (so.y != kNever && h.bit(so.y));
      if (active) s_list[atomicAdd(&s_n[par], 1u)] = threadIdx.x | (so.y == kNever ? 1u << 31 : 0u);
    }
    sync();
    const uint32_t n = s_n[par];
    // The next round's count.  Its readers were before this barrier; its next
    // writers come after the one that ends the round.
    if (threadIdx.x == 0) s_n[par ^ 1u] = 0;
    for (uint32_t j = threadIdx.x >> 5; j < n; j += n_thr >> 5) {
      const uint32_t v = s_list[j];
      uint32_t k, o0;
      stdp_sub(a, b + (v & 0xFFFFu), &k, &o0);
      stdp_unit<BF16, true, EARLY>(a, PullUnit{k, o0}, h, pad, recent, v >> 31);
    }
    if (n || b + n_thr < n_sub) sync();
  }
}

template <bool BF16, uint32_t MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_persistent_pull(StepArgs a, uint32_t n_steps) {
  const uint32_t n_thr = blockDim.x, n_wrp = n_thr >> 5;  // pull_threads
  __shared__ uint2 s_items[kGenItems];
  __shared__ uint32_t s_icnt[2];
  __shared__ uint32_t s_wsum[kPersistBlock / 32];
  __shared__ uint32_t s_act[kPersistBlock];  // active plastic sub-units
  __shared__ uint32_t s_nact[2], s_n1, s_n2;
  __shared__ uint32_t s_od[kPersistBlock];  // out-degree of each thread's cell
  __shared__ int s_ok;
  const uint32_t n_rows = pull_rows(a), row_words = n_rows * a.n_words;
  const uint32_t mine = (a.n_pull_units + gridDim.x - 1u - blockIdx.x) / gridDim.x;
  const uint32_t held = min(mine, a.pull_held);
  ProjDev* s_proj = reinterpret_cast<ProjDev*>(g_dyn + seg_smem_bytes_dev(a));
  uint32_t* s_hist = reinterpret_cast<uint32_t*>(g_dyn + seg_smem_bytes_dev(a) + pull_proj_bytes(a));
  uint32_t* s_sum = s_hist + row_words;  // bit w: word w of the rows is not 0
  uint32_t* s_ent = s_sum + pull_sum_words(a);
  PullInfo* s_info = reinterpret_cast<PullInfo*>(s_ent + (size_t)held * kPullUnit);
  uint2* s_sub = reinterpret_cast<uint2*>(s_info + held);
  uint32_t* s_rng = reinterpret_cast<uint32_t*>(s_sub + (a.n_plast ? held * kSub : 0u));
  uint16_t* s_g1 = reinterpret_cast<uint16_t*>(s_rng + held * kGroups);
  uint16_t* s_g2 = s_g1 + held * kGroups;  // groups with delay-1 entries; with later ones
  {
    const uint4* src = reinterpret_cast<const uint4*>(a.segs);
    uint4* dst = reinterpret_cast<uint4*>(g_dyn);
    for (uint32_t j = threadIdx.x; j < a.n_segs * (uint32_t)(sizeof(SegDev) / 16); j += n_thr)
      dst[j] = src[j];
    const uint2* ss = reinterpret_cast<const uint2*>(a.srcs);
    uint2* sd = reinterpret_cast<uint2*>(g_dyn + seg_table_bytes(a.n_segs));
    for (uint32_t j = threadIdx.x; j < a.n_srcs * (uint32_t)(sizeof(SrcDev) / 8); j += n_thr)
      sd[j] = ss[j];
    const uint2* ps = reinterpret_cast<const uint2*>(a.projs);
    for (uint32_t j = threadIdx.x; j < a.n_projs * (uint32_t)(sizeof(ProjDev) / 8); j += n_thr)
      reinterpret_cast<uint2*>(s_proj)[j] = ps[j];
  }
  const SegDev* segs = reinterpret_cast<const SegDev*>(g_dyn);
  const SrcDev* srcs = reinterpret_cast<const SrcDev*>(g_dyn + seg_table_bytes(a.n_segs));
  Ctl* ctl = a.ctl;
  StepIdx ix = step_of(a);
  const unsigned long long t0 = ix.t;
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  // A rule that reads the step's own spikes changes weights between a step's
  // publication and its pulls, so then no pull goes ahead.
  const bool ahead = a.n_plast == 0u || a.stdp_early != 0u;
  if (threadIdx.x == 0) s_icnt[0] = s_icnt[1] = s_nact[0] = s_nact[1] = s_n1 = s_n2 = 0;
  // The rows of steps t0 - 1, t0 - 2, ...; row 0 (step t0) follows in the loop.
  for (uint32_t j = a.n_words / 4u + threadIdx.x; j < row_words / 4u; j += n_thr)
    reinterpret_cast<uint4*>(s_hist)[j] = __ldcg(reinterpret_cast<const uint4*>(hist_base(a, ix.hrow)) + j);
  for (uint32_t j = threadIdx.x; j < pull_sum_words(a); j += n_thr) s_sum[j] = 0u;
  constexpr uint32_t kQ = kPullUnit / 4;  // 16-byte loads per unit
  const uint4* ents = reinterpret_cast<const uint4*>(a.pull_sorted);
  const uint32_t n_held = held * kGroups, n_mine = mine * kGroups;  // groups
  for (uint32_t q = threadIdx.x; q < held * kQ; q += n_thr)
    reinterpret_cast<uint4*>(s_ent)[q] = __ldg(ents + (size_t)(blockIdx.x + (q / kQ) * gridDim.x) * kQ + q % kQ);
  for (uint32_t k = threadIdx.x; k < held; k += n_thr)
    reinterpret_cast<uint4*>(s_info)[k] = __ldg(a.pull_info + blockIdx.x + k * gridDim.x);
  if (a.n_plast)
    for (uint32_t x = threadIdx.x; x < held * kSub; x += n_thr) {
      uint32_t k, o0;
      s_sub[x] = stdp_sub(a, x, &k, &o0);
    }
  const uint2* subs = a.n_plast && held == mine ? s_sub : nullptr;
  __syncthreads();
  for (uint32_t j = a.n_words + threadIdx.x; j < row_words; j += n_thr)
    if (s_hist[j]) atomicOr(s_sum + (j >> 5), 1u << (j & 31u));
  // A group's words: first << 6 | span, span 0 for more than 32 words or
  // several rows, where every lane looks its own word up.
  for (uint32_t x = threadIdx.x; x < n_held; x += n_thr) {
    const PullInfo& f = s_info[x / kGroups];
    const uint32_t g = x % kGroups * kGroup, n1 = ahead ? f.n1 : f.n;
    const uint32_t w0 = s_ent[x * kGroup] >> kWordShift, w1 = s_ent[x * kGroup + kGroup - 1u] >> kWordShift;
    s_rng[x] = (w0 << 6) | (w0 / a.n_words == w1 / a.n_words && w1 - w0 < 32u ? w1 - w0 + 1u : 0u);
    if (g < n1) s_g1[atomicAdd(&s_n1, 1u)] = (uint16_t)x;
    if (g + kGroup > n1 && g < f.n) s_g2[atomicAdd(&s_n2, 1u)] = (uint16_t)x;
  }
  // Words are dealt round-robin over the blocks (word slot = warp x blocks + block).
  const uint32_t ws = wib * gridDim.x + blockIdx.x;
  const bool has = ws < a.n_upd_words;
  uint32_t w = 0, seg = 0, i = 0;
  bool valid = false, lif = false, stim = false;
  s_od[threadIdx.x] = 0;
  float4 st = make_float4(0.f, 0.f, 0.f, 0.f);
  unsigned long long reg = 0;  // the cell's spike register, bit j = step t - j
  if (has) {
    w = __ldg(a.upd_words + ws);
    seg = __ldg(a.seg_of_word + w);
    i = (w << 5) + lane;
    const SegDev& sd = a.segs[seg];
    valid = i - sd.base < sd.count;
    lif = sd.kind == kSegLif;
    if (valid) {
      if (lif) st = state_in(a.su[i], a.sg[i], sd.Vr); else stim = __ldg(a.src_mask + i) != 0u;
      s_od[threadIdx.x] = __ldg(a.outdeg + i);
      if (a.recent) reg = a.recent[((t0 + 1ull) & 1ull) * a.n_pad + i];
    }
  }
  __syncthreads();
  const bool rd = lif && valid;
  unsigned long long target = 0;
  uint32_t walked = 0, hits = 0;
  int2* ring2 = reinterpret_cast<int2*>(a.ring);
  uint32_t tri = (uint32_t)(t0 % 3ull);  // buffer of the last published step
  // Publishes the spikes of step px.t (chunk row px.rel): bitmap, counts,
  // spike register, and push items of parity par.
  auto publish = [&](bool fired, const StepIdx& px, uint32_t par) {
    if (!has) return;
    if (a.recent && valid) {
      reg = (reg << 1) | (fired ? 1ull : 0ull);
      a.recent3[(size_t)tri * a.n_pad + i] = reg;
    }
    uint32_t r0 = 0, r1 = 0;
    if (fired && a.any_push) {
      r0 = __ldg(a.push_row + i);
      r1 = __ldg(a.push_row + i + 1);
    }
    walked += publish_word<BF16, true>(a, w, seg, i, fired, r0, r1, s_od[threadIdx.x], px,
                                       BlockItems{s_items, &s_icnt[par]});
  };
  auto push = [&](const StepIdx& px, uint32_t par) {  // after a block barrier
    const uint32_t n_items = min(s_icnt[par], kGenItems);
    if (threadIdx.x == 0) s_icnt[par ^ 1u] = 0;
    for (uint32_t u = wib; u < n_items; u += n_wrp) walked += push_item<BF16>(a, s_items[u], px.slot);
  };
  const uint32_t split = ahead ? a.n_words : row_words;
  // Whether one of the group's words is set (one group per lane).
  auto may_hit = [&](const HistRows& h, uint32_t rng) -> bool {
    const uint32_t span = rng & 63u;
    uint32_t x = h.base + (rng >> 6);
    x = min(x, x - h.total);
    const uint32_t* p = s_sum + (x >> 5);
    return span == 0u || (__funnelshift_r(p[0], p[1], x) & (0xFFFFFFFFu >> (32u - span))) != 0u;
  };
  // Delivery of the lane's entry e of a unit, if its bit is set and its word is
  // in [lo, hi) (padding lies beyond).  The first one waits in (pend_a,
  // pend_w) with its weight's load in flight until flush().
  uint32_t pend_a = kNever;
  float pend_w = 0.f;
  auto test = [&](const HistRows& h, uint32_t e, uint32_t lo, uint32_t hi) -> bool {
    const uint32_t w = e >> kWordShift;
    return ((h.word(w) >> (e & 31u)) & 1u) != 0u && w - lo < hi - lo;
  };
  auto hit = [&](const PullInfo& f, uint32_t e, uint32_t slot) {
    ++hits;
    const uint32_t o = f.o0 + ((e >> 5) & (kPullUnit - 1u));
    const ProjDev& P = s_proj[f.proj];
    if (pend_a == kNever) {
      pend_w = pull_weight<BF16>(P, o);
      pend_a = (uint32_t)pull_target(a, P, o, slot);
    } else {
      pull_hit<BF16>(a, P, o, slot);
    }
  };
  // A warp's share (of n_w warps) of a work list: a group per lane against the
  // summaries, then the few that pass, an entry per lane.
  auto pull = [&](const HistRows& h, const uint16_t* list, uint32_t n, uint32_t lo, uint32_t hi,
                  uint32_t slot, uint32_t n_w) {
    for (uint32_t c0 = wib; c0 < n; c0 += 32u * n_w) {
      const uint32_t c = c0 + lane * n_w;
      const uint32_t x = c < n ? list[c] : 0u;
      uint32_t todo = __ballot_sync(kFull, c < n && may_hit(h, s_rng[x]));
      while (todo) {
        const uint32_t g = __shfl_sync(kFull, x, __ffs(todo) - 1);
        todo &= todo - 1u;
        const uint32_t e = s_ent[g * kGroup + lane];
        if (test(h, e, lo, hi)) hit(s_info[g / kGroups], e, slot);
      }
    }
  };
  auto flush = [&]() {
    if (pend_a != kNever) atomicAdd(a.ring + pend_a, __float2int_rn(pend_w));
    pend_a = kNever;
  };
  const auto draw = [&](unsigned long long t) {
    return stim && input_fire(a, srcs, segs[seg], i - segs[seg].base, __ldg(a.src_mask + i), t);
  };
  HistRows rows{s_hist, 0u, row_words};  // newest row: step t
  uint32_t act_par = 0;
  bool in_next = false, aborted = false;
  if (n_steps) {
    if (a.n_plast && a.stdp_early)
      stdp_own<BF16, true>(a, rows, a.recent + ((t0 + 1ull) & 1ull) * a.n_pad, subs, s_act, s_nact,
                           act_par, n_thr);
    ix.rel = 0;
    clear_next_summary(a, ix, blockIdx.x * n_thr + threadIdx.x, gridDim.x * n_thr);
    publish(valid && (lif ? st.x > segs[seg].Vth : draw(t0)), ix, 0u);
    __syncthreads();
    if (ahead) {
      // The later delays' deliveries into slot t0 + 1, from steps before t0.
      const uint32_t slot1 = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
      pull(rows, s_g2, s_n2, split, row_words, slot1, n_wrp);
      flush();
    }
    push(ix, 0u);
    grid_arrive(a, target);
    if (n_steps > 1) in_next = draw(t0 + 1ull);
    aborted = !grid_wait(a, target);
  }
  for (uint32_t s = 0; s < n_steps && !aborted; ++s) {
    const bool more = s + 1u < n_steps;
    // Row of step t and ring slot t: one round trip for both.
    const uint4* src = reinterpret_cast<const uint4*>(hist_base(a, ix.hrow));
    uint4* dst = reinterpret_cast<uint4*>(s_hist + rows.base);
    const uint32_t n4 = a.n_words / 4u;
    uint4 hv = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < n4) hv = __ldcg(src + threadIdx.x);
    int2 acc = make_int2(0, 0);
    if (rd) acc = __ldcg(ring2 + (ix.roff + i));
    flush();  // delivered behind the last arrival, read from step t + 1 on
    const uint32_t consumed = ix.roff;
    auto store = [&](uint32_t j, uint4 v) {  // four words of the row and their summary bits
      dst[j] = v;
      const uint32_t b = (v.x ? 1u : 0u) | (v.y ? 2u : 0u) | (v.z ? 4u : 0u) | (v.w ? 8u : 0u);
      if (b) atomicOr(s_sum + (rows.base >> 5) + (j >> 3), b << ((4u * j) & 31u));
    };
    for (uint32_t j = n_thr + threadIdx.x; j < n4; j += n_thr) store(j, __ldcg(src + j));
    if (threadIdx.x < n4) store(threadIdx.x, hv);
    // From here on ix is step t + 1, whose spikes this step publishes.
    ix.t += 1ull;
    ix.rel = s + 1u;
    ix_advance(a, ix);
    const unsigned long long* rec_t = a.recent3 + (size_t)tri * a.n_pad;  // registers of step t
    if (more) tri = tri == 2u ? 0u : tri + 1u;
    clear_next_summary(a, ix, blockIdx.x * n_thr + threadIdx.x, gridDim.x * n_thr);
    bool fired = in_next;
    if (has && lif) {
      const LifK k = lif_k(segs[seg]);
      if (rd) lif_update<1>(k, 1, st, acc);
      fired = valid && st.x > k.Vth;
      if (acc.x | acc.y) __stcg(ring2 + (consumed + i), make_int2(0, 0));
    }
    const uint32_t par = (s + 1u) & 1u;
    if (more) publish(fired, ix, par);
    __syncthreads();
    if (a.n_plast && !a.stdp_early)
      stdp_own<BF16, false>(a, rows, rec_t, subs, s_act, s_nact, act_par, n_thr);
    // Deliveries into slot t + 1: the delay-1 entries (every entry, when none
    // goes ahead, and of the units that are not held).
    pull(rows, s_g1, s_n1, 0u, split, ix.slot, n_wrp);
    for (uint32_t c = n_held + wib; c < n_mine; c += n_wrp) {
      const uint32_t u = blockIdx.x + (c / kGroups) * gridDim.x;
      const uint32_t e = __ldg(a.pull_sorted + (size_t)u * kPullUnit + (c % kGroups) * kGroup + lane);
      if (test(rows, e, 0u, row_words)) {
        const uint4 f = __ldg(a.pull_info + u);
        hit(PullInfo{f.x, f.y, f.z, f.w}, e, ix.slot);
      }
    }
    flush();
    if (a.any_push) {
      __syncthreads();
      push(ix, par);
    }
    // The last warp arrives, its release waiting for the block's writes, and
    // polls; the others go on.
    __syncthreads();
    target += gridDim.x;
    if (threadIdx.x == n_thr - 32u)
      asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(a.bar) : "memory");
    if (s + 2u < n_steps) in_next = draw(ix.t + 1ull);
    if (wib == n_wrp - 1u) {
      if (lane == 0) s_ok = poll_arrivals(a, target);
      __syncwarp();
    } else if (more && ahead) {
      // As step t + 1 sees the rows: its offsets of a delay of 1 fall on the row
      // that it is going to load (a group's test reads it, and drops the result).
      const HistRows next{s_hist, rows.base == 0u ? row_words - a.n_words : rows.base - a.n_words,
                          row_words};
      if (a.n_plast)
        stdp_own<BF16, true>(a, next, rec_t, subs, s_act, s_nact, act_par, n_thr - 32u);
      const uint32_t slot2 = ix.slot + 1u == a.ring_slots ? 0u : ix.slot + 1u;
      pull(next, s_g2, s_n2, split, row_words, slot2, n_wrp - 1u);
    }
    rows.base = rows.base == 0u ? row_words - a.n_words : rows.base - a.n_words;
    // The summary of the row that the next step replaces; the pulls made just
    // above may still test it for groups that also hold later rows' entries, and
    // drop what it says.
    for (uint32_t j = threadIdx.x; j < a.n_swords; j += n_thr) s_sum[(rows.base >> 5) + j] = 0u;
    __syncthreads();
    aborted = !s_ok;
  }
  if (valid && lif) state_out(a, i, st);
  if (a.recent && valid && n_steps) a.recent[((t0 + n_steps + 1ull) & 1ull) * a.n_pad + i] = reg;
  if (a.raster_cap && blockIdx.x == 0) raster_offsets_from_counts(a, n_steps, s_wsum);
  if (__ldcg(&ctl->error) & kErrBarrierTimeout) return;
  hits = __reduce_add_sync(kFull, hits);
  if (lane == 0 && walked) atomicAdd(&ctl->delivered, (unsigned long long)walked);
  if (lane == 0 && hits) atomicAdd(&ctl->pulled, (unsigned long long)hits);
  if (leader) {
    ctl->step = t0 + n_steps;
    ctl->ring_slot = ix.slot;
    ctl->hist_row = ix.hrow;
    ctl->t_rel = n_steps;
  }
}

// Fused form (resident networks whose projections are all event-driven): a
// step's deliveries only target ring slots t+1 .. t+D while its update only
// reads slot t, so update and push of the same step share one phase and a
// step needs one grid barrier.
//   What bounds a step is not its mean work but its slowest block: with every
// row pushed by the block that holds its cell, blocks did 2,900 cycles of work
// a step on average, and the slowest of them 5,600 (a Golgi cell's 1,600
// scattered reductions leave one SM at about three cycles each).  So long rows
// are not pushed by their block:
//   Heavy words (32-cell words of long rows, chosen by the host).  Every block
// keeps the heavy cells' synapses onto its own cells in shared memory (very long
// rows' partly in global memory, FAR), grouped by heavy cell, and an own delay
// line of increments (s_line) for its cells.  A heavy word's spikes of step t go
// onto a board in global memory, one 64-bit word {step tag, spike bits} per heavy
// word; in step t one warp of every block reads the board, adds what its cells
// receive into its line's slots t + d, d >= 1, and the block barrier that ends
// the step hands them to the update of t + 1.  Bits and tag share a word, so the
// board needs no fence and no barrier of its own.  A Golgi spike becomes ten
// additions in each block's shared memory; many spikes at once are dealt over the
// warp's lanes (board_many).  When the stimulus alone keeps that warp too busy, a
// launch goes without heavy words (a.hv_busy).  At the end of a launch the line's
// pending slots are added to the ring, so a launch leaves what the other kernels
// expect.
//   Other rows are pushed by the spiking cell's own warp, from a copy of the
// block's rows in shared memory (row_smem; rows past the capacity stay in
// global memory); only rows over a.direct_row synapses, in a block that has any,
// are cut into items for all of the block's warps, at the price of a block
// barrier a step.
//   A step's stimulus decisions share what does not depend on the cell: which
// sources are on or fire periodically in each substep is worked out once per
// block, by that warp, a lane per source and substep (s_on).
//   Per step, without heavy words and with every row as items -> now: 92,550 cells
// 2.24 -> 1.74 us, with 16-bit weights 2.45 -> 1.75; 9,256 cells 1.71 -> 1.49;
// 152,700 cells (two words a warp) 2.69 -> 2.03; 97,020 cells in steps of ten
// substeps 6.84 -> 4.21.
constexpr uint32_t kBlockItems = 1024;  // push items per block and step (8 KiB)
constexpr uint32_t kSrcCache = 16;      // stimulus sources kept in shared memory
constexpr uint32_t kOnSubsteps = 32;    // substeps whose source states are shared
// Items are ranges of 2^a.item_log2 synapses (64 or 128) of a long row: (first
// synapse, length << 23 | 1 when it is in shared memory).
// States of n_srcs sources in the substeps of step t, by the lanes of one warp.
__device__ __forceinline__ void source_states(const SrcDev* srcs, uint2* on, uint32_t n_srcs,
                                           uint32_t substeps, unsigned long long t) {
  const uint32_t lane = threadIdx.x & 31u;
  if (lane < substeps) on[lane] = make_uint2(0u, 0u);
  __syncwarp();
#pragma unroll 1
  for (uint32_t p = lane; p < n_srcs * substeps; p += 32u) {
    const uint32_t s = p / n_srcs, j = p - s * n_srcs;
    const SrcDev& src = srcs[j];
    const int64_t k = (int64_t)t * substeps + s;
    if (!window_on(src, k)) continue;
    if (src.kind == SGB_INPUT_POISSON)
      atomicOr(&on[s].x, 1u << j);
    else if (periodic_fire(src, k))
      atomicOr(&on[s].y, 1u << j);
  }
  __syncwarp();
}

// Shared memory of the heavy words: the line, where each heavy cell's synapses
// start, and up to hv_held of them.
__host__ __device__ __forceinline__ uint32_t hv_line_slots(const StepArgs& a) { return a.max_delay + 1u; }
__host__ __device__ __forceinline__ size_t hv_bytes(const StepArgs& a, uint32_t blocks) {
  if (!a.hv_words) return 0;
  const size_t cells = ((size_t)a.n_upd_words + blocks - 1u) / blocks * 32u;
  const size_t line = hv_line_slots(a) * cells * sizeof(int2);
  const size_t off = ((size_t)(a.hv_words * 32u + 1u) * sizeof(uint16_t) + 15) & ~(size_t)15;
  return line + off + (size_t)a.hv_held * sizeof(uint2);
}

// Words of a block, at most: one per warp up to kFusedSingle, else two.
constexpr uint32_t kFusedSingle = 22;  // beyond, 24 warps of 80 registers are not enough
__host__ __device__ constexpr uint32_t fused_max_words(uint32_t w) {
  return w == 1u ? kFusedSingle : (uint32_t)kPersistBlock / 32u;
}
__host__ __device__ constexpr uint32_t fused_max_threads(uint32_t w) {
  return 32u * ((fused_max_words(w) + w - 1u) / w + 2u);
}

// The heavy words' spikes of one step, when they are many, into a block's delay
// line (k_persistent_fused), by one warp: listed, then 32 cells at a time, their
// synapses dealt over the lanes, where one cell after another costs about 110
// cycles each.  got: the lane's words, 32 apart.  Returns the synapses added.
// 4,000 heavy cells: at 150 Hz (60 spikes a step) 10.3 -> 2.7 us per step with 128
// synapses each, 8.2 -> 3.8 with 600; at 4 Hz in ten substeps (16 a step) 5.4 ->
// 3.9.  Out of line for one word per warp, where inlined it costs the common step
// 4 % (92,550 cells 1.70 us without it, 1.73 out of line, 1.77 inlined).
constexpr uint32_t kBoardFew = 5;     // lanes with spiking cells, up to which they are few
constexpr uint32_t kBoardList = 256;  // cells listed at a time
template <bool FAR>
__device__ __forceinline__ uint32_t board_many(uint4 gotv, const uint16_t* s_hoff, const uint2* s_hsyn, int2* s_line,
                                               uint16_t* s_list, uint32_t at, uint32_t n_line, uint32_t n_cell,
                                               const uint2* far, uint32_t held) {
  const uint32_t lane = threadIdx.x & 31u;
  static_assert(kHeavyWords == 128, "four words per lane");
  uint32_t got[4] = {gotv.x, gotv.y, gotv.z, gotv.w}, walked = 0;
#pragma unroll 1
  while (true) {
    uint32_t n_sp = 0;
#pragma unroll
    for (uint32_t k = 0; k < kHeavyWords / 32u; ++k) n_sp += __popc(got[k]);
    uint32_t to = n_sp;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(kFull, to, o);
      if (lane >= (uint32_t)o) to += v;
    }
    const uint32_t all = min(__shfl_sync(kFull, to, 31), kBoardList);
    if (!all) return walked;
    to -= n_sp;
#pragma unroll
    for (uint32_t k = 0; k < kHeavyWords / 32u; ++k)
#pragma unroll 1
      while (got[k] && to < kBoardList) {
        s_list[to++] = (uint16_t)((32u * k + lane) * 32u + __ffs(got[k]) - 1u);
        got[k] &= got[k] - 1u;
      }
    __syncwarp();
#pragma unroll 1
    for (uint32_t i0 = 0; i0 < all; i0 += 32u) {
      uint32_t q0 = 0, len = 0;
      if (i0 + lane < all) {
        const uint32_t c = s_list[i0 + lane];
        q0 = s_hoff[c];
        len = s_hoff[c + 1u] - q0;
      }
      uint32_t incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      const uint32_t total = __shfl_sync(kFull, incl, 31);
      const uint32_t base = q0 - (incl - len);  // of the owner's synapses, less its first piece
#pragma unroll 1
      for (uint32_t t0 = 0; t0 < total; t0 += 32u) {
        const uint32_t t = min(t0 + lane, total - 1u);
        uint32_t owner = 0;
#pragma unroll
        for (uint32_t d = 16; d; d >>= 1)
          if (__shfl_sync(kFull, incl, owner + d - 1u) <= t) owner += d;
        const uint32_t q = __shfl_sync(kFull, base, owner) + t;
        if (t0 + lane < total) {
          // {cell | delay << 10 | accumulator << 14, increment}
          const uint2 e = FAR && q >= held ? __ldg(far + q) : s_hsyn[q];
          uint32_t slot = at + ((e.x >> 10) & 15u);
          if (slot >= n_line) slot -= n_line;
          atomicAdd(reinterpret_cast<int*>(s_line + slot * n_cell + (e.x & 1023u)) + (e.x >> 14), (int)e.y);
        }
      }
      walked += total;
    }
    __syncwarp();
  }
}

template <bool FAR>
__device__ __noinline__ uint32_t board_many_call(uint4 gotv, const uint16_t* s_hoff, const uint2* s_hsyn,
                                                 int2* s_line, uint16_t* s_list, uint32_t at, uint32_t n_line,
                                                 uint32_t n_cell, const uint2* far, uint32_t held) {
  return board_many<FAR>(gotv, s_hoff, s_hsyn, s_line, s_list, at, n_line, n_cell, far, held);
}

// TL: the step's timeline -- 0 spikes in their own step; for one-substep steps
// 1 late push, 2 late push with a split grid barrier (see the loops below).
// W: words per warp.  A warp that holds two words shares a step's bookkeeping
// between them and has two independent chains of loads and arithmetic in
// flight, and the smaller block has the registers for it (with the shared
// memory this kernel takes, little is left for L1, and a spilled register
// costs an L2 round trip).  Two more warps hold no word: the last keeps the grid
// barrier, the one before it reads the board and prepares the sources.
// FAR: some of the heavy words' synapses are in global memory.
template <bool BF16, uint32_t TL, uint32_t W, bool FAR>
__global__ void __launch_bounds__(fused_max_threads(W), 1) k_persistent_fused(StepArgs a,
                                                                              uint32_t n_steps) {
  __shared__ uint2 s_items[kBlockItems];
  __shared__ uint32_t s_n[2];  // item count of step parity p; the other one is reset
  __shared__ uint32_t s_wsum[kPersistBlock / 32];
  __shared__ uint32_t s_ptot;
  // Out-degree of each of the block's cells (word j of the block: cells 32 j ..).
  __shared__ uint32_t s_od[fused_max_words(W) * 32u];
  // Segment descriptors and stimulus sources, read every step, in shared
  // memory (when few enough): a miss in the small L1 that this kernel's
  // shared-memory carve-out leaves would cost an L2 round trip per step.
  constexpr uint32_t kSegCache = 16;
  __shared__ SegDev s_seg[kSegCache];
  __shared__ SrcDev s_src[kSrcCache];
  // Sources by substep of step t, buffer t mod 2: Poisson sources that are on,
  // periodic sources that fire.
  __shared__ uint2 s_on[2][kOnSubsteps];
  __shared__ int s_ok[2], s_board_ok;
  __shared__ uint16_t s_list[kBoardList];  // board_many
  extern __shared__ uint2 s_dyn[];
  const uint32_t n_thr = blockDim.x, n_wrp = n_thr >> 5, last = n_wrp - 1u;  // fused_threads
  const uint32_t aide = last - 1u, nw = aide;  // nw: warps that may hold words
  const bool heavy = a.hv_words != 0u && gridDim.x == a.hv_grid;
  const uint32_t n_own = (a.n_upd_words + gridDim.x - 1u) / gridDim.x;  // words of a block, at most
  const uint32_t nwk = (n_own + W - 1u) / W;                            // warps that hold them
  const uint32_t n_line = hv_line_slots(a), n_cell = n_own * 32u;
  int2* s_line = reinterpret_cast<int2*>(s_dyn);  // [n_line][n_cell]
  uint16_t* s_hoff = reinterpret_cast<uint16_t*>(s_line + (heavy ? n_line * n_cell : 0u));
  uint2* s_rows = s_dyn + hv_bytes(a, gridDim.x) / sizeof(uint2);
  uint2* s_hsyn = s_rows - (heavy ? a.hv_held : 0u);
  const uint2* far = FAR ? a.hv_syn + (size_t)blockIdx.x * a.hv_cap : nullptr;
  const SegDev* segs = a.n_segs <= kSegCache ? s_seg : a.segs;
  const SrcDev* srcs = a.n_srcs <= kSrcCache ? s_src : a.srcs;
  const bool shared_src = a.n_srcs <= kSrcCache && a.substeps <= (int)kOnSubsteps;
  if (a.n_segs <= kSegCache && threadIdx.x < a.n_segs) s_seg[threadIdx.x] = a.segs[threadIdx.x];
  if (a.n_srcs <= kSrcCache && threadIdx.x < a.n_srcs) s_src[threadIdx.x] = a.srcs[threadIdx.x];
  Ctl* ctl = a.ctl;
  const StepIdx ix0 = step_of(a);
  const unsigned long long t0 = ix0.t;
  uint32_t slot = ix0.slot;  // ring slot of the step at hand
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t wib = threadIdx.x >> 5;
  const bool leader = blockIdx.x == 0 && threadIdx.x == 0;
  // Words are dealt round-robin over the blocks (word j of block b is slot j x
  // blocks + b), so every SM holds about the same number of cells and spikes;
  // warp v holds the block's words v and v + nwk.
  // st: a LIF cell's state {u, g0, g1, ref}; an input cell's source mask and
  // index within its segment (bits of st.x, st.y).
  bool has[W], valid[W], lif[W], rd[W];
  uint32_t seg[W], i[W], cell[W], hw[W];  // cell: index in the block
  uint2 row[W];                           // first synapse, length | 1 << 31 when in shared memory
  float4 st[W];
#pragma unroll
  for (uint32_t k = 0; k < W; ++k) {
    const uint32_t j = wib + k * nwk, ws = j * gridDim.x + blockIdx.x;
    has[k] = wib < nwk && j < n_own && ws < a.n_upd_words;
    valid[k] = lif[k] = false;
    seg[k] = i[k] = 0;
    hw[k] = 0xFFFFu;
    cell[k] = has[k] ? j * 32u + lane : 0u;
    st[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    row[k] = make_uint2(0u, 0u);
    if (has[k]) {
      const uint32_t w = __ldg(a.upd_words + ws);
      seg[k] = __ldg(a.seg_of_word + w);
      i[k] = (w << 5) + lane;
      const SegDev& sd = a.segs[seg[k]];
      const uint32_t local = i[k] - sd.base;
      valid[k] = local < sd.count;
      lif[k] = sd.kind == kSegLif;
      if (heavy) hw[k] = __ldg(a.hv_index + w);
      uint32_t od = 0;
      if (valid[k]) {
        if (lif[k])
          st[k] = state_in(a.su[i[k]], a.sg[i[k]], sd.Vr);
        else
          st[k] = make_float4(__uint_as_float(__ldg(a.src_mask + i[k])), __uint_as_float(local), 0.f, 0.f);
        od = __ldg(a.outdeg + i[k]);
        const uint32_t r0 = __ldg(a.push_row + i[k]);
        const uint32_t r1 = heavy ? __ldg(a.push_split + i[k]) : __ldg(a.push_row + i[k] + 1);
        row[k] = make_uint2(r0, r1 - r0);
      }
      s_od[cell[k]] = od;
    }
    rd[k] = lif[k] && valid[k];
  }
  if (heavy) {
    for (uint32_t j = threadIdx.x; j < n_line * n_cell; j += n_thr) s_line[j] = make_int2(0, 0);
    const uint32_t n_off = a.hv_words * 32u + 1u;
    const uint16_t* off = a.hv_off + (size_t)blockIdx.x * n_off;
    // Within this launch's list also when the caller replays captured steps
    // whose tables have changed since.
    const uint32_t n = min((uint32_t)__ldg(off + n_off - 1u), a.hv_cap);
    for (uint32_t j = threadIdx.x; j < n_off; j += n_thr) s_hoff[j] = (uint16_t)min((uint32_t)__ldg(off + j), n);
    const uint2* src = a.hv_syn + (size_t)blockIdx.x * a.hv_cap;
    for (uint32_t j = threadIdx.x; j < (FAR ? min(n, a.hv_held) : n); j += n_thr) s_hsyn[j] = __ldg(src + j);
  }
  uint32_t stim = 0;  // bit k: the thread's cell of word k is a stimulated input cell
#pragma unroll
  for (uint32_t k = 0; k < W; ++k)
    if (valid[k] && !lif[k] && __float_as_uint(st[k].x) != 0u) stim |= 1u << k;
  if (threadIdx.x == 0) {
    s_n[0] = s_n[1] = 0;
    s_board_ok = 1;
  }
  const bool blk_stim = __syncthreads_or((int)stim) != 0;  // also publishes s_seg / s_src
  auto sources = [&](unsigned long long t) {
    source_states(s_src, s_on[t & 1ull], a.n_srcs, (uint32_t)a.substeps, t);
  };
  // Element k of a pair, without indexing registers.
  auto pick = [](uint32_t k, uint32_t x, uint32_t y) { return k ? y : x; };
  // The stimulus decisions of the thread's input cells in step t, bit k for word k.
  auto draw = [&](unsigned long long t) -> uint32_t {
    uint32_t fire = 0;
#pragma unroll 1
    for (uint32_t k = 0; k < W; ++k) {
      if (!((stim >> k) & 1u)) continue;
      const SegDev& sd = segs[pick(k, seg[0], seg[W - 1])];
      const uint32_t mask = __float_as_uint(k ? st[W - 1].x : st[0].x);
      const uint32_t local = __float_as_uint(k ? st[W - 1].y : st[0].y);
      if (!shared_src) {
        fire |= (input_fire(a, srcs, sd, local, mask, t) ? 1u : 0u) << k;
        continue;
      }
      bool f = false;
      U4 r{};
#pragma unroll 1
      for (int s = 0; s < a.substeps; ++s) {
        if ((s & 3) == 0) r = philox_draw(sd.seed, sd.key_base + local, t, kTagInput, (uint32_t)(s >> 2));
        const uint32_t x = u4_get(r, s & 3);
        const uint2 on = s_on[t & 1ull][s];
        f |= (mask & on.y) != 0u;
#pragma unroll 1
        for (uint32_t m = mask & on.x; m; m &= m - 1u) f |= (uint64_t)x < s_src[__ffs(m) - 1].thresh;
      }
      fire |= (f ? 1u : 0u) << k;
    }
    return fire;
  };
  const bool shared_on = blk_stim && shared_src;
  uint32_t walked = 0;
  constexpr uint32_t kBatch = W == 1u ? 2u : 3u;  // synapses a lane has in flight; one more would spill
  // Pushes m synapses from b0 of the block's rows or of the table; delays count
  // from ring slot `own`.
  auto push_range = [&](uint32_t b0, uint32_t m, bool smem, uint32_t own) {
#pragma unroll 1
    for (uint32_t j0 = lane; j0 < m; j0 += 32u * kBatch) {
      uint2 e[kBatch];
#pragma unroll
      for (uint32_t k = 0; k < kBatch; ++k) {
        const uint32_t j = j0 + 32u * k;
        if (j >= m) break;
        e[k] = smem ? s_rows[b0 + j]
                    : make_uint2(__ldg(a.push_syn + b0 + j),
                                 (uint32_t)__float2int_rn(load_weight<BF16>(a.push_w, b0 + j)));
      }
#pragma unroll
      for (uint32_t k = 0; k < kBatch; ++k) {
        if (j0 + 32u * k >= m) break;
        uint32_t slot = own + ((e[k].x >> kPushPostBits) & 15u);
        if (slot >= a.ring_slots) slot -= a.ring_slots;
        atomicAdd(a.ring + (((size_t)slot * a.n_pad + (e[k].x & kPushPostMask)) << 1) + (e[k].x >> 31),
                  (int)e[k].y);
      }
    }
    walked += m;
  };
  // Input cells: the decision of the coming step is drawn ahead (it depends
  // only on the step index).  The launch's first two come from the general
  // form; the loops draw the later ones with the shared source states.
  uint32_t next_in = 0, next1 = 0;
#pragma unroll
  for (uint32_t k = 0; k < W; ++k)
    if ((stim >> k) & 1u) {
#pragma unroll 1
      for (uint32_t q = 0; q < 2u && q < n_steps; ++q) {
        const bool f = input_fire(a, srcs, segs[seg[k]], __float_as_uint(st[k].y), __float_as_uint(st[k].x), t0 + q);
        if (f) (q ? next1 : next_in) |= 1u << k;
      }
      if (shared_src) st[k].x = __uint_as_float(__float_as_uint(st[k].x) << segs[seg[k]].src_first);
    }
  // Push rows into shared memory.  Rows of at least kLongRow synapses are
  // placed first (a spike of such a cell is the most work to push), then the
  // others, each in word order; a row that no longer fits stays in global memory.
  constexpr uint32_t kLongRow = 128;
  const size_t hv = hv_bytes(a, gridDim.x);
  const uint32_t cap = a.row_smem > hv ? (uint32_t)((a.row_smem - hv) / sizeof(uint2)) : 0u;
  uint32_t used = 0;
  bool has_long = false;
#pragma unroll
  for (uint32_t k = 0; k < W; ++k) has_long |= row[k].y > a.direct_row;
#pragma unroll 1
  for (uint32_t pass = 0; pass < 2u && cap; ++pass) {
#pragma unroll
    for (uint32_t k = 0; k < W; ++k) {
      const uint32_t lp = !(row[k].y >> 31) && (row[k].y >= kLongRow) == (pass == 0) ? row[k].y : 0u;
      uint32_t incl = lp;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += v;
      }
      __syncthreads();  // s_wsum's previous readers are done
      if (lane == 31) s_wsum[wib] = incl;
      __syncthreads();
      if (wib == 0) {
        uint32_t x = lane < n_wrp ? s_wsum[lane] : 0u, xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(kFull, xi, o);
          if (lane >= (uint32_t)o) xi += v;
        }
        s_wsum[lane] = xi - x;
        if (lane == 31) s_ptot = xi;
      }
      __syncthreads();
      const uint32_t base = used + s_wsum[wib] + incl - lp;
      used += s_ptot;
      const bool fits = lp && base <= cap && lp <= cap - base;
      uint32_t todo = __ballot_sync(kFull, fits);
#pragma unroll 1
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint32_t q0 = __shfl_sync(kFull, row[k].x, src), n = __shfl_sync(kFull, lp, src);
        const uint32_t b0 = __shfl_sync(kFull, base, src);
        for (uint32_t j = lane; j < n; j += 32)
          s_rows[b0 + j] = make_uint2(__ldg(a.push_syn + q0 + j),
                                      (uint32_t)__float2int_rn(load_weight<BF16>(a.push_w, q0 + j)));
      }
      if (fits) row[k] = make_uint2(base, lp | 0x80000000u);
    }
  }
  const bool blk_long = __syncthreads_or((int)has_long) != 0;  // also: rows are in place
  const uint32_t clog = a.item_log2, chunk = 1u << clog;  // push-item width
  unsigned long long target = 0;
  bool aborted = false;
  // History and summary rows are for the other kernels and the host: a launch
  // writes those of its last hist_rows steps (rel: chunk step), and clears their
  // summary rows and its successor's before.
  const uint32_t n_hist = a.hist_rows;
  auto keeps = [&](uint32_t rel) { return rel + n_hist >= n_steps; };
  auto clear_summary = [&](uint32_t rel, uint32_t gtid, uint32_t gthreads) {
    if (!keeps(rel) || rel > n_steps) return;
    const uint32_t row = (ix0.srow + rel) % (n_hist + 1u);
    for (uint32_t j = gtid; j < a.n_swords; j += gthreads)
      __stcg(a.hsum + (size_t)row * a.n_swords + j, 0u);
  };
  // Spike bookkeeping of this warp's words for the spikes of chunk step `rel`
  // (ring slot px; fired: bit k for word k): the board, history, per-segment
  // count, events, raster entries; then the spiking cells' rows, pushed from
  // here, or cut into the items of parity rel & 1.
  auto publish = [&](uint32_t fired, uint32_t rel, uint32_t px) {
    uint32_t b[W];
#pragma unroll
    for (uint32_t k = 0; k < W; ++k) b[k] = __ballot_sync(kFull, (fired >> k) & 1u);
    if ((hw[0] & hw[W - 1]) != 0xFFFFu && lane < W) {
      const uint32_t h = pick(lane, hw[0], hw[W - 1]);
      const unsigned long long v = ((unsigned long long)(rel + 1u) << 32) | pick(lane, b[0], b[W - 1]);
      if (h != 0xFFFFu)
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(a.board + (rel & 3u) * kHeavyWords + h),
                     "l"(v) : "memory");
    }
    if (keeps(rel) && lane == 0) {
      StepIdx hx = ix0;
      hx.hrow = (ix0.hrow + rel) % n_hist;
      hx.srow = (ix0.srow + rel) % (n_hist + 1u);
      ix_rows(a, hx);
#pragma unroll
      for (uint32_t k = 0; k < W; ++k)
        if (has[k]) put_hist(a, hx, i[k] >> 5, b[k]);
    }
    if (__builtin_expect((b[0] | b[W - 1]) == 0u, 0)) return;
#pragma unroll 1
    for (uint32_t k = 0; k < W; ++k) {
      const uint32_t ballot = pick(k, b[0], b[W - 1]);
      if (!ballot) continue;
      const bool mine = (ballot >> lane) & 1u;
      if (lane == 0)
        atomicAdd(&a.counts[(size_t)rel * a.n_segs + pick(k, seg[0], seg[W - 1])], (uint32_t)__popc(ballot));
      if (mine) atomicAdd(&ctl->events, (unsigned long long)s_od[pick(k, cell[0], cell[W - 1])]);
      const uint32_t rx = pick(k, row[0].x, row[W - 1].x), ry = pick(k, row[0].y, row[W - 1].y);
      const uint32_t n = ry & 0x7FFFFFFFu;
      uint32_t todo = __ballot_sync(kFull, mine && n != 0u && n <= a.direct_row);
#pragma unroll 1
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1u;
        const uint32_t b0 = __shfl_sync(kFull, rx, src), l0 = __shfl_sync(kFull, ry, src);
        push_range(b0, l0 & 0x7FFFFFFFu, (l0 >> 31) != 0u, px);
      }
      if (blk_long) {
        // Long rows: items of the block's list, and from here what it has no room for.
        uint32_t from = 0;
        const bool is_long = mine && n > a.direct_row;
        if (is_long) {
          const uint32_t nit = (n + chunk - 1u) >> clog;
          const uint32_t off = atomicAdd(&s_n[rel & 1u], nit);
          const uint32_t put = off < kBlockItems ? min(nit, kBlockItems - off) : 0u;
#pragma unroll 1
          for (uint32_t q = 0; q < put; ++q)
            s_items[off + q] = make_uint2(rx + (q << clog), (min(chunk, n - (q << clog)) << 23) | (ry >> 31));
          from = min(n, put << clog);
        }
        todo = __ballot_sync(kFull, is_long && from < n);
#pragma unroll 1
        while (todo) {
          const int src = __ffs(todo) - 1;
          todo &= todo - 1u;
          const uint32_t b0 = __shfl_sync(kFull, rx, src), l0 = __shfl_sync(kFull, ry, src);
          const uint32_t f0 = __shfl_sync(kFull, from, src);
          push_range(b0 + f0, (l0 & 0x7FFFFFFFu) - f0, (l0 >> 31) != 0u, px);
        }
      }
      if (a.raster_cap) {
        uint32_t roff = 0;
        if (lane == 0) roff = atomicAdd(&ctl->raster_count, (uint32_t)__popc(ballot));
        roff = __shfl_sync(kFull, roff, 0);
        if (mine) {
          const uint32_t to = roff + __popc(ballot & ((1u << lane) - 1u));
          if (to < a.raster_cap)
            a.raster[to] = raster_record(pick(k, i[0], i[W - 1]), rel);
          else
            atomicOr(&ctl->error, kErrRasterOverflow);
        }
      }
    }
  };
  // Blocks with long rows: the items of parity par, by the first n_w warps (when
  // not all, they meet on block barrier 1); delays count from ring slot `own`.
  auto deliver = [&](uint32_t par, uint32_t own, uint32_t n_w) {
    if (!blk_long) return;
    if (n_w == n_wrp) __syncthreads(); else bar_sync_first(n_w * 32u);
    const uint32_t n_items = min(s_n[par], kBlockItems);
    // The other parity's count was last read before this block barrier.
    if (threadIdx.x == 0) s_n[par ^ 1u] = 0;
#pragma unroll 1
    for (uint32_t u = wib; u < n_items; u += n_w) {
      const uint2 it = s_items[u];
      push_range(it.x, it.y >> 23, (it.y & 1u) != 0u, own);
    }
  };
  // The heavy words' spikes of chunk step rel into the line, whose slot of that
  // step is `at`; one warp.  A word's tag comes before its owner's arrival
  // at the barrier that this step waits for; the wait has that barrier's limit.
  auto board = [&](uint32_t rel, uint32_t at) {
    // Up to four words per lane, read together.
    uint32_t got[kHeavyWords / 32u];
    {
      const unsigned long long* p = a.board + (rel & 3u) * kHeavyWords + lane;
      unsigned long long w0 = 0;
      uint32_t it = 0;
      while (true) {
        bool all = true;
        unsigned long long v[kHeavyWords / 32u];
#pragma unroll
        for (uint32_t k = 0; k < kHeavyWords / 32u; ++k) {
          v[k] = (unsigned long long)(rel + 1u) << 32;
          if (lane + 32u * k < a.hv_words)
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[k]) : "l"(p + 32u * k) : "memory");
        }
#pragma unroll
        for (uint32_t k = 0; k < kHeavyWords / 32u; ++k) {
          all = all && (uint32_t)(v[k] >> 32) == rel + 1u;
          got[k] = (uint32_t)v[k];
        }
        if (__all_sync(kFull, all)) break;
        if ((++it & 255u) == 0u) {
          const unsigned long long now = global_ns();
          if (w0 == 0) w0 = now;
          const bool out = now - w0 > kBarrierTimeoutNs || (__ldcg(&ctl->error) & kErrBarrierTimeout);
          if (__any_sync(kFull, out)) {
            if (lane == 0) {
              atomicOr(&ctl->error, kErrBarrierTimeout);
              s_board_ok = 0;
            }
            return;
          }
        }
        __nanosleep(32);
      }
    }
    uint32_t nz = 0;
#pragma unroll
    for (uint32_t k = 0; k < kHeavyWords / 32u; ++k) nz |= got[k];
    const uint32_t busy = __popc(__ballot_sync(kFull, nz != 0u));
    if (busy > kBoardFew) {
      const uint4 g = make_uint4(got[0], got[1], got[2], got[3]);
      walked += W == 1u ? board_many_call<FAR>(g, s_hoff, s_hsyn, s_line, s_list, at, n_line, n_cell, far, a.hv_held)
                        : board_many<FAR>(g, s_hoff, s_hsyn, s_line, s_list, at, n_line, n_cell, far, a.hv_held);
      return;
    }
#pragma unroll
    for (uint32_t k = 0; k < kHeavyWords / 32u; ++k) {
      const uint32_t k0 = 32u * k, bits = got[k];
      uint32_t words = __ballot_sync(kFull, bits != 0u);
#pragma unroll 1
      while (words) {
        const int src = __ffs(words) - 1;
        words &= words - 1u;
        uint32_t b = __shfl_sync(kFull, bits, src);
#pragma unroll 1
        while (b) {
          const uint32_t c = (k0 + src) * 32u + __ffs(b) - 1u;
          b &= b - 1u;
          const uint32_t q1 = s_hoff[c + 1u];
          walked += q1 - s_hoff[c];
#pragma unroll 1
          for (uint32_t q = s_hoff[c] + lane; q < q1; q += 32u) {
            // {cell | delay << 10 | accumulator << 14, increment}
            const uint2 e = FAR && q >= a.hv_held ? __ldg(far + q) : s_hsyn[q];
            uint32_t slot = at + ((e.x >> 10) & 15u);
            if (slot >= n_line) slot -= n_line;
            atomicAdd(reinterpret_cast<int*>(s_line + slot * n_cell + (e.x & 1023u)) + (e.x >> 14), (int)e.y);
          }
        }
      }
    }
  };
  // The increments of the thread's cells in ring slot `slot` and the line's slot
  // `at`; clear_in takes them out of the ring (the line's go as they are read).
  int2* ring2 = reinterpret_cast<int2*>(a.ring);
  uint32_t at = 0;  // the line's slot of the step at hand
  auto take = [&](int2 (&in)[W], int2 (&acc)[W]) {
#pragma unroll
    for (uint32_t k = 0; k < W; ++k) {
      in[k] = make_int2(0, 0);
      if (rd[k]) in[k] = __ldcg(ring2 + (slot * a.n_pad + i[k]));
    }
#pragma unroll
    for (uint32_t k = 0; k < W; ++k) {
      acc[k] = in[k];
      if (heavy && rd[k]) {
        int2* p = s_line + at * n_cell + cell[k];
        const int2 l = *p;
        if (l.x | l.y) *p = make_int2(0, 0);
        acc[k] = make_int2(in[k].x + l.x, in[k].y + l.y);
      }
    }
  };
  auto clear_in = [&](uint32_t from, const int2 (&in)[W]) {
#pragma unroll
    for (uint32_t k = 0; k < W; ++k)
      if (in[k].x | in[k].y) __stcg(ring2 + (from * a.n_pad + i[k]), make_int2(0, 0));
  };
  auto next_step = [&]() {
    at = at + 1u == n_line ? 0u : at + 1u;
    slot = slot + 1u == a.ring_slots ? 0u : slot + 1u;
  };
  if (TL == 0) {
    // Step t: update (slot t), spikes of t, their pushes; one grid barrier.
    for (uint32_t s = 0; s < n_steps; ++s) {
      clear_summary(s + 1u, blockIdx.x * n_thr + threadIdx.x, gridDim.x * n_thr);
      if (wib < nwk) {
        uint32_t fired = next_in;
        int2 in[W], acc[W];
        take(in, acc);
        clear_in(slot, in);
#pragma unroll
        for (uint32_t k = 0; k < W; ++k)
          if (lif[k] && lif_step(lif_k(segs[seg[k]]), a.substeps, st[k], acc[k]) && valid[k]) fired |= 1u << k;
        publish(fired, s, slot);
      }
      deliver(s & 1u, slot, n_wrp);
      grid_arrive(a, target);
      if (stim && s + 1 < n_steps) next_in = s == 0u ? next1 : draw(t0 + s + 1ull);
      if (wib == aide) {
        if (heavy) board(s, at);
        if (shared_on) sources(t0 + s + 2ull);
      }
      next_step();
      if (!grid_wait(a, target, last * 32u) || !s_board_ok) {
        aborted = true;
        break;
      }
    }
  } else {
    // Late-push timelines (one substep per step).  A cell's spike of step t + 1
    // is decided by its potential after the update of step t (the spike test
    // reads the potential before the step's integration), so step t updates
    // with ring slot t and publishes the spikes of t + 1, whose pushes target
    // slots t + 2 and later: they are first read after the barrier of step
    // t + 1.
    //   TL 1: a block arrives at step t's barrier as soon as its cells are
    // updated, and only then makes the step's writes -- the clears of the slot
    // it consumed, the history words, counts and pushes of the new spikes --
    // while the other blocks arrive: the next arrival's release carries them.
    // A clear made after step t's arrival is ordered before the pushes of step
    // t + 2 and later only; with max_delay + 3 ring slots no push of step t + 1
    // targets slot t again.
    //   TL 2: every write of step t is first read in step t + 2, so the barrier
    // is split: at the top of step t + 1, after the block barrier that ends
    // step t, the last warp fences the block's writes of step t and arrives;
    // the block waits for the other blocks' arrivals only at the end of step
    // t + 1, before step t + 2 reads slot t + 2.  Arrival, fence and barrier
    // latency overlap a step's work, and blocks run at most one step apart:
    // the last warp clears the summary row of step t + 2 at the top of step t,
    // before its fence (its bits are set in step t + 1), and the raster
    // records of neighbouring steps may interleave (each record carries its
    // step mod 4).
    //   The last warp arrives and polls while the others work (they meet on block
    // barrier 1), so the arrival's release stalls no warp with work.
    // The prologue is the loop's round s = -1: it only publishes and pushes.
    uint32_t in_next = next_in;  // input spikes of step t + 1, drawn a step ahead
    if (TL == 2) clear_summary(1u, blockIdx.x * n_thr + threadIdx.x, gridDim.x * n_thr);
#pragma unroll 1
    for (int s = -1; s < (int)n_steps; ++s) {
      const uint32_t rel = (uint32_t)(s + 1);  // the chunk step whose spikes this round publishes
      const bool more = rel < n_steps;
      if (s < 0 && !more) break;
      int2 in[W];
      const uint32_t consumed = slot;
      uint32_t fired = in_next;
      if (s >= 0) {
        target += gridDim.x;
        if (TL == 2 && wib == last) {
          clear_summary(rel + 1u, blockIdx.x * 32u + lane, gridDim.x * 32u);
          __syncwarp();
          if (lane == 0) grid_arrive_fenced(a);
          __syncwarp();
        }
      }
      if (wib < nwk) {
        int2 acc[W];
        if (s >= 0) take(in, acc);
        LifK c = lif_k(segs[seg[0]]);
#pragma unroll
        for (uint32_t k = 0; k < W; ++k) {
          if (k && seg[k] != seg[0]) c = lif_k(segs[seg[k]]);
          if (s >= 0 && rd[k]) lif_update<1>(c, 1, st[k], acc[k]);
          if (rd[k] && st[k].x > c.Vth) fired |= 1u << k;
        }
      }
      const uint32_t line_at = at;
      if (s >= 0) next_step();  // from here on slot and at are those of step `rel`
      if (TL == 1) {
        clear_summary(rel + 1u, blockIdx.x * n_thr + threadIdx.x, gridDim.x * n_thr);
        __syncthreads();  // the block's updates (and the previous step's writes) are done
        if (s >= 0 && threadIdx.x == last * 32u)
          asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(a.bar) : "memory");
      }
      if (wib < nw) {
        if (wib < nwk) {
          if (s >= 0) clear_in(consumed, in);
          if (more) publish(fired, rel, slot);
        }
        deliver(rel & 1u, slot, nw);
        if (stim && rel + 1u < n_steps) in_next = s < 0 ? next1 : draw(t0 + rel + 1ull);
      }
      if (wib == aide) {
        if (heavy && s >= 0) board((uint32_t)s, line_at);
        if (shared_on) sources(t0 + rel + 2ull);
      }
      if (s < 0) {
        if (TL == 1) {
          grid_arrive(a, target);  // with the prologue's writes, before the first update's
          if (threadIdx.x == last * 32u) s_ok[rel & 1u] = poll_arrivals(a, target);
        } else if (threadIdx.x == 0) {
          s_ok[rel & 1u] = 1;
        }
      } else if (threadIdx.x == last * 32u) {
        // A board that ran out of time ends the launch here or a round later.
        s_ok[rel & 1u] = poll_arrivals(a, target) && *(volatile int*)&s_board_ok;
      }
      __syncthreads();  // ends the step: the next arrival's release carries its writes
      if (!s_ok[rel & 1u]) {
        aborted = true;
        break;
      }
    }
  }
  // The line's pending increments (steps t0 + n_steps and later) into the ring.
  if (heavy && !aborted) {
#pragma unroll 1
    for (uint32_t d = 0; d < a.max_delay; ++d) {
#pragma unroll
      for (uint32_t k = 0; k < W; ++k) {
        if (!rd[k]) continue;
        const int2 l = s_line[at * n_cell + cell[k]];
        int* p = a.ring + (((size_t)slot * a.n_pad + i[k]) << 1);
        if (l.x) atomicAdd(p, l.x);
        if (l.y) atomicAdd(p + 1, l.y);
      }
      next_step();
    }
  }
#pragma unroll
  for (uint32_t k = 0; k < W; ++k)
    if (rd[k]) state_out(a, i[k], st[k]);
  if (a.raster_cap && blockIdx.x == 0) raster_offsets_from_counts(a, n_steps, s_wsum);
  if (__ldcg(&ctl->error) & kErrBarrierTimeout) return;
  if (lane == 0 && walked) atomicAdd(&ctl->delivered, (unsigned long long)walked);
  if (leader) {
    ctl->step = t0 + n_steps;
    ctl->ring_slot = (ix0.slot + n_steps) % a.ring_slots;
    ctl->hist_row = (ix0.hrow + n_steps) % n_hist;
    ctl->t_rel = n_steps;
  }
}

}  // namespace

cudaError_t launch_chunk_begin(const StepArgs& a, uint32_t steps, uint32_t n_bar, const SrcDev* srcs,
                               cudaStream_t s) {
  const size_t n = std::max<size_t>((size_t)steps * a.n_segs, n_bar);
  k_chunk_begin<<<(int)std::min<size_t>(n / (4 * kBlock) + 1, a.sms), kBlock, 0, s>>>(a, steps, n_bar, srcs);
  return cudaGetLastError();
}

cudaError_t launch_state_out(const StepArgs& a, const long long* first, float* u, float2* g, int32_t* ref,
                             cudaStream_t s) {
  k_state_out<<<(a.n_pad + kBlock - 1) / kBlock, kBlock, 0, s>>>(a, first, u, g, ref);
  return cudaGetLastError();
}

// Launches a kernel of a step behind the previous one; without plastic
// projections (whose plasticity runs on a forked stream) as its programmatic
// dependent.
static cudaError_t step_launch(void (*fn)(StepArgs), const StepArgs& a, int blocks, int threads, size_t smem,
                               cudaStream_t s) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = a.n_plast ? 0 : 1;
  return cudaLaunchKernelEx(&cfg, fn, a);
}

cudaError_t launch_update(const StepArgs& a, cudaStream_t s) {
  if (!a.n_upd_words) return cudaSuccess;
  // The loop's warps get their words ahead, so words that differ much in work
  // (input cells draw for each substep) are better left to waves of blocks:
  // 370,200 cells, ten substeps, 14.4 us per step in waves, 16.4 looped.
  const uint32_t blocks = (a.n_words + kBlock / 32 - 1) / (kBlock / 32), most = a.sms * kUpdateBlocks;
  const bool loop = blocks > most && a.substeps == 1;
  return step_launch(loop ? k_update<true> : k_update<false>, a, loop ? most : blocks, kBlock, 0, s);
}

cudaError_t launch_deliver(const StepArgs& a, int blocks, cudaStream_t s) {
  // Without push rows only the step's bookkeeping is left, one block's work.
  // All projections dense, 92,550 cells: 12.1 -> 10.9 us per step.
  return step_launch(a.bf16 ? k_deliver<true> : k_deliver<false>, a, a.any_push ? blocks : 1, kBlock, 0, s);
}

size_t pull_sum_bytes(const StepArgs& a) { return ((size_t)a.hist_rows * a.n_swords + 1) * 4; }
size_t seg_smem_bytes(const StepArgs& a) { return seg_smem_bytes_dev(a); }

static size_t pull_smem_bytes(const StepArgs& a) { return a.pull_sum ? pull_sum_bytes(a) : 0; }

cudaError_t launch_pull(const StepArgs& a, int blocks, cudaStream_t s) {
  if (!a.n_pull_units) return cudaSuccess;
  if (a.pull_sum == 2u)
    return step_launch(a.bf16 ? k_pull_vec<true> : k_pull_vec<false>, a, blocks, kPullBlock, pull_sum_bytes(a), s);
  void (*fn)(StepArgs) = a.bf16 ? (a.pull_sum ? k_pull<true, true> : k_pull<true, false>)
                                : (a.pull_sum ? k_pull<false, true> : k_pull<false, false>);
  return step_launch(fn, a, blocks, kPullBlock, pull_smem_bytes(a), s);
}

cudaError_t launch_stdp(const StepArgs& a, int blocks, cudaStream_t s, bool early) {
  if (!a.n_stdp_units) return cudaSuccess;
  if (a.bf16) {
    if (early) k_stdp<true, true><<<blocks, kBlock, 0, s>>>(a);
    else k_stdp<true, false><<<blocks, kBlock, 0, s>>>(a);
  } else {
    if (early) k_stdp<false, true><<<blocks, kBlock, 0, s>>>(a);
    else k_stdp<false, false><<<blocks, kBlock, 0, s>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_plast_reset(const StepArgs& a, int blocks, cudaStream_t s) {
  if (!a.n_stdp_units) return cudaSuccess;
  if (a.bf16)
    k_plast_reset<true><<<blocks, kBlock, 0, s>>>(a);
  else
    k_plast_reset<false><<<blocks, kBlock, 0, s>>>(a);
  return cudaGetLastError();
}

// k_persistent_pull by [BF16][block size up to kPullSmall or any]: with at most
// 24 warps its threads may have 80 registers, so that nothing spills.
// A warp for each of the block's words and one that keeps the grid barrier, at
// least kPullWarps for the entries (16 warps: 2 % slower, 32 with 64
// registers: 7 %).
constexpr uint32_t kPullSmall = 768, kPullWarps = 24;
static const void* const kPullKernels[] = {
    (const void*)k_persistent_pull<false, kPullSmall>, (const void*)k_persistent_pull<false, kPersistBlock>,
    (const void*)k_persistent_pull<true, kPullSmall>, (const void*)k_persistent_pull<true, kPersistBlock>};
static uint32_t pull_threads(const StepArgs& a, int blocks) {
  const uint32_t words = (a.n_upd_words + (uint32_t)blocks - 1u) / (uint32_t)blocks;
  return 32u * std::min(std::max(words + 1u, kPullWarps), (uint32_t)kPersistBlock / 32u);
}
static const void* pull_kernel(const StepArgs& a, int blocks) {
  return kPullKernels[(a.bf16 ? 2 : 0) + (pull_threads(a, blocks) > kPullSmall ? 1 : 0)];
}

// Dynamic shared memory a kernel can take beside its static part.
static size_t dyn_smem_max(const void* fn) {
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  cudaFuncAttributes fa{};
  if (cudaFuncGetAttributes(&fa, fn) != cudaSuccess || (size_t)optin <= fa.sharedSizeBytes) return 0;
  return ((size_t)optin - fa.sharedSizeBytes) & ~(size_t)255;
}

// The fused kernel's forms: [FAR][BF16][timeline][words per warp - 1].
#define SGB_FUSED_FORMS(B, F)                                                        \
  (const void*)k_persistent_fused<B, 0, 1, F>, (const void*)k_persistent_fused<B, 0, 2, F>,     \
      (const void*)k_persistent_fused<B, 1, 1, F>, (const void*)k_persistent_fused<B, 1, 2, F>, \
      (const void*)k_persistent_fused<B, 2, 1, F>, (const void*)k_persistent_fused<B, 2, 2, F>
constexpr uint32_t kFusedForms = 6;
static const void* const kFusedKernels[] = {SGB_FUSED_FORMS(false, false), SGB_FUSED_FORMS(true, false),
                                            SGB_FUSED_FORMS(false, true), SGB_FUSED_FORMS(true, true)};
#undef SGB_FUSED_FORMS

cudaError_t pull_setup() {
  const int mx = (int)kPullSumMax;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(k_pull_vec<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_pull_vec<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;

  if ((e = cudaFuncSetAttribute(k_pull<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_pull<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_pull<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_pull<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  // The persistent kernels stage the same summary rows before their deliveries.
  if ((e = cudaFuncSetAttribute(k_persistent<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_persistent<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_persistent<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_persistent<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_persistent<true, true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_persistent<false, true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx))) return e;
  if ((e = cudaFuncSetAttribute(k_persistent_resident<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx)))
    return e;
  // The limit belongs to the function, for every handle of the process, so it
  // is the most that the function can take; a launch names its own size.
  for (const void* fn : kFusedKernels)
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_smem_max(fn))))
      return e;
  for (const void* fn : kPullKernels)
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn_smem_max(fn))))
      return e;
  return cudaFuncSetAttribute(k_persistent_resident<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
}

int pull_blocks_per_sm(const StepArgs& a) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_pull<true, true>, kPullBlock, pull_smem_bytes(a));
  return n > 0 ? n : 1;
}

cudaError_t launch_chunk_end(const StepArgs& a, uint32_t* host_err, uint32_t* host_counts, cudaStream_t s) {
  k_chunk_end<<<std::max(a.n_segs, 1u), kBlock, 0, s>>>(a, host_err, host_counts);
  return cudaGetLastError();
}

// Words per block, at most, and per warp: a warp without a word still runs a
// step's bookkeeping, and in steps bound by latency those instructions delay
// the warps with work, so blocks are no larger than needed (9,256 cells, two
// words a block: 1.73 us per step with 32 warps, 1.58 with 8).
static uint32_t fused_words(const StepArgs& a, int blocks) {
  return (a.n_upd_words + (uint32_t)blocks - 1u) / (uint32_t)blocks;
}
static uint32_t fused_per_warp(const StepArgs& a, int blocks) {
  return fused_words(a, blocks) <= kFusedSingle ? 1u : 2u;
}
constexpr uint32_t kFusedWarps = 8;  // at least
static uint32_t fused_threads(const StepArgs& a, int blocks) {
  const uint32_t w = fused_per_warp(a, blocks);
  return 32u * std::max((fused_words(a, blocks) + w - 1u) / w + 2u, kFusedWarps);
}
size_t fused_heavy_bytes(const StepArgs& a, int blocks) { return hv_bytes(a, (uint32_t)blocks); }

// The timeline and item width the fused kernel runs with for these arguments.
uint32_t fused_timeline(const StepArgs& a) { return a.substeps == 1 ? std::min(a.ahead, 2u) : 0u; }
uint32_t fused_item_log2(const StepArgs& a) {
  return fused_timeline(a) ? (a.item_log2 >= 7 ? 7u : 6u) : 6u;
}

static const void* fused_kernel(const StepArgs& a, int blocks) {
  const uint32_t far = a.hv_words && a.hv_held < a.hv_cap ? 2u * kFusedForms : 0u;
  return kFusedKernels[far + (a.bf16 ? kFusedForms : 0u) + 2u * fused_timeline(a) + fused_per_warp(a, blocks) - 1u];
}

static int fused_blocks_per_sm() {
  int n = 1 << 20;
  for (uint32_t k = 0; k < 4u * kFusedForms; ++k) {
    int f = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f, kFusedKernels[k], (int)fused_max_threads(k % 2u + 1u), 0);
    n = f < n ? f : n;
  }
  return n;
}

int persistent_blocks_per_sm(bool bf16) {
  int n = 0, m = 0;
  int f = 0;
  int o = 0;
  if (bf16) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_persistent<true, true>, kPersistBlock, 0);
    int q = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, k_persistent<true, true, 2>, kPersistBlock, 0);
    o = o < q ? o : q;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_persistent<true, false>, kPersistBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_persistent_resident<true>, kPersistBlock, 0);
    f = fused_blocks_per_sm();
  } else {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_persistent<false, true>, kPersistBlock, 0);
    int q = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&q, k_persistent<false, true, 2>, kPersistBlock, 0);
    o = o < q ? o : q;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_persistent<false, false>, kPersistBlock, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_persistent_resident<false>, kPersistBlock, 0);
    f = fused_blocks_per_sm();
  }
  n = n < m ? n : m;
  n = n < o ? n : o;
  return n < f ? n : f;
}

// The general kernel's one-barrier form: no dense pulls, no plastic rule
// that reads the step's own spikes.
bool general_one_barrier(const StepArgs& a) {
  return a.n_pull_units == 0 && (a.n_plast == 0 || a.stdp_early);
}

int persistent_kernel_kind(const StepArgs& a, int blocks) {
  const bool resident = (uint64_t)a.n_upd_words * 32u <= (uint64_t)blocks * kPersistBlock;
  if (!resident) return SGB_KERNEL_GENERAL;
  return a.n_pull_units == 0 ? SGB_KERNEL_FUSED : SGB_KERNEL_RESIDENT;
}

// Resident networks with dense pulls, one substep a step: k_persistent_pull,
// when the history rows it keeps fit shared memory, no writer of row t + 1 can
// meet a reader of row t (two rows), and the plastic windows, if any, come
// from the spike registers.  Sets its dynamic shared memory (0: the two-barrier
// form runs) and the pull units per block whose entries that holds.
void plan_persistent_pull(StepArgs& a, int blocks) {
  a.pull_smem = a.pull_held = 0;
  if (blocks <= 0 || !a.n_pull_units || a.substeps != 1 || a.hist_rows < 2u || (a.n_plast && !a.recent3)) return;
  if (persistent_kernel_kind(a, blocks) != SGB_KERNEL_RESIDENT) return;
  const size_t most = dyn_smem_max(pull_kernel(a, blocks));
  const size_t fixed = pull_fixed_bytes(a);
  // The word of an entry's spike bit shares 32 bits with its place in the unit.
  if (fixed > most || pull_rows(a) * a.n_words >= 1u << (32 - kWordShift)) return;
  const uint32_t mine = (a.n_pull_units + (uint32_t)blocks - 1u) / (uint32_t)blocks;
  a.pull_held = (uint32_t)std::min<size_t>(mine, (most - fixed) / pull_unit_bytes(a));
  a.pull_smem = (uint32_t)(fixed + (size_t)a.pull_held * pull_unit_bytes(a));
}

cudaError_t launch_pull_sort(const StepArgs& a, cudaStream_t s) {
  k_pull_sort<<<a.n_pull_units, kPullUnit / 2, 0, s>>>(a, const_cast<uint32_t*>(a.pull_sorted),
                                                       const_cast<uint4*>(a.pull_info));
  return cudaGetLastError();
}

cudaError_t launch_persistent(const StepArgs& a, uint32_t n_steps, int blocks, cudaStream_t s) {
  StepArgs args = a;
  uint32_t n = n_steps;
  void* params[] = {&args, &n};
  const int kind = persistent_kernel_kind(a, blocks);
  // Without heavy words every row is pushed by its cell's block; the delay line
  // is handed back to the ring at a launch's end, so launches may differ.
  if (a.hv_busy) args.hv_words = 0;
  if (kind == SGB_KERNEL_RESIDENT && a.pull_smem)
    return cudaLaunchCooperativeKernel(pull_kernel(a, blocks), dim3(blocks),
                                       dim3(pull_threads(a, blocks)), params, a.pull_smem, s);
  const bool resident = kind != SGB_KERNEL_GENERAL;
  const bool fused = kind == SGB_KERNEL_FUSED;
  const void* fn = fused      ? fused_kernel(a, blocks)
                   : resident ? (a.bf16 ? (const void*)k_persistent_resident<true>
                                        : (const void*)k_persistent_resident<false>)
                   : general_one_barrier(a)
                       ? (a.n_plast == 0 && a.lane_cells == 2u
                              ? (a.bf16 ? (const void*)k_persistent<true, true, 2>
                                        : (const void*)k_persistent<false, true, 2>)
                              : (a.bf16 ? (const void*)k_persistent<true, true>
                                        : (const void*)k_persistent<false, true>))
                       : (a.bf16 ? (const void*)k_persistent<true, false>
                                 : (const void*)k_persistent<false, false>);
  const size_t smem = fused ? a.row_smem
                     : (a.seg_smem ? seg_smem_bytes(a) : 0) +
                           ((a.n_pull_units && a.pull_sum) ? pull_sum_bytes(a) : 0);
  // Heavy words without the shared memory that the kernel addresses for them.
  if (fused && a.hv_words && a.row_smem < fused_heavy_bytes(a, blocks)) return cudaErrorInvalidValue;
  const uint32_t threads = fused ? fused_threads(a, blocks) : kPersistBlock;
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(threads), params, smem, s);
}

uint32_t fused_row_smem_max() {
  size_t most = ~(size_t)0;
  for (const void* fn : kFusedKernels) most = std::min(most, dyn_smem_max(fn));
  return (uint32_t)most;
}

}  // namespace sgb
