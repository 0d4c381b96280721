// Standalone delivery operator on caller-owned device buffers.
//
// The reference exposes its propagation as free-standing kernels called once
// per projection and step (spike_propagation, spike_propagation_mThreads,
// spike_propagation_PR; Simulation_header.cu:83-303).  sgb_deliver_spikes is
// the same operation for callers that run their own neuron update: given one
// step's spike flags it adds every synapse of every spiking cell into the
// fixed-point delay ring, event-driven, in one kernel without scratch memory.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/scaffold_gb300.h"
#include "sgb_device.h"
#include "sgb_model.h"

namespace sgb {
namespace {

constexpr unsigned kFullMask = 0xffffffffu;

// One step's delivery in one launch.  A block takes kBlock x V cells, in groups
// of 8 (V = 1) or 16 dealt round-robin over the blocks, so that neighbours with
// long rows that spike together (a population of Golgi cells) fall to different
// blocks, and few cells to many blocks.  It collects the spiking ones (first
// synapse and row length) in shared memory, cuts their rows into items of kOpsItem synapses (a running item
// count per cell), and its warps take the items in turn, finding an item's
// cell by bisection of the counts; four loads per lane are in flight before an
// item's reductions.  No scratch, no list in global memory, and a long row
// (a Golgi cell's 1,200 synapses, a mossy fibre's thousands) spreads over the
// block's warps instead of staying with one.
//
// What bounds it is latency, not bytes: spike flag, row bounds, synapses are
// three dependent reads, then the reductions.  V = 1 spreads the few spikes of
// a step over as many blocks as possible; V = 4 (one 32-bit load per thread)
// above kOpsWide cells, where 256-cell blocks are no longer resident together
// and most of them would only find silent cells (900,000 cells, 0.5 % spiking:
// 6.0 us with V = 1, 4.3 us with V = 4; 320,000: 3.4 and 3.6 us).  The line is
// a constant, GB300's 152 SMs with 8 blocks each: asking the device for its SM
// count costs 35 ns of the host's 2.6 us per call.
//
// Per call on the device, 29.5 synapses a cell: 92,550 cells with 0.5 % spiking
// 10.3 -> 2.7 us, with 5 % 13.9 -> 4.3 us; 9,000 cells 7.8 -> 2.3 us; 900,000
// cells 15.0 -> 4.2 us (5 %: 56.6 -> 14.9 us).  Before: clear, compaction into
// a list from the stream-ordered pool, one warp per spiking cell; after a
// synchronisation the pool's allocation made a call 220 us.  Neighbouring long
// rows spiking together, 250 with 1,600 synapses among 92,550 cells: 24 us before,
// 345 with consecutive cells in a block, 15 dealt in groups; 500 of 1,000 cells
// with 2,000: 40, 233, 28 us.  Single cells dealt out would cost the usual call
// 10 % (92,550 cells 3.1 us); groups of 16 cost 900,000 cells 7 %.
constexpr uint32_t kOpsItem = 128;
constexpr uint32_t kOpsWide = 152u * 8u * kBlock;  // cells of one resident wave of V = 1 blocks
constexpr uint32_t kOpsBlocks = 2u * 152u;          // blocks at least, with a group of cells each
constexpr uint32_t ops_group(int v) { return v == 1 ? 8u : 4u; }  // threads with neighbouring cells

template <bool BF16, int V>
__global__ void __launch_bounds__(kBlock) k_ops_deliver(const uint8_t* __restrict__ spikes,
                                                        const uint32_t* __restrict__ row,
                                                        const uint32_t* __restrict__ syn,
                                                        const void* __restrict__ w, int* ring,
                                                        uint32_t n, uint32_t slots,
                                                        uint32_t slot0) {
  // Ring slot of each delay field value d = 0..15: (step + d) % slots, exact
  // for every delay the 4-bit field can hold, whatever the ring's size.
  __shared__ uint32_t s_slot[16];
  __shared__ uint32_t s_n;
  __shared__ uint2 s_row[kBlock * V];      // {first synapse, length} of the spiking cells
  __shared__ uint32_t s_cum[kBlock * V];   // items up to and including each of them
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  if (tid == 0) s_n = 0;
  if (tid < 16) s_slot[tid] = (slot0 + tid) % slots;
  constexpr uint32_t G = ops_group(V);
  const uint32_t j0 = ((tid / G * gridDim.x + blockIdx.x) * G + tid % G) * V;
  uint32_t act = 0;  // bit v: cell j0 + v spiked
  if (V == 4 && j0 + 4u <= n && ((uintptr_t)spikes & 3u) == 0u) {
    const uint32_t f = __ldg(reinterpret_cast<const uint32_t*>(spikes + j0));
#pragma unroll
    for (int v = 0; v < V; ++v) act |= (((f >> (8 * v)) & 0xFFu) ? 1u : 0u) << v;
  } else {
#pragma unroll
    for (int v = 0; v < V; ++v)
      if (j0 + v < n && __ldg(spikes + j0 + v)) act |= 1u << v;
  }
  if (!__syncthreads_or((int)act)) return;
  if (act) {
    uint32_t at = atomicAdd(&s_n, (uint32_t)__popc(act));
#pragma unroll
    for (int v = 0; v < V; ++v)
      if ((act >> v) & 1u) {
        const uint32_t r0 = __ldg(row + j0 + v), r1 = __ldg(row + j0 + v + 1);
        s_row[at++] = make_uint2(r0, r1 > r0 ? r1 - r0 : 0u);
      }
  }
  __syncthreads();
  const uint32_t n_act = s_n;
  if (tid < 32) {
    uint32_t run = 0;
    for (uint32_t b = 0; b < n_act; b += 32) {
      const uint32_t len = b + lane < n_act ? s_row[b + lane].y : 0u;
      uint32_t incl = len / kOpsItem + (len % kOpsItem ? 1u : 0u);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= (uint32_t)o) incl += x;
      }
      if (b + lane < n_act) s_cum[b + lane] = run + incl;
      run += __shfl_sync(kFullMask, incl, 31);
    }
  }
  __syncthreads();
  const uint32_t total = s_cum[n_act - 1u];
  for (uint32_t it = tid >> 5; it < total; it += kBlock / 32) {
    uint32_t lo = 0, hi = n_act - 1u;  // first cell whose items reach past `it`
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (s_cum[mid] > it) hi = mid; else lo = mid + 1u;
    }
    const uint2 r = s_row[lo];
    const uint32_t o0 = (it - (lo ? s_cum[lo - 1u] : 0u)) * kOpsItem;
    const uint32_t q0 = r.x + o0, len = min(kOpsItem, r.y - o0);
    uint32_t wd[kOpsItem / 32];
    float wv[kOpsItem / 32];
#pragma unroll
    for (uint32_t k = 0; k < kOpsItem / 32; ++k) {
      const uint32_t q = 32u * k + lane;
      if (q >= len) continue;
      wd[k] = __ldg(syn + q0 + q);
      wv[k] = BF16 ? __uint_as_float(((uint32_t)__ldg((const unsigned short*)w + q0 + q)) << 16)
                   : __ldg((const float*)w + q0 + q);
    }
#pragma unroll
    for (uint32_t k = 0; k < kOpsItem / 32; ++k) {
      if (32u * k + lane >= len) break;
      const uint32_t slot = s_slot[(wd[k] >> kPushPostBits) & 15u];
      atomicAdd(ring + (((size_t)slot * n + (wd[k] & kPushPostMask)) << 1) + (wd[k] >> 31),
                __float2int_rn(wv[k]));
    }
  }
}

}  // namespace

int deliver_check(int32_t n_cells, int32_t weight_type, int32_t ring_slots, int64_t step,
                  const void* spikes, const void* row, const void* syn, const void* w,
                  const void* ring) {
  if (n_cells < 0 || (uint32_t)n_cells > kPushPostMask)
    return set_error(SGB_ERR_ARG, "n_cells %d not in 0..2^27-1", n_cells);
  if (weight_type != SGB_WEIGHT_FP32 && weight_type != SGB_WEIGHT_BF16)
    return set_error(SGB_ERR_ARG, "unknown weight type %d", weight_type);
  if (ring_slots < 2 || ring_slots > kMaxDelay + 1)
    return set_error(SGB_ERR_ARG, "ring_slots %d not in 2..%d", ring_slots, kMaxDelay + 1);
  if (step < 0) return set_error(SGB_ERR_ARG, "step is negative");
  if (n_cells && (!spikes || !row || !syn || !w || !ring))
    return set_error(SGB_ERR_ARG, "NULL device buffer");
  return SGB_OK;
}

// Blocks of the delivery kernel for n cells: V cells per thread.
cudaError_t deliver_enqueue(const uint8_t* spikes, int32_t n_cells, const uint32_t* row,
                            const uint32_t* syn, const void* w, int32_t weight_type, int32_t* ring,
                            int32_t ring_slots, int64_t step, cudaStream_t st) {
  if (!n_cells) return cudaSuccess;
  const uint32_t n = (uint32_t)n_cells, slots = (uint32_t)ring_slots;
  const uint32_t slot0 = (uint32_t)(step % ring_slots);
  const bool bf16 = weight_type == SGB_WEIGHT_BF16, wide = n > kOpsWide;
  const uint32_t per = kBlock * (wide ? 4u : 1u), grp = wide ? 4u * ops_group(4) : ops_group(1);
  const uint32_t blocks = std::max((n + per - 1) / per, std::min((n + grp - 1) / grp, kOpsBlocks));
  auto* fn = wide ? (bf16 ? k_ops_deliver<true, 4> : k_ops_deliver<false, 4>)
                  : (bf16 ? k_ops_deliver<true, 1> : k_ops_deliver<false, 1>);
  fn<<<blocks, kBlock, 0, st>>>(spikes, row, syn, w, ring, n, slots, slot0);
  return cudaGetLastError();
}

}  // namespace sgb

using namespace sgb;

extern "C" int sgb_deliver_spikes(const uint8_t* spikes, int32_t n_cells, const uint32_t* row,
                                  const uint32_t* syn, const void* weights, int32_t weight_type,
                                  int32_t* ring, int32_t ring_slots, int64_t step, void* stream) {
  const int rc =
      deliver_check(n_cells, weight_type, ring_slots, step, spikes, row, syn, weights, ring);
  if (rc) return rc;
  const cudaError_t e = deliver_enqueue(spikes, n_cells, row, syn, weights, weight_type, ring,
                                        ring_slots, step, (cudaStream_t)stream);
  if (e) return set_error(SGB_ERR_CUDA, "delivery launch failed: %s", cudaGetErrorString(e));
  return SGB_OK;
}

// The entry point for callers that cannot allocate at delivery time.  Both
// entry points run the one kernel above, which allocates nothing; this one
// keeps its stated limit on n_cells.
static constexpr uint32_t kStaticMaxCells = 1u << 20;  // 1,048,576 cells

extern "C" int sgb_deliver_spikes_static(const uint8_t* spikes, int32_t n_cells,
                                         const uint32_t* row, const uint32_t* syn,
                                         const void* weights, int32_t weight_type, int32_t* ring,
                                         int32_t ring_slots, int64_t step, void* stream) {
  if (n_cells > 0 && (uint32_t)n_cells > kStaticMaxCells)
    return set_error(SGB_ERR_RANGE,
                     "n_cells %d exceeds this entry point's limit of %u cells (a former static scratch)", n_cells,
                     kStaticMaxCells);
  return sgb_deliver_spikes(spikes, n_cells, row, syn, weights, weight_type, ring, ring_slots, step,
                            stream);
}
