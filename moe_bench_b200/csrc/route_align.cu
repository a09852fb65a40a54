// Routing front end and the sort-and-pad ("moe_align") step.
//
//  * route_topk: softmax over the expert logits, top-k selection, weights
//    renormalised over the selected experts.  One warp per token; the selection
//    is k rounds of a warp arg-max on ordered integer keys (largest logit first,
//    lowest expert index wins ties).  The reference has no router (data.py:178-235 draws the
//    ids directly); this is the front end a caller with logits needs.
//
//  * align: stable counting sort of the flat assignment index n = token*k+kpos
//    by local expert slot, every expert segment padded to pad_rows rows.  It
//    reproduces the slot order of the reference's schedule builder on one rank
//    (tk_scheme.py:98-126, equal to the argsort key of tk_scheme.py:338-342)
//    and replaces the moe_align_block_size step inside fused_experts
//    (baseline.py:67).  Work is cut into contiguous chunks of assignments, one
//    warp each: per-warp histograms (match.any), exclusive scans over warps,
//    blocks and experts, then a scatter that replays the same match.any ranks,
//    so the order inside an expert is ascending n whatever the grid.

#include "align_row.h"
#include "layer.cuh"

namespace mb200 {

namespace {

// ---------------------------------------------------------------- route_topk
constexpr int kRouteMaxExperts = 1024;

// Order-preserving image of a logit in uint32: larger logit <-> larger key, -0 == +0, NaN below
// -inf, and 0 below all of them for what cannot be selected (an earlier winner, a slot past the last
// expert).  Every expert of the row has a key above 0 until it is selected, so topk <= experts rounds
// give topk different experts, whatever the logits are.
constexpr uint32_t kKeyNone = 0u, kKeyNan = 1u;  // logit_key(-inf) = 0x007FFFFF
__device__ __forceinline__ uint32_t logit_key(float v) {
  const uint32_t u = __float_as_uint(v + 0.0f);  // -0 + 0 = +0
  const uint32_t key = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return v != v ? kKeyNan : key;
}
__device__ __forceinline__ float key_logit(uint32_t key) {
  if (key <= kKeyNan) return -INFINITY;  // a NaN logit weighs nothing beside others
  return __uint_as_float((key & 0x80000000u) ? (key ^ 0x80000000u) : ~key);
}

// One warp per token, lane l holds experts l, l+32, ... (coalesced loads) as ordered integer
// keys.  Instruction issue bounds this kernel (the 8 MB of logits are two microseconds of HBM), so
// the k rounds are kept short: each lane caches its own best (key, expert); a round is two warp
// reductions (redux.sync: largest key, then lowest expert among the lanes that hold it) and a
// rescan of kPerLane registers after the winner is retired.  kPerLane is a template parameter so
// that the rescan has exactly as many steps as the expert count needs.  8192 x 256 logits, top-8:
// 12.3 us against 41.0 us with ten shuffles and 32 predicated compares per round.
template <int kPerLane>
__global__ void route_topk_kernel(const float* __restrict__ logits, int tokens, int experts,
                                  int topk, int* __restrict__ ids, float* __restrict__ weights) {
  const int warps_per_block = blockDim.x >> 5;
  const int token = blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (token >= tokens) return;
  const float* row = logits + size_t(token) * experts;

  uint32_t key[kPerLane];
#pragma unroll
  for (int i = 0; i < kPerLane; ++i) {
    const int e = i * 32 + lane;
    key[i] = e < experts ? logit_key(__ldg(row + e)) : kKeyNone;
  }
  uint32_t best;
  int best_e;
  auto rescan = [&]() {  // lowest index first on ties (i ascending, strict >)
    best = kKeyNone;
    best_e = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < kPerLane; ++i)
      if (key[i] > best) { best = key[i]; best_e = i * 32 + lane; }
  };
  rescan();

  float mx = 0.f;      // the first winner's logit
  float sel_sum = 0.f;
  uint32_t my_key = 0;  // lane j keeps the j-th winner of the current 32
  int my_id = 0;
  for (int j = 0; j < topk; ++j) {
    const uint32_t win = __reduce_max_sync(0xffffffffu, best);
    const int win_e = __reduce_min_sync(0xffffffffu, best == win ? best_e : 0x7fffffff);
    if (j == 0) mx = key_logit(win);
    if (lane == (j & 31)) { my_key = win; my_id = win_e; }
    // retire the winner
    if (best_e == win_e) {
#pragma unroll
      for (int i = 0; i < kPerLane; ++i)
        if (i * 32 + lane == win_e) key[i] = kKeyNone;
      rescan();
    }
    if ((j & 31) == 31 || j == topk - 1) {
      // up to 32 selections; beyond 32 the sum is not final yet, so the weights are written
      // unnormalised and scaled below
      const int base = j & ~31;
      const int n = j - base + 1;
      float p = expf(key_logit(my_key) - mx);
      for (int i = 0; i < n; ++i) sel_sum += __shfl_sync(0xffffffffu, p, i);
      if (topk <= 32) p *= 1.0f / sel_sum;
      if (lane < n) {
        ids[size_t(token) * topk + base + lane] = my_id;
        weights[size_t(token) * topk + base + lane] = p;
      }
    }
  }
  if (topk > 32) {
    __syncwarp();
    const float inv = 1.0f / sel_sum;
    for (int j = lane; j < topk; j += 32) weights[size_t(token) * topk + j] *= inv;
  }
}

// ---------------------------------------------------------------- align
// The flat assignments are cut into chunks, one per warp, and the warps into blocks.  At most two
// launches: `align_count_kernel` writes one histogram per block, `align_scatter_kernel` sums the
// histograms of the blocks before its own, scans the experts and places its assignments, every
// block redoing the (small) scans for itself, so no single-block pass sits between the two.  One
// block needs no histogram but its own: up to kOneBlockAssignments a single launch does it all.
// The work is latency, not bandwidth (8192 tokens x top-8: 0.8 MB): chunks are short, so that many
// warps wait at the same time, and everything a block shares stays in shared memory.  16 warps of at
// least 32 assignments, at every size: fewer warps leave more histograms for every block to sum and
// fewer threads to sum them (65536 assignments over 1024 experts: 8 warps 58.9 us, 16 warps 40.7; count,
// one-block scan and scatter as three kernels 42.0), more warps or longer chunks lengthen the walks of
// one block (4096 over 256: 32 warps of 128 in one block 18.8 us, 16 warps of 32 in 8 blocks 8.9).
// Device time of a call, one B200, the three kernels against these two: 512 over 256 experts 10.4 / 10.2
// us, 8192 over 256 27.7 / 9.1, 65536 over 256 25.2 / 14.8, 524288 over 32 25.8 / 17.7.
constexpr int kMaxAlignBlocks = 256;       // one histogram each: scratch is this many ints per expert
constexpr int kAlignWarps = 16;            // per block
constexpr int kMinChunk = 32;              // assignments per warp
// Above a block of shortest chunks, because a second launch costs what it saves: 1024 assignments over 8
// experts 5.7 us in one block, 6.8 in two (over 256 experts 11.8 and 10.3).
constexpr int kOneBlockAssignments = 1024;

struct AlignShape {
  int blocks;
  int64_t chunk;
};
AlignShape align_shape(int64_t assignments) {
  AlignShape s;
  constexpr int64_t kMaxWarps = int64_t(kMaxAlignBlocks) * kAlignWarps;  // of the whole grid
  const int64_t warps = assignments <= kOneBlockAssignments ? kAlignWarps : kMaxWarps;
  const int64_t chunk = ((assignments + warps - 1) / warps + 31) / 32 * 32;
  s.chunk = chunk < kMinChunk ? kMinChunk : chunk;
  const int64_t per_block = s.chunk * kAlignWarps;
  s.blocks = assignments <= per_block ? 1 : int((assignments + per_block - 1) / per_block);
  return s;
}

__device__ __forceinline__ int slot_of(const int* topk_ids, const int* expert_map, int64_t n,
                                       int local_experts) {
  int e = __ldg(topk_ids + n);
  if (expert_map) e = (e >= 0) ? __ldg(expert_map + e) : -1;
  return (e >= 0 && e < local_experts) ? e : -1;
}

// Walk one chunk in order, 32 assignments at a time (the loads of four steps in flight
// together).  Emit(n, slot, before, peers): `peers` are the lanes with the same slot, `before`
// how many of them come first; called by the whole warp, converged (slot -1 and n >= end where a lane
// has no assignment).
template <class Emit>
__device__ __forceinline__ void walk_chunk(const int* topk_ids, const int* expert_map, int64_t begin,
                                           int64_t end, int local_experts, Emit emit) {
  constexpr int kSteps = 4;
  const int lane = threadIdx.x & 31;
  for (int64_t base = begin; base < end; base += 32 * kSteps) {
    int slot[kSteps];
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      const int64_t n = base + 32 * i + lane;
      slot[i] = n < end ? slot_of(topk_ids, expert_map, n, local_experts) : -1;
    }
#pragma unroll
    for (int i = 0; i < kSteps; ++i) {
      if (base + 32 * i >= end) break;
      const int64_t n = base + 32 * i + lane;
      const unsigned peers = __match_any_sync(0xffffffffu, slot[i]);
      emit(n, slot[i], __popc(peers & ((1u << lane) - 1u)), peers);
      __syncwarp();
    }
  }
}

__global__ void align_count_kernel(const int* __restrict__ topk_ids, const int* __restrict__ expert_map,
                                   int64_t assignments, int local_experts, int64_t chunk,
                                   int* __restrict__ block_hist) {
  extern __shared__ int hist[];  // [E]
  pdl_trigger();
  for (int e = threadIdx.x; e < local_experts; e += blockDim.x) hist[e] = 0;
  __syncthreads();
  const int64_t unit = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t begin = unit * chunk < assignments ? unit * chunk : assignments;
  const int64_t end = begin + chunk < assignments ? begin + chunk : assignments;
  walk_chunk(topk_ids, expert_map, begin, end, local_experts, [&](int64_t, int slot, int before, unsigned peers) {
    if (slot >= 0 && before == 0) atomicAdd(hist + slot, __popc(peers));
  });
  __syncthreads();
  for (int e = threadIdx.x; e < local_experts; e += blockDim.x)
    block_hist[size_t(blockIdx.x) * local_experts + e] = hist[e];
}

// Shared memory, ints: per_warp [warps][E] | total [E] | base [E] | prefix [E+1] | part [2][threads]
__global__ void __launch_bounds__(kAlignWarps * 32)
align_scatter_kernel(const int* __restrict__ topk_ids, const int* __restrict__ expert_map, int64_t assignments,
                     int local_experts, int64_t chunk, const int* block_hist,
                     int* __restrict__ counts, int* __restrict__ mtile_prefix, int* __restrict__ sorted_ids,
                     int* __restrict__ inverse, int64_t row_capacity, int pad, int* __restrict__ clear,
                     int64_t clear_ints) {
  extern __shared__ int smem[];
  const int E = local_experts;
  constexpr int warps = kAlignWarps;
  static_assert(kAlignWarps % 8 == 0, "the warps' counters are read eight at a time");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* per_warp = smem;
  int* total = per_warp + warps * E;
  int* base = total + E;
  int* prefix = base + E;
  int* part = prefix + E + 1;
  const int nb = gridDim.x;
  pdl_trigger();

  // counters of the kernels that follow (arrivals per granule / token block)
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < clear_ints; i += int64_t(nb) * blockDim.x)
    clear[i] = 0;

  // 1. this block's assignments per (warp, expert)
  const int64_t unit = int64_t(blockIdx.x) * warps + warp;
  const int64_t begin = unit * chunk < assignments ? unit * chunk : assignments;
  const int64_t end = begin + chunk < assignments ? begin + chunk : assignments;
  int* running = per_warp + warp * E;
  for (int e = lane; e < E; e += 32) running[e] = 0;
  __syncwarp();
  walk_chunk(topk_ids, expert_map, begin, end, E, [&](int64_t, int slot, int before, unsigned peers) {
    if (slot >= 0 && before == 0) running[slot] += __popc(peers);
  });
  pdl_wait();  // the blocks' histograms
  __syncthreads();

  // 2. total[e] over all blocks, base[e] over the blocks before this one.  Thread groups of E
  // threads take every groups-th row of the histogram (or of per_warp when there is one block).
  const int rows = nb > 1 ? nb : warps;
  constexpr int kMaxGroups = 32;
  int groups = E < int(blockDim.x) ? int(blockDim.x) / E : 1;
  if (groups > kMaxGroups) groups = kMaxGroups;
  for (int e0 = 0; e0 < E; e0 += blockDim.x) {
    const int g = groups > 1 ? int(threadIdx.x) / E : 0;
    const int e = e0 + (groups > 1 ? int(threadIdx.x) % E : int(threadIdx.x));
    if (e < E && g < groups) {
      int all = 0, prev = 0;
      for (int r0 = g; r0 < rows; r0 += 8 * groups) {
        int v[8];  // loads first, so eight of them are in flight together
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = r0 + i * groups;
          v[i] = r >= rows ? 0 : nb > 1 ? __ldcg(block_hist + size_t(r) * E + e) : per_warp[r * E + e];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          all += v[i];
          if (nb > 1 && r0 + i * groups < int(blockIdx.x)) prev += v[i];
        }
      }
      if (groups == 1) {
        total[e] = all;
        base[e] = prev;
      } else {
        part[g * E + e] = all;
        part[blockDim.x + g * E + e] = prev;
      }
    }
  }
  __syncthreads();
  if (groups > 1) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
      int all = 0, prev = 0;
      for (int g = 0; g < groups; ++g) {
        all += part[g * E + e];
        prev += part[blockDim.x + g * E + e];
      }
      total[e] = all;
      base[e] = prev;
    }
    __syncthreads();
  }

  // 3. cumulative row blocks per expert: each lane of warp 0 owns a run of experts
  if (warp == 0) {
    const int per = (E + 31) / 32;
    const int lo = lane * per < E ? lane * per : E;
    const int hi = lo + per < E ? lo + per : E;
    int sum = 0;
    for (int e = lo; e < hi; ++e) sum += (total[e] + pad - 1) / pad;
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    int run = incl - sum;
    for (int e = lo; e < hi; ++e) {
      prefix[e] = run;
      run += (total[e] + pad - 1) / pad;
    }
    if (lane == 31) prefix[E] = incl;
  }
  __syncthreads();

  // 4. assignments of the expert ahead of every (warp, expert): blocks before + warps before
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int run = base[e];
    for (int w0 = 0; w0 < warps; w0 += 8) {
      int v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = per_warp[(w0 + i) * E + e];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        per_warp[(w0 + i) * E + e] = run;
        run += v[i];
      }
    }
  }
  if (blockIdx.x == 0) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) counts[e] = total[e];
    for (int e = threadIdx.x; e <= E; e += blockDim.x) mtile_prefix[e] = prefix[e];
  }
  __syncthreads();

  // 5. place this warp's assignments; the experts' padding rows are shared out over all warps
  walk_chunk(topk_ids, expert_map, begin, end, E, [&](int64_t n, int slot, int before, unsigned peers) {
    const int seen = slot >= 0 ? running[slot] : 0;
    // All lanes have read their counters.  One barrier for the warp: with one per group of peers the
    // groups, up to 32, run one after the other (4096 assignments over 256 experts in one block: 23.0
    // against 18.8 us).
    __syncwarp();
    if (slot >= 0) {
      const int64_t row = sorted_row(prefix[slot], pad, seen + before);
      if (row < row_capacity) sorted_ids[row] = int(n);
      inverse[n] = int(row);
      if (before == 0) running[slot] = seen + __popc(peers);
    } else if (n < end) {
      inverse[n] = -1;
    }
  });
  for (int e = blockIdx.x * warps + warp; e < E; e += nb * warps) {
    int64_t stop = sorted_row(prefix[e + 1], pad, 0);
    if (stop > row_capacity) stop = row_capacity;
    for (int64_t p = sorted_row(prefix[e], pad, total[e]) + lane; p < stop; p += 32) sorted_ids[p] = -1;
  }
}

}  // namespace

int launch_route_topk(const float* logits, int tokens, int experts, int topk, int* ids,
                      float* weights, cudaStream_t stream) {
  MB200_REQUIRE(experts >= 1 && experts <= kRouteMaxExperts, kUnsupportedShape,
                "route_topk: %d experts, supported 1..%d", experts, kRouteMaxExperts);
  MB200_REQUIRE(topk >= 1 && topk <= experts, kInvalidArgument, "route_topk: topk=%d with %d experts",
                topk, experts);
  if (tokens == 0) return kOk;
  const int warps = 4;
  const int blocks = (tokens + warps - 1) / warps;
  const int per_lane = (experts + 31) / 32;
  auto launch = [&](auto kernel) {
    kernel<<<blocks, warps * 32, 0, stream>>>(logits, tokens, experts, topk, ids, weights);
  };
  if (per_lane <= 1) launch(route_topk_kernel<1>);
  else if (per_lane <= 2) launch(route_topk_kernel<2>);
  else if (per_lane <= 4) launch(route_topk_kernel<4>);
  else if (per_lane <= 8) launch(route_topk_kernel<8>);
  else if (per_lane <= 16) launch(route_topk_kernel<16>);
  else launch(route_topk_kernel<32>);
  MB200_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

int64_t align_scratch_ints(int64_t assignments, int experts) {
  (void)assignments;
  return int64_t(kMaxAlignBlocks) * experts;
}

int launch_align(const int* topk_ids, int64_t assignments, const int* expert_map, int local_experts,
                 Schedule sched, int64_t row_capacity, int* scratch, cudaStream_t stream) {
  MB200_REQUIRE(local_experts >= 1 && local_experts <= kMaxExperts, kUnsupportedShape,
                "align: %d local experts, supported 1..%d", local_experts, kMaxExperts);
  MB200_REQUIRE(assignments >= 0 && assignments < (int64_t(1) << 31) - 4096, kUnsupportedShape,
                "align: %lld assignments do not fit 32-bit row indices", (long long)assignments);
  const int pad = sched.pad_rows;
  MB200_REQUIRE(pad >= 1 && pad <= 1024, kInvalidArgument, "align: pad_rows=%d (1..1024)", pad);
  const AlignShape sh = align_shape(assignments);
  constexpr int threads = kAlignWarps * 32;
  if (sh.blocks > 1) {
    align_count_kernel<<<sh.blocks, threads, size_t(local_experts) * sizeof(int), stream>>>(
        topk_ids, expert_map, assignments, local_experts, sh.chunk, scratch);
    MB200_CHECK_CUDA(cudaGetLastError());
  }
  auto smem_bytes = [](int experts) { return size_t(kAlignWarps * experts + 3 * experts + 1 + 2 * threads) * sizeof(int); };
  const size_t smem = smem_bytes(local_experts);
  if (smem > 48 * 1024)  // more than 592 experts
    MB200_CHECK_CUDA(cudaFuncSetAttribute(align_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          int(smem_bytes(kMaxExperts))));
  // The first kernel of the sort is an ordinary launch: what came before it on the stream is
  // complete, so the second may overlap the first up to the histograms.
  if (sh.blocks > 1)
    return launch_chained(align_scatter_kernel, dim3(sh.blocks), threads, smem, stream, false, sched.chained, topk_ids, expert_map,
                          assignments, local_experts, sh.chunk, scratch, sched.counts, sched.mtile_prefix,
                          sched.sorted_ids, sched.inverse, row_capacity, pad, sched.clear, sched.clear_ints);
  align_scatter_kernel<<<1, threads, smem, stream>>>(
      topk_ids, expert_map, assignments, local_experts, sh.chunk, scratch, sched.counts, sched.mtile_prefix,
      sched.sorted_ids, sched.inverse, row_capacity, pad, sched.clear, sched.clear_ints);
  MB200_CHECK_CUDA(cudaGetLastError());
  return kOk;
}

}  // namespace mb200

// ---------------------------------------------------------------------------
// Sort-and-pad without caller-provided scratch.
//
// Some hosts of this library must not allocate device memory once they are
// running: an inference server that handed (nearly) all HBM to its own pool at
// start-up has nothing left for a later cudaMalloc, and inside a latency-
// critical decode loop cudaMalloc/cudaFree would stall the whole device.  For
// them the blocks' histograms of the sort live in the fixed array below instead of
// a buffer the caller allocates.  The price: 256 KiB of every GPU that loads the
// library is held until the process exits, the problem size is capped, and all
// calls on a device share the one array.
// ---------------------------------------------------------------------------
#include <mutex>

#include "../../include/moe_bench_b200.h"

namespace mb200 {
namespace {

constexpr int kNoAllocMaxExperts = MB200_NOALLOC_MAX_LOCAL_EXPERTS;          // 256
constexpr int64_t kNoAllocMaxAssignments = MB200_NOALLOC_MAX_ASSIGNMENTS;    // 2^20
// blocks (<= 256) x experts (<= 256) histogram entries = 256 KiB
static __device__ __align__(256) int g_noalloc_align_scratch[kMaxAlignBlocks * kNoAllocMaxExperts];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
int* g_noalloc_scratch_ptr[kNoAllocMaxDevices] = {};

// Device address of the array on the CURRENT device, looked up once per device.
// In host code the array's name is only a handle for the runtime, never an
// address a kernel may use, hence cudaGetSymbolAddress.
int noalloc_scratch(int** out) {
  int dev = -1;
  MB200_CHECK_CUDA(cudaGetDevice(&dev));
  MB200_REQUIRE(dev >= 0 && dev < kNoAllocMaxDevices, kUnsupportedShape,
                "align_noalloc: device index %d, supported 0..%d", dev, kNoAllocMaxDevices - 1);
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_scratch_ptr[dev]) {
    void* p = nullptr;
    MB200_CHECK_CUDA(cudaGetSymbolAddress(&p, g_noalloc_align_scratch));
    g_noalloc_scratch_ptr[dev] = static_cast<int*>(p);
  }
  *out = g_noalloc_scratch_ptr[dev];
  return kOk;
}

}  // namespace
}  // namespace mb200

extern "C" int mb200_align_noalloc(const int32_t* topk_ids, int64_t tokens, int topk,
                                   const int32_t* expert_map, int local_experts, int32_t* counts,
                                   int32_t* mtile_prefix, int32_t* sorted_ids, int32_t* inverse,
                                   int64_t row_capacity, int pad_rows, void* stream) {
  using namespace mb200;
  MB200_REQUIRE(pad_rows >= 1 && pad_rows <= 1024, kInvalidArgument, "align_noalloc: pad_rows=%d", pad_rows);
  MB200_REQUIRE(tokens >= 0 && topk >= 1, kInvalidArgument, "align_noalloc: tokens=%lld topk=%d",
                (long long)tokens, topk);
  MB200_REQUIRE(local_experts >= 1 && local_experts <= kNoAllocMaxExperts, kUnsupportedShape,
                "align_noalloc: %d local experts exceed the built-in scratch (at most %d); "
                "use mb200_align with a caller-provided scratch buffer",
                local_experts, kNoAllocMaxExperts);
  // compared before multiplying: tokens * topk must not wrap around on its way to the limit check
  const int64_t assignments = tokens <= kNoAllocMaxAssignments / topk ? tokens * topk : kNoAllocMaxAssignments + 1;
  MB200_REQUIRE(assignments <= kNoAllocMaxAssignments, kUnsupportedShape,
                "align_noalloc: %lld assignments exceed the built-in scratch (at most %lld); "
                "use mb200_align with a caller-provided scratch buffer",
                (long long)assignments, (long long)kNoAllocMaxAssignments);
  MB200_REQUIRE(counts && mtile_prefix && sorted_ids && (tokens == 0 || (topk_ids && inverse)),
                kInvalidArgument, "align_noalloc: null pointer");
  const int64_t touched = assignments < local_experts ? assignments : local_experts;
  const int64_t need = (assignments + touched * (pad_rows - 1) + pad_rows - 1) / pad_rows * pad_rows;
  MB200_REQUIRE(row_capacity >= need, kWorkspaceTooSmall, "align_noalloc: row capacity %lld < %lld",
                (long long)row_capacity, (long long)need);
  int* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  // Every histogram entry a launch reads is written earlier by the same launch
  // sequence, so nothing left over from the previous call has to be cleared.
  Schedule s{counts, mtile_prefix, sorted_ids, inverse, pad_rows};
  return launch_align(topk_ids, assignments, expert_map, local_experts, s, row_capacity, scratch,
                      reinterpret_cast<cudaStream_t>(stream));
}
