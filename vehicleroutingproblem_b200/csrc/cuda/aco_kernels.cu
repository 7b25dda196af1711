// aco_kernels.cu -- sm_100a kernels of the ACO-for-CVRP hot path.
//
//   k_knn_levels      candidate lists + eta levels + fallback lists, warp per node
//                     (reference: kernel_build_candidate_lists,
//                      src/cuda/aco_cuda_kernels.cu:164-214)
//   k_weights         per-epoch integer weights from the quantized pheromone
//                     (role of seq_shared_update_scores,
//                      src/seq/aco_sequential.c:410-442)
//   k_construct       warp-per-ant route construction with the sequential
//                     path's rules (src/seq/aco_sequential.c:477-681) over
//                     candidate tables staged in shared memory by the TMA
//                     engine (reference kernel: aco_cuda_kernels.cu:447-562)
//   k_best_cluster    iteration best, global best, stop rules and both
//                     deposits of the pipelined epoch over a cluster of 8
//                     blocks (src/cuda/aco_cuda.cu:83-126, :331-399)
//   k_evap_deposit    128-bit streaming evaporation, then the deposit of two
//                     given solutions by the last block
//                     (aco_cuda_kernels.cu:145-155, :569-668)
#include "aco_internal.cuh"

#include <cooperative_groups.h>

#include <cfloat>
#include <climits>

namespace acob200 {

// ===========================================================================
// Candidate lists and eta levels
// ===========================================================================

__device__ __forceinline__ int level_of(float d2, const float *thr, int J) {
  int lo = 0, hi = J;  // number of thresholds <= d2
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (__ldg(thr + mid) <= d2) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Candidate list and levels of one node by one warp and, given their rows, the
// fallback's lists: the 64 neighbours after its k candidates (ranks k+1 ..
// k+64) and the kTier2Len after those, each 32 keys after the last list's
// last, in the candidates' order (ascending d^2 bits, then node).  0 marks an
// empty slot; an empty last slot means the lists hold every other customer.
constexpr int kKnnThreads = 256;
constexpr int kKnnPool = 448;  // keys collected for the second tier, per warp

__device__ __forceinline__ void knn_rows(const float2 *coords, int n, int k, int i,
                                         const float *thr, int J, uint16_t *cand, uint16_t *lvl,
                                         uint16_t *tier, uint16_t *tier2,
                                         unsigned long long *buf, unsigned long long *pool,
                                         int lane) {
  const unsigned long long kNone = ~0ull;
  unsigned long long key = warp_knn(coords, n, k, i, lane, buf);
  if (lane < k) {
    const int node = (key == kNone) ? 0 : (int)(key & 0xffffffffu);
    const float d2 = __uint_as_float((unsigned)(key >> 32));
    cand[lane] = (uint16_t)node;
    lvl[lane] = (uint16_t)(node ? level_of(d2, thr, J) : 0);
  }
  if (!tier) return;
  unsigned long long last = __shfl_sync(kFull, key, k - 1);
  constexpr int kRanks = kTierLen + kTier2Len;
  const int parts = tier2 ? kRanks / 32 : kTierLen / 32;
  // Eight more lists: the keys that can be on them are collected first, below
  // a bound on the squared distance scaled up from that of the last rank
  // listed (the count grows with the area) until it leaves enough but not too
  // many; the lists are then taken from those instead of from every node
  // (n=16000: 3.3 -> 1.0 ms for all nodes).  A bound that brings no key more
  // than the one before has the edge of a clump behind it; collecting starts
  // again once a list has come past that bound (set-up of n=16000 in clumps of
  // 100 5.2 ms with every list from every node, 5.7 with six passes in vain
  // before, now 2.9).
  const float2 pi = coords[i];
  int held = 0, starts = 0;
  bool collected = false;
  float few = -1.f;  // this bound leaves too few
  auto collect = [&](float d2, int need, int listed) {
    float bound = d2 * (1.3f * (float)(need + listed) / (float)listed);
    int before = -1;
#pragma unroll 1
    for (int tries = 0; tries < 6; ++tries) {
      const unsigned long long top =
          ((unsigned long long)__float_as_uint(bound) << 32) | 0xffffffffull;
      // Keys of one distance come in the order of the nodes: the first ones
      // are enough (customers at the row's own place).
      const int enough = bound == 0.f ? need - 1 : kKnnPool;
      held = 0;
#pragma unroll 1
      for (int g = 0; 32 * g < n && held <= enough; g += 4) {
        unsigned long long x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = node_key(coords, n, i, pi, 1 + 32 * (g + u) + lane);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool in = x[u] > last && x[u] <= top && x[u] != kNone;
          const unsigned m = __ballot_sync(kFull, in);
          const int at = held + __popc(m & ((1u << lane) - 1u));
          if (in && at < kKnnPool) pool[at] = x[u];
          held += __popc(m);
        }
      }
      if (held >= need && held <= kKnnPool) return true;
      if (held < need) few = bound;
      if (held < need && (held == before || bound == 0.f)) return false;
      before = held;
      bound *= held > kKnnPool ? 0.7f : 1.2f * (float)(need + 32) / (float)(held + 32);
    }
    few = FLT_MAX;
    return false;
  };
#pragma unroll 1
  for (int r = 0; r < parts; ++r) {
    if (tier2 && !collected && last != kNone && starts < 3) {
      const float d2 = __uint_as_float((unsigned)(last >> 32));
      if (d2 > few) {
        ++starts;
        collected = collect(d2, kRanks - 32 * r, k + 32 * r);
        __syncwarp();
      }
    }
    if (last == kNone) {
      key = kNone;
    } else if (collected) {
      key = warp_smallest(
          [&](int g) {
            const int at = 32 * g + lane;
            const unsigned long long x = at < held ? pool[at] : kNone;
            return x <= last ? kNone : x;
          },
          (held + 31) / 32, 32, lane, buf);
    } else {
      key = warp_knn(coords, n, 32, i, lane, buf, last);
    }
    const uint16_t node = (uint16_t)(key == kNone ? 0u : (unsigned)(key & 0xffffffffu));
    if (r < kTierLen / 32) tier[32 * r + lane] = node;
    else tier2[32 * (r - kTierLen / 32) + lane] = node;
    last = __shfl_sync(kFull, key, 31);
  }
  __syncwarp();
}

__global__ void __launch_bounds__(kKnnThreads) k_knn_levels(
    const float2 *__restrict__ coords, int n, int k,
    const float *__restrict__ thr, int J, uint16_t *__restrict__ cand,
    uint16_t *__restrict__ lvl, uint16_t *__restrict__ tier, uint16_t *__restrict__ tier2) {
  __shared__ unsigned long long s_buf[kKnnThreads / 32][64];
  extern __shared__ unsigned long long s_pool[];  // [warps][kKnnPool] with tier2
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int i = blockIdx.x * (blockDim.x >> 5) + warp; i <= n; i += warps)
    knn_rows(coords, n, k, i, thr, J, cand + (size_t)i * k, lvl + (size_t)i * k,
             tier ? tier + (size_t)i * kTierLen : nullptr,
             tier2 ? tier2 + (size_t)i * kTier2Len : nullptr, s_buf[warp],
             s_pool + warp * kKnnPool, lane);
}

cudaError_t launch_knn_levels(const float2 *coords, int n, int k,
                              const float *thr, int J, uint16_t *cand,
                              uint16_t *lvl, uint16_t *tier, uint16_t *tier2, cudaStream_t s) {
  if (k < 1 || k > kMaxCand) return cudaErrorInvalidValue;
  int rows = n + 1;
  int blocks = (rows + 7) / 8;
  if (blocks > 148 * 16) blocks = 148 * 16;
  const size_t pool = tier2 ? sizeof(unsigned long long) * kKnnPool * (kKnnThreads / 32) : 0;
  k_knn_levels<<<blocks, kKnnThreads, pool, s>>>(coords, n, k, thr, J, cand, lvl, tier, tier2);
  return cudaGetLastError();
}

// Lists of many instances in one launch.  Instance s owns rows [seg_off[s],
// seg_off[s] + seg_n[s] + 1) of the concatenated coordinates (seg_off
// ascending); each warp finds its row's instance by binary search and writes
// the same lists as k_knn_levels on that instance alone.
__global__ void __launch_bounds__(kKnnThreads) k_knn_levels_multi(
    const float2 *__restrict__ coords, const long long *__restrict__ seg_off,
    const int *__restrict__ seg_n, int count, long long rows, int k,
    const float *__restrict__ thr, int J, uint16_t *__restrict__ cand,
    uint16_t *__restrict__ lvl, uint16_t *__restrict__ tier) {
  __shared__ unsigned long long s_buf[kKnnThreads / 32][64];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = (long long)blockIdx.x * (blockDim.x >> 5) + warp; r < rows; r += warps) {
    int lo = 0, hi = count;  // last s with seg_off[s] <= r
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__ldg(seg_off + mid) <= r) lo = mid; else hi = mid;
    }
    const long long off = __ldg(seg_off + lo);
    const int n = __ldg(seg_n + lo);
    const int i = (int)(r - off);
    if (i > n) continue;  // gap rows (none when the segments are packed)
    knn_rows(coords + off, n, k, i, thr, J, cand + (size_t)r * k, lvl + (size_t)r * k,
             tier ? tier + (size_t)r * kTierLen : nullptr, nullptr, s_buf[warp], nullptr, lane);
  }
}

cudaError_t launch_knn_levels_multi(const float2 *coords, const long long *seg_off,
                                    const int *seg_n, int count, long long rows, int k,
                                    const float *thr, int J, uint16_t *cand, uint16_t *lvl,
                                    uint16_t *tier, cudaStream_t s) {
  if (count < 1 || rows < 1 || k < 1 || k > kMaxCand) return cudaErrorInvalidValue;
  long long blocks = (rows + 7) / 8;
  if (blocks > 148 * 16) blocks = 148 * 16;
  k_knn_levels_multi<<<(int)blocks, kKnnThreads, 0, s>>>(coords, seg_off, seg_n, count, rows, k,
                                                         thr, J, cand, lvl, tier);
  return cudaGetLastError();
}

// eta level of d(i,0)^2 for every node (reference-CUDA depot rule).
__global__ void k_depot_levels(const float2 *__restrict__ coords, int n,
                               const float *__restrict__ thr, int J, uint16_t *lvl0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n) return;
  lvl0[i] = (uint16_t)level_of(dist2f(coords[i], coords[0]), thr, J);
}

cudaError_t launch_depot_levels(const float2 *coords, int n, const float *thr, int J,
                                uint16_t *lvl0, cudaStream_t s) {
  k_depot_levels<<<(n + 1 + 255) / 256, 256, 0, s>>>(coords, n, thr, J, lvl0);
  return cudaGetLastError();
}

// ===========================================================================
// Byte fill (pheromone initialisation, kernel_init_tau :131-136)
// ===========================================================================

__global__ void k_fill_u8(uint8_t *p, unsigned long long count, uint8_t v) {
  const unsigned long long nvec = count / 16;
  const uint32_t w = 0x01010101u * v;
  const uint4 vv = make_uint4(w, w, w, w);
  uint4 *p4 = reinterpret_cast<uint4 *>(p);
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
       i < nvec; i += stride)
    p4[i] = vv;
  if (blockIdx.x == 0) {
    for (unsigned long long i = nvec * 16 + threadIdx.x; i < count; i += blockDim.x) p[i] = v;
  }
}

cudaError_t launch_fill_u8(uint8_t *p, unsigned long long count, uint8_t v,
                           cudaStream_t s) {
  unsigned long long nvec = count / 16;
  unsigned long long blocks = (nvec + 255) / 256;
  if (blocks < 1) blocks = 1;
  if (blocks > 148 * 8) blocks = 148 * 8;
  k_fill_u8<<<(unsigned)blocks, 256, 0, s>>>(p, count, v);
  return cudaGetLastError();
}

// ===========================================================================
// Per-epoch weights
// ===========================================================================

// Weights of every row, a warp per row.  Bound by the round trips to L2 (row
// and state, then pheromone cells); the level and weight tables are in shared
// memory, fetched before this launch waits for the previous epoch.
// (Evaporating a small matrix in further blocks of this launch, which leaves
// the side stream out, measured the same: n=24 14.9 -> 14.7 us per epoch,
// n=250 64.1 -> 64.7; so did evaporation, deposits and the next weights in
// one launch: n=24 15.1 -> 15.3, n=1000 214 -> 227.)
constexpr int kWeightThreads = 256;

__global__ void __launch_bounds__(kWeightThreads) k_weights(InstanceView iv, PheromoneView pv,
                                                            EpochTables et, DevState *st) {
  __shared__ int32_t s_A[256];
  __shared__ uint32_t s_lut[256];
  const int lane = threadIdx.x & 31;
  const int k = iv.k;
  const size_t stride = (size_t)iv.n + 1;
  let_next_start();
  s_A[threadIdx.x] = __ldg(et.A + threadIdx.x);
  s_lut[threadIdx.x] = __ldg(et.lut + threadIdx.x);
  wait_for_previous();
  // This warp's first row's candidates and levels, the buffer selector and
  // the stop flag are all requested before any of them is used, so that
  // their round trips overlap.
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int i0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int c = 0, lv = 0;
  if (i0 <= iv.n && lane < k) {
    c = iv.cand[(size_t)i0 * k + lane];
    lv = iv.lvl[(size_t)i0 * k + lane];
  }
  const uint8_t *tau = cur_tau(pv.tau, et.tau_alt, st);
  if (st) {
    int stop = *(volatile int *)&st->stop_flags;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->skip = stop ? 1 : 0;
      if (!stop && st->start_ns == 0ull) st->start_ns = global_timer_ns();
    }
    if (stop) return;
  }
  __syncthreads();
  for (int i = i0; i <= iv.n; i += warps) {
    if (i != i0 && lane < k) {
      c = iv.cand[(size_t)i * k + lane];
      lv = iv.lvl[(size_t)i * k + lane];
    }
    const int q = c > 0 ? (int)tau[(size_t)i * stride + c] : 0;
    const int e = c > 0 ? s_A[q] - lv : INT_MIN;
    const int emax = __reduce_max_sync(kFull, e);
    if (et.rdep && lane == 0)
      et.rdep[i] = (emax == INT_MIN) ? 0 : emax - (et.e_dep - (int)et.lvl0[i]);
    if (lane < k) {
      uint32_t w = 0u;
      uint8_t rel = (uint8_t)kRelMax;
      if (c > 0) {
        int r = emax - e;
        if (r > kRelMax) r = kRelMax;
        rel = (uint8_t)r;
        w = s_lut[r];
      }
      et.w[(size_t)i * k + lane] = w;
      et.rel[(size_t)i * k + lane] = rel;
    }
  }
}

cudaError_t launch_weights(const InstanceView &iv, const PheromoneView &pv,
                           const EpochTables &et, DevState *st,
                           cudaStream_t s) {
  int rows = iv.n + 1;
  int blocks = (rows + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  return launch_after(k_weights, blocks, kWeightThreads, 0, s, iv, pv, et, st);
}

// ===========================================================================
// Construction
// ===========================================================================

// Draws of one ant come 128 at a time into a per-warp shared buffer: draw d
// is word d%4 of Philox({d/4, ant, epoch, stream}, {seed, kDrawKey1}) >> 8;
// lane L computes block 32 b + L of batch b and stores its 4 words (kept
// shifted left, as next_draws writes them).

template <int L>
struct Tables {
  const uint16_t *tier;   // global, or null
  const uint16_t *tier2;  // global, or null
  // This lane's column of the candidate and weight rows: entry nb of cand
  // (w, rel) is row nb / k's.  Lanes without a candidate (k < 32) read one
  // fixed zero entry (column step 0).
  const uint16_t *cand;
  const uint32_t *w;
  const uint8_t *rel;
  uint32_t step;          // 1, or 0 for a lane without a candidate
  const uint32_t *lut;
  const float2 *coords;

  __device__ __forceinline__ int candidate(uint32_t nb) const {
    if (L == kLayoutGlobal) return (int)__ldg(cand + nb * step);
    return (int)cand[nb * step];
  }
  __device__ __forceinline__ uint32_t weight(uint32_t nb) const {
    if (L == kLayoutSmemPacked) return lut[rel[nb * step]];
    // Not the read-only path: k_weights writes them while blocks of this
    // launch are there already.
    return w[nb * step];
  }
  __device__ __forceinline__ float2 coord(int node) const {
    if (L == kLayoutGlobal) return __ldg(coords + node);
    return coords[node];
  }
};

// Nearest unvisited customer that fits (find_nearest_unvisited,
// src/seq/aco_sequential.c:477-493: strict '<' over ascending nodes, so the
// lowest index wins ties).  0 if none.
template <int L, int E>
__device__ __forceinline__ int nearest_unvisited(const Tables<L> &tb, const Unserved<E> &us,
                                                 int n, float2 pc, uint32_t room, int lane) {
  uint32_t best_h;
  uint32_t best_n;
  constexpr bool kG = L == kLayoutGlobal;
  if (kG) best_n = scan_pairs<kG, E, 16>(tb.coords, us, n, pc, room, lane, &best_h);
  else if (n < 256) best_n = scan_pairs<kG, E, 2>(tb.coords, us, n, pc, room, lane, &best_h);
  else best_n = scan_pairs<kG, E, 8>(tb.coords, us, n, pc, room, lane, &best_h);
  const uint32_t mh = __reduce_min_sync(kFull, best_h);
  const uint32_t mn = __reduce_min_sync(kFull, best_h == mh ? best_n : 0xffffffffu);
  return (mh == 0xffffffffu) ? 0 : (int)mn;
}

// The first eligible node of a row of kLen ranks: the node (> 0); 0 when the
// row lists every remaining customer and none is eligible; -1 when none of
// the row is eligible and the row is full (customers beyond it remain).  All
// of the row is loaded at once.
template <int E, int kLen>
__device__ __forceinline__ int tier_row_first(const uint16_t *row, const Unserved<E> &us,
                                              uint32_t room, int lane) {
  constexpr int kParts = kLen / 32;
  int nodes[kParts];
  uint32_t e[kParts];
#pragma unroll
  for (int r = 0; r < kParts; ++r) nodes[r] = (int)__ldg(row + 32 * r + lane);
#pragma unroll
  for (int r = 0; r < kParts; ++r) e[r] = us.get(nodes[r]);  // node 0 (empty slot): visited
#pragma unroll
  for (int r = 0; r < kParts; ++r) {
    const unsigned m = __ballot_sync(kFull, e[r] <= room);
    if (m) return __shfl_sync(kFull, nodes[r], __ffs(m) - 1);
  }
  return (__shfl_sync(kFull, nodes[kParts - 1], 31) == 0) ? 0 : -1;
}

// Second tier: out of line, it is rare.
template <int E>
__device__ __noinline__ int tier2_first(const uint16_t *row, Unserved<E> us, uint32_t room,
                                        int lane) {
  return tier_row_first<E, kTier2Len>(row, us, room, lane);
}

// Nearest eligible customer of the fallback, when no candidate of row cur
// has a weight (find_nearest_unvisited's rule, as nearest_unvisited): the
// first eligible candidate (okm: the row's eligible candidates, the first in
// the highest lane; they come first in the order), else the first eligible
// node of the tier row (the next 64 ranks of the same order), else of the
// second tier row, else the full scan; 0 when the lists hold every customer
// and none is eligible.
template <int L, int E>
__device__ __forceinline__ int nearest_eligible(const Tables<L> &tb, const Unserved<E> &us,
                                                int n, int cur, unsigned okm, int c,
                                                uint32_t room, int lane) {
  if (okm) return __shfl_sync(kFull, c, 31 - __clz(okm));
  if (tb.tier) {
    int r = tier_row_first<E, kTierLen>(tb.tier + (size_t)cur * kTierLen, us, room, lane);
    if (r >= 0) return r;
    if (tb.tier2) {
      r = tier2_first<E>(tb.tier2 + (size_t)cur * kTier2Len, us, room, lane);
      if (r >= 0) return r;
    }
  }
  return nearest_unvisited<L, E>(tb, us, n, tb.coord(cur), room, lane);
}

struct ConstructArgs {
  InstanceView iv;
  EpochTables et;
  AntBuffers ab;
  SmemPlan plan;
  DevState *st;
  uint32_t seed;
  uint32_t epoch;
  uint32_t stream;
  int use_state_epoch;  // 1: epoch number = st->epoch (graph replays)
  const uint32_t *draw_src;  // test hook: recorded draws [m][draw_per_ant], or null
  uint32_t draw_per_ant;
};

// Next 128 draws of an ant, each in the upper 24 bits of its word, or 1 for
// a draw of 0: Philox, or (test hook) the recorded stream, whose draws past
// its end read as 0.
__device__ __noinline__ void next_draws(const ConstructArgs &a, uint32_t *buf, uint32_t d,
                                        uint32_t seed, uint32_t epoch, uint32_t gant, int ant,
                                        int lane) {
  __syncwarp();
  if (a.draw_src) {
    const uint32_t *src = a.draw_src + (size_t)ant * a.draw_per_ant;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t idx = d + 4u * (uint32_t)lane + (uint32_t)q;
      buf[4 * lane + q] =
          max(idx < a.draw_per_ant ? (src[idx] << (32 - kDrawBits)) : 0u, 1u);
    }
  } else {
    uint32_t r[4];
    philox4x32_10((d >> 2) + (uint32_t)lane, gant, epoch, a.stream, seed, kDrawKey1, r);
    constexpr uint32_t kMask = ~0u << (32 - kDrawBits);
    reinterpret_cast<uint4 *>(buf)[lane] =
        make_uint4(max(r[0] & kMask, 1u), max(r[1] & kMask, 1u), max(r[2] & kMask, 1u),
                   max(r[3] & kMask, 1u));
  }
  __syncwarp();
}

// FP64 cost of a compact route sequence, summed in route order
// (solution_cost, src/common/solution.c:126-137).  Lanes compute the arc
// lengths, the sum runs in order in every lane; the (0,0) pairs between
// consecutive routes add +0.0, which leaves the sum unchanged.  128 arcs at
// a time: their end points and square roots overlap (one 32-arc batch at a
// time the root's latency came on top of every batch's adds: 25 cycles per
// arc, of which the dependent add is 9), and the next 128 arcs' end points are loaded
// while the current ones are summed.  A zero length is not given to the
// square root, whose special-case path a single lane would take the warp to.
// kB = 1 is for routes of at most 33 entries.
template <int L, int kB>
__device__ __forceinline__ double route_cost(const Tables<L> &tb, const int *route, int entries,
                                             int lane) {
  double acc = 0.0;
  const int arcs = entries - 1;
  int u[kB], v[kB];
  auto load = [&](int b) {
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      const int j = b + 32 * q + lane;
      u[q] = j < arcs ? route[j] : 0;
      v[q] = j < arcs ? route[j + 1] : 0;
    }
  };
  load(0);
  for (int b = 0; b < arcs; b += 32 * kB) {
    double dj[kB];
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      const float2 pu = tb.coord(u[q]), pv = tb.coord(v[q]);
      const double dx = __dsub_rn((double)pu.x, (double)pv.x);
      const double dy = __dsub_rn((double)pu.y, (double)pv.y);
      dj[q] = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
    }
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      const double r = __dsqrt_rn(dj[q] == 0.0 ? 1.0 : dj[q]);
      dj[q] = dj[q] == 0.0 ? 0.0 : r;
    }
    load(b + 32 * kB);
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      const int cnt = arcs - b - 32 * q;
      if (cnt >= 32) {
#pragma unroll
        for (int t = 0; t < 32; ++t) acc = __dadd_rn(acc, __shfl_sync(kFull, dj[q], t));
      } else {
        for (int t = 0; t < cnt; ++t) acc = __dadd_rn(acc, __shfl_sync(kFull, dj[q], t));
      }
    }
  }
  return acc;
}

// Depot-close weight of the reference-CUDA rule on the scale of the row's
// candidate weights: 2^23 2^(-r/16) for r = rdep (may be negative, i.e. above
// the row maximum), exact in FP64 as LUT[r mod 16] 2^(-floor(r/16)); 0 from
// r = 255 on, like the candidate weights.
__device__ __forceinline__ double depot_weight(int r, const uint32_t *lut) {
  if (r >= kRelMax) return 0.0;
  const int q = (r >= 0) ? (r / 16) : -((-r + 15) / 16);
  return ldexp((double)__ldg(lut + (r - 16 * q)), -q);
}

__device__ __forceinline__ int clamp_int(long long v) {
  return v < 0 ? 0 : (v > INT_MAX ? INT_MAX : (int)v);
}

// One ant, one warp.  Rules of build_ant_solution
// (src/seq/aco_sequential.c:616-681) with the demand extension:
//   vehicle v extends while remaining > 0, remaining demand > (K-v-1) Q and
//   load < Q; the next customer is drawn by roulette over the eligible
//   candidates (unvisited, load + d <= Q), else the nearest eligible one;
//   customers left over are added by the backward repair pass.
// CREF (reference-CUDA depot rule, kernel_construct_solutions,
// src/cuda/aco_cuda_kernels.cu:487-520): vehicle v extends while customers
// remain and load < Q; once the remaining demand fits the later vehicles
// (<= (K-v-1) Q) the route may close: at the depot it closes at once (the
// reference's 2 (1/(0+eps))^beta dwarfs every candidate), with no eligible
// candidate it closes, and after a roulette draw a second draw u closes it
// when u (denom + w_depot) >= denom, w_depot = depot_weight(rdep[cur]).
//
// What bounds it: the latency of the step's dependent chain (row load, the
// candidates' elements, sums, choice, next row's address) at one or two
// warps per scheduler, about 200 cycles of a step's 270 at n=1000.  Candidate t sits in lane
// 31 - t, so that "the first candidate" is the highest lane.
template <int L, int E, bool CREF>
__device__ __forceinline__ void build_ant(const ConstructArgs &a, const Tables<L> &tb,
                                          Unserved<E> &us, uint32_t *dbuf, int *route_s, int ant,
                                          uint32_t epoch, uint32_t seed, int lane) {
  const InstanceView &iv = a.iv;
  const int k = iv.k, K = iv.K, R = iv.route_stride;
  const int cap = (int)iv.cap;
  // The route is built in shared memory where the plan has room for it
  // (route_s), and copied out once it is complete.
  int *route = route_s ? route_s : a.ab.routes + (size_t)ant * R;
  int *lens = a.ab.lens + (size_t)ant * K;
  int *loads = a.ab.loads + (size_t)ant * K;

  // Draws are keyed by the ant's global id (ant_base > 0 when the colony is
  // split over several devices).  128 at a time in dbuf, from the d0-th on:
  // r_next is the current one, left counts it and those after it, da is the
  // next one's shared address.
  const uint32_t gant = (uint32_t)(ant + iv.ant_base);
  uint32_t d0 = 0;
  int left = 128;
  uint32_t da = smem_addr(dbuf), r_next;
  auto next_draw = [&]() {
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r_next) : "r"(da));
    da += 4u;
  };
  auto refill = [&](uint32_t d) {
    next_draws(a, dbuf, d, seed, epoch, gant, ant, lane);
    d0 = d;
    left = 128;
    da = smem_addr(dbuf);
    next_draw();
  };
  refill(0u);
  // Lanes 24..31 hold the first 8 candidates.  A shuffle down by o from lane
  // 31 - j with o > j finds no lane and returns the lane's own weight: 7 - j
  // of the 7 shuffles below do, which the weight's factor 1 - (7 - j) undoes.
  const bool first8 = lane >= 24;
  const uint32_t own = first8 ? 1u - (uint32_t)(lane - 24) : 1u;

  int rem_dem = (int)iv.total_demand;
  int pos = 0;
  // Length and load of vehicle v in lane v mod 32, of the last 32 vehicles.
  int len_r = 0, load_r = 0;

  for (int v = 0; v < K; ++v) {
    const int start = pos;
    if (lane == 0) route[pos] = 0;
    ++pos;
    int cur = 0;
    int room = cap;
    // Demand and room fall together, so "remaining demand > limit and load <
    // Q" is one test of the room against a bound fixed for the vehicle.
    // (Every demand is >= 1, so remaining demand > 0 implies customers left.)
    const long long future = (long long)(K - v - 1) * iv.cap;
    const int floor_room = clamp_int((CREF ? 0 : future) - ((long long)rem_dem - cap));
    // CREF: the route may close once remaining demand <= future; a vehicle
    // that may close at the depot does.
    const long long close64 = future - ((long long)rem_dem - cap);
    const int close_room = close64 < 0 ? -1 : clamp_int(close64);
    bool open = !(CREF && room <= close_room);
    // Row of the current node: candidates, weights and the candidates'
    // elements, requested as soon as the node is known, ahead of the step's
    // bookkeeping and loop test.
    int c = tb.candidate(0u);
    uint32_t w = tb.weight(0u);
    uint32_t e = us.get(c);
    auto take_step = [&](int nx, uint32_t dnx, bool draw) {
      const uint32_t base = (uint32_t)nx * (uint32_t)k;
      c = tb.candidate(base);
      // From shared memory the candidates' elements, which wait for the row's
      // candidates, come before its weights, which do not; a row on its way
      // from L2 is asked for as a whole first (clustered n=2000 483 -> 464 us,
      // n=3000 997 -> 991 us).
      if (L == kLayoutGlobal) w = tb.weight(base);
      us.mark(nx);
      if (L != kLayoutGlobal) {
        e = us.get(c);
        w = tb.weight(base);
      }
      // A draw is consumed only by a roulette selection.
      if (draw) {
        --left;
        next_draw();
      }
      route[pos] = nx;  // every lane stores the same value
      ++pos;
      room -= (int)dnx;
      cur = nx;
      if (L == kLayoutGlobal) e = us.get(c);
    };
    while (open && room > floor_room) {
      // The step loop proper.  Its one loop test is a vote, so that the
      // branch is known to be the warp's, and what is rare (new draws, the
      // fallback) is outside of it: with calls inside, the loop was 37 %
      // slower per step whether or not they were made.
#pragma unroll 1
      while (__any_sync(kFull, room > floor_room && left > 0)) {
        const uint32_t lim = us.limit(room);
        // Lane and candidate (and, where it fits, the candidate's demand) in
        // one word: the largest such word of the lanes past the threshold is
        // the first one's, so one reduction (20 cycles) chooses the customer,
        // where ballot, find-leading-one and shuffle took 60.
        const uint32_t word = E == 1 ? (uint32_t)c | (e << 16) | ((uint32_t)(lane + 1) << 24)
                                     : (uint32_t)c | ((uint32_t)(lane + 1) << 16);
        const uint32_t wv = e <= lim ? w : 0u;
        const uint32_t denom = __reduce_add_sync(kFull, wv);
        // cum 2^24 >= r denom  <=>  cum >= ceil(r denom / 2^24)  <=>
        // cum > floor((R denom - 1) / 2^32) for the draw R = 2^8 r (1 for
        // r = 0: the first sum that is not 0); no sum passes for denom = 0.
        const uint32_t thr = (uint32_t)(((unsigned long long)r_next * denom - 1ull) >> 32);
        // Sum of the 8 masked weights from this lane's on towards lane 31
        // (lanes 24..31: the inclusive prefix, where most draws land) from 7
        // independent shuffles and an add tree: one shuffle latency on the
        // chain instead of the scan's three.  The windows beyond are added
        // only if needed (always: n=1000 195 -> 202 us).
        uint32_t u[8];
        u[0] = wv * own;
#pragma unroll
        for (int o = 1; o < 8; ++o) u[o] = __shfl_down_sync(kFull, wv, o);
        uint32_t cum = ((u[1] + u[2]) + (u[3] + u[4])) + ((u[5] + u[6]) + (u[7] + u[0]));
        uint32_t first = __reduce_max_sync(kFull, first8 && cum > thr ? word : 0u);
        if (first == 0u) {
          const uint32_t t8 = __shfl_down_sync(kFull, cum, 8);
          const uint32_t t16 = __shfl_down_sync(kFull, cum, 16);
          const uint32_t t24 = __shfl_down_sync(kFull, cum, 24);
          cum += (lane < 24 ? t8 : 0u) + (lane < 16 ? t16 : 0u) + (lane < 8 ? t24 : 0u);
          first = __reduce_max_sync(kFull, cum > thr ? word : 0u);
          if (first == 0u) break;  // no eligible candidate has a weight
        }
        const int next = (int)(first & 0xffffu);
        const uint32_t dn = E == 1 ? (first >> 16) & 0xffu : us.get(next);
        if (CREF && room <= close_room) {
          // The roulette draw is spent, and a second one decides.
          if (--left == 0) refill(d0 + 128u); else next_draw();
          const uint32_t r2 = r_next >> (32 - kDrawBits);
          const double wd = depot_weight(a.et.rdep[cur], a.et.lut);
          open = __dmul_rn((double)r2, __dadd_rn((double)denom, wd)) <
                 (double)denom * 16777216.0;
          if (!open) {
            --left;
            next_draw();
            break;
          }
        }
        if (E != 1) __syncwarp();  // every lane has read the element that the step marks
        take_step(next, dn, true);
      }
      if (!open || room <= floor_room) break;
      if (left == 0) {
        refill(d0 + 128u);
        continue;
      }
      // No eligible candidate has a weight: the reference-CUDA rule closes
      // the route when it may; otherwise the nearest eligible customer,
      // which consumes no draw.
      if (CREF && room <= close_room) break;
      const uint32_t lim = us.limit(room);
      const int nx = nearest_eligible<L, E>(tb, us, iv.n, cur, __ballot_sync(kFull, e <= lim), c,
                                            lim, lane);
      if (nx <= 0) break;
      const uint32_t dnx = us.get(nx);
      __syncwarp();  // every lane has read the element that the step marks
      take_step(nx, dnx, false);
    }
    rem_dem -= cap - room;
    if (lane == 0) {
      route[pos] = 0;
      lens[v] = pos + 1 - start;
      loads[v] = cap - room;
    }
    ++pos;
    if (lane == (v & 31)) {
      len_r = pos - start;
      load_r = cap - room;
    }
  }

  int remaining = iv.n - (pos - 2 * K);
  if (remaining > 0) {
    // Backward repair (aco_sequential.c:659-680): from the last vehicle down,
    // reopen the route and append the nearest eligible customers.  The
    // lengths, loads and additions of 32 vehicles at a time are held by the
    // lanes; those of the last 32 never leave them.  The additions are listed
    // in the draw buffer, which is no longer needed, if it holds them all.
    __syncwarp();
    int *rep = remaining <= 128 ? reinterpret_cast<int *>(dbuf) : a.ab.rep + (size_t)ant * iv.n;
    int *repc = a.ab.repc + (size_t)ant * K;
    const int top = (K - 1) & ~31;  // first vehicle of the last group
    int cnt_r = 0;
    int nrep = 0;
    int off_end = pos;
    for (int g = top; g >= 0; g -= 32) {
      const bool read = g < top;
      const int len_l = read ? lens[g + lane] : len_r, load_l = read ? loads[g + lane] : load_r;
      int cnt_l = 0;
      for (int v = min(K - 1, g + 31); v >= g && remaining > 0; --v) {
        const int len_v = __shfl_sync(kFull, len_l, v & 31);
        off_end -= len_v;
        int cur = route[off_end + len_v - 2];
        int load = __shfl_sync(kFull, load_l, v & 31);
        int cnt = 0;
        while (remaining > 0 && load < cap) {
          const int next =
              nearest_unvisited<L, E>(tb, us, iv.n, tb.coord(cur), us.limit(cap - load), lane);
          if (next <= 0) break;
          if (lane == 0) rep[nrep + cnt] = next;
          load += (int)us.get(next);
          __syncwarp();  // every lane has read the element that mark replaces
          us.mark(next);
          __syncwarp();
          ++cnt;
          --remaining;
          cur = next;
        }
        if (lane == (v & 31)) cnt_l = cnt;
        nrep += cnt;
      }
      if (g < top) repc[g + lane] = cnt_l;
      else cnt_r = cnt_l;
    }
    __syncwarp();
    if (nrep > 0) {
      // Re-lay the compact routes with each vehicle's additions appended
      // before its closing depot: vehicles are moved right, last first, down
      // to the first vehicle with an addition; each move takes 32 entries at
      // a time from its end.
      int off_total = pos;
      int add_after = 0;  // additions of vehicles > v (stored first)
      int shift = nrep;   // additions of vehicles <= v
      for (int g = top; g >= 0 && shift > 0; g -= 32) {
        const bool read = g < top, mine = g + lane < K;
        const int len_l = read ? lens[g + lane] : len_r, cnt_l = read ? repc[g + lane] : cnt_r;
        if (mine && cnt_l > 0) lens[g + lane] = len_l + cnt_l;
        for (int v = min(K - 1, g + 31); v >= g && shift > 0; --v) {
          const int len_v = __shfl_sync(kFull, len_l, v & 31);
          const int cnt = __shfl_sync(kFull, cnt_l, v & 31);
          off_total -= len_v;
          shift -= cnt;  // now: additions of vehicles < v
          const int new_off = off_total + shift, main_len = len_v - 1;
          if (shift > 0) {
            for (int t0 = (main_len - 1) & ~31; t0 >= 0; t0 -= 32) {
              const bool in = t0 + lane < main_len;
              const int x = in ? route[off_total + t0 + lane] : 0;
              __syncwarp();
              if (in) route[new_off + t0 + lane] = x;
              __syncwarp();
            }
          }
          for (int j = lane; j < cnt; j += 32) route[new_off + main_len + j] = rep[add_after + j];
          if (lane == 0) route[new_off + main_len + cnt] = 0;
          __syncwarp();
          add_after += cnt;
        }
      }
    }
    pos += nrep;
  }
  __syncwarp();
  const double cost = pos <= 33 ? route_cost<L, 1>(tb, route, pos, lane)
                                : route_cost<L, 4>(tb, route, pos, lane);
  if (route_s) {
    int *g = a.ab.routes + (size_t)ant * R;
    for (int j = lane; j < pos; j += 32) g[j] = route_s[j];
  }
  if (lane == 0) {
    a.ab.cost[ant] = cost;
    a.ab.feasible[ant] = (remaining == 0) ? 1 : 0;
    a.ab.steps[ant] = pos - K;
    a.ab.draws[ant] = d0 + 128u - (uint32_t)left;
  }
}

// What lanes without a candidate read from the global tables.
__device__ const uint32_t g_zero_entry = 0u;

template <int L, int E, bool CREF>
__global__ void __launch_bounds__(512, 1) k_construct(const __grid_constant__ ConstructArgs a) {
  let_next_start();
  extern __shared__ __align__(128) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SmemPlan &pl = a.plan;
  const InstanceView &iv = a.iv;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem);  // fixed tables; weights
  const int t = 31 - lane;  // this lane's candidate
  const bool has = t < iv.k;

  Tables<L> tb;
  tb.tier = iv.tier;
  tb.tier2 = iv.tier2;
  tb.step = has ? 1u : 0u;
  tb.lut = reinterpret_cast<const uint32_t *>(smem + pl.off_lut);
  if (L == kLayoutGlobal) {
    // (The levels and their weights' table instead of the weights put a
    // shared load on the chain behind the row's: n=16000 6450 -> 6640 us.)
    const uint32_t *zero = &g_zero_entry;
    tb.cand = has ? iv.cand + t : reinterpret_cast<const uint16_t *>(zero);
    tb.w = has ? a.et.w + t : zero;
    tb.rel = nullptr;
    tb.coords = iv.coords;
  } else {
    // Bytes 16..23 of the block's shared memory hold the zero entry.
    tb.cand = reinterpret_cast<const uint16_t *>(smem + (has ? pl.off_cand + 2u * t : 16u));
    tb.w = reinterpret_cast<const uint32_t *>(smem + (has ? pl.off_w + 4u * t : 16u));
    tb.rel = smem + (has ? pl.off_w + t : 20u);
    tb.coords = reinterpret_cast<const float2 *>(smem + pl.off_coords);
  }
  if (L == kLayoutSmemPacked) {
    uint32_t *lut = reinterpret_cast<uint32_t *>(smem + pl.off_lut);
    for (int r = threadIdx.x; r < 256; r += blockDim.x) lut[r] = __ldg(a.et.lut + r);
  }
  // Staging by bulk copies: the tables that no epoch changes and every ant's
  // elements on the first barrier, before this launch waits for the kernel
  // that makes the weights; the weights on the second one.
  constexpr bool kElems = !elem_is_bits(E);
  constexpr bool kFixed = L != kLayoutGlobal || kElems, kWeights = L != kLayoutGlobal;
  const uint32_t kChunk = 32768u;
  auto issue = [&](unsigned char *dst, const void *src, uint32_t bytes, uint64_t *on) {
    const unsigned char *sp = reinterpret_cast<const unsigned char *>(src);
    for (uint32_t o = 0; o < bytes; o += kChunk) {
      const uint32_t b = bytes - o < kChunk ? bytes - o : kChunk;
      bulk_g2s(dst + o, sp + o, b, on);
    }
  };
  if (kFixed && threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_init(bar + 1, 1);
    fence_mbar_init();
    reinterpret_cast<uint32_t *>(smem)[4] = 0u;
    reinterpret_cast<uint32_t *>(smem)[5] = kRelMax;  // packed levels: weight 0
    const uint32_t ants = blockDim.x >> 5;
    mbar_arrive_expect_tx(bar, pl.bytes_cand + pl.bytes_coords + (kElems ? ants * pl.vis_bytes : 0u) +
                                   (uint32_t)iv.stage_extra_tx);
    if (kElems)
      for (uint32_t i = 0; i < ants; ++i)
        issue(smem + pl.off_vis + i * pl.vis_bytes, iv.elems, pl.vis_bytes, bar);
    if (L != kLayoutGlobal) {
      issue(smem + pl.off_cand, iv.cand, pl.bytes_cand, bar);
      issue(smem + pl.off_coords, iv.coords, pl.bytes_coords, bar);
    }
  }

  uint32_t *dbuf = reinterpret_cast<uint32_t *>(smem + pl.off_draw) + (size_t)warp * 128;
  Unserved<E> us;
  us.base = smem_addr(smem + pl.off_vis + (size_t)warp * pl.vis_bytes);
  us.chunks = pl.vis_bytes / 16u;
  us.dem = iv.demand;
  if (!kElems) {
    us.init_bits(iv.n, lane);
    __syncwarp();
  }

  wait_for_previous();
  // Graph replays read the epoch number and the seed from the device state,
  // so one captured graph serves every solve of a context.
  uint32_t epoch = a.epoch, seed = a.seed;
  int skip = 0;
  if (a.st) {
    skip = *(volatile int *)&a.st->skip;
    if (a.use_state_epoch) {  // requested with the flag: one round trip
      epoch = *(volatile uint32_t *)&a.st->epoch;
      seed = *(volatile uint32_t *)&a.st->seed;
    }
  }
  if (kWeights && threadIdx.x == 0) {
    mbar_arrive_expect_tx(bar + 1, pl.bytes_w);
    issue(smem + pl.off_w, L == kLayoutSmemPacked ? (const void *)a.et.rel : (const void *)a.et.w,
          pl.bytes_w, bar + 1);
  }
  if (kFixed) {
    // Bounded wait for the staged tables.  The decision is the block's: it
    // goes on only when every thread saw the tables arrive, so no warp
    // enters the full-mask collectives of build_ant with lanes or warps
    // gone.  On time-out the block flags the error, waits (bounded again)
    // for its copies still in flight and exits.  The injected time-out
    // expects stage_extra_tx bytes that no copy brings; thread 0 marks them
    // arrived, so that second wait ends once the real copies have landed.
    // After a genuine time-out the second wait may run out as well; the
    // block then exits with the error flag set.  A skipped epoch waits too:
    // the copies have to land before the block leaves.
    __syncthreads();  // the barriers are initialised
    const uint32_t limit = iv.stage_extra_tx ? (1u << 14) : (1u << 22);
    bool here = mbar_wait_bounded(bar, 0, limit);
    if (kWeights) here = mbar_wait_bounded(bar + 1, 0, limit) && here;
    const bool ok = __syncthreads_and(here ? 1 : 0) != 0;
    if (!ok) {
      if (threadIdx.x == 0) {
        if (a.st && !skip) atomicOr(&a.st->error, kErrStageTimeout);
        if (iv.stage_extra_tx) mbar_complete_tx(bar, (uint32_t)iv.stage_extra_tx);
      }
      __syncthreads();
      mbar_wait_bounded(bar, 0, limit << 2);
      if (kWeights) mbar_wait_bounded(bar + 1, 0, limit << 2);
      __syncthreads();
      return;
    }
  }
  if (skip) return;

  const int ant = blockIdx.x * pl.wpb + warp;
  if (ant >= iv.m) return;
  int *route_s = pl.route_smem
                     ? reinterpret_cast<int *>(smem + pl.off_route) + (size_t)warp * iv.route_stride
                     : nullptr;
  build_ant<L, E, CREF>(a, tb, us, dbuf, route_s, ant, epoch, seed, lane);
}

static int g_max_smem = 0;

int construct_max_smem() {
  if (g_max_smem == 0) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    g_max_smem = v;
  }
  return g_max_smem;
}

static uint32_t pad16(size_t b) { return (uint32_t)((b + 15) & ~size_t(15)); }

SmemPlan plan_construct(const InstanceView &iv, int layout, int num_sms,
                        int max_smem) {
  SmemPlan p = {};
  const size_t rows = (size_t)iv.n + 1;
  int wpb = (iv.m + num_sms - 1) / num_sms;
  if (wpb < 1) wpb = 1;
  if (wpb > 16) wpb = 16;
  const int elem = demand_bytes(iv.max_demand), bit = iv.unit ? kElemUnitBits : kElemBits;
  auto finish = [&](int lay, int el, int ants) {
    p.layout = lay;
    p.elem = el;
    p.wpb = ants;
    p.vis_bytes = unserved_bytes(iv.n, el);
    uint32_t off = 32;  // two barriers, zero entry
    if (lay == kLayoutGlobal) {
      p.bytes_cand = p.bytes_w = p.bytes_coords = 0;
      p.off_cand = p.off_w = p.off_coords = p.off_lut = off;
    } else {
      p.bytes_cand = pad16(rows * iv.k * sizeof(uint16_t));
      p.bytes_coords = pad16(rows * sizeof(float2));
      p.bytes_w = (lay == kLayoutSmemPacked) ? pad16(rows * iv.k) : pad16(rows * iv.k * 4);
      p.off_cand = off; off += p.bytes_cand;
      p.off_w = off; off += p.bytes_w;
      p.off_coords = off; off += p.bytes_coords;
      p.off_lut = off; off += (lay == kLayoutSmemPacked) ? 1024u : 0u;
    }
    p.off_draw = off;
    off += (uint32_t)ants * 512u;
    p.off_vis = off;
    off += (uint32_t)ants * p.vis_bytes;
    p.total = off;
    // Each ant's route in shared memory too, with the tables in shared
    // memory, where it fits and the launch is one block per SM anyway (so
    // the space costs no residency): n=1000 265.0 -> 260.4 us, n=100 34.1
    // -> 33.4 us.  Not with rows from global memory: the space comes out of
    // the L1 that serves those rows (n=3000 1418 -> 1638 us).
    p.route_smem = 0;
    p.off_route = off;
    const size_t rb = pad16((size_t)ants * (size_t)iv.route_stride * 4u);
    if (lay != kLayoutGlobal && off + rb <= (size_t)max_smem &&
        (iv.m + ants - 1) / ants <= num_sms) {
      p.route_smem = 1;
      p.total = off + (uint32_t)rb;
    }
    return (int)p.total <= max_smem;
  };
  // With more ants per block than their elements leave room for, bitmaps (1/8
  // byte per node) instead.
  auto fits = [&](int lay, int ants) { return finish(lay, elem, ants) || finish(lay, bit, ants); };
  // Packed levels with bitmaps come before rows from global memory with
  // elements where the demands, then read through what is left of L1 (24 KB),
  // fit there, and up to 12 ants per block: beyond, the bitmaps' bits cost more
  // to form than the rows' way takes (construction, packed | global: n=2000
  // demands to 1000, 7 ants 625 | 723 us, 11 693 | 721, 16 787 | 774; n=5000
  // k=12, 4 ants 1695 | 1845; n=7000 k=8 2443 | 2414).  Unit demands are not
  // read: n=2000, 16 ants 579 | 651, n=6900 k=8, 4 ants 1494 | 2278.
  const bool bits = iv.unit || (wpb <= 12 && rows <= 6144);
  auto packed_or_global = [&]() {
    if (!finish(kLayoutSmemPacked, elem, wpb) && !(bits && finish(kLayoutSmemPacked, bit, wpb)))
      fits(kLayoutGlobal, wpb);
  };
  if (layout == kLayoutGlobal) {
    fits(kLayoutGlobal, wpb);
  } else if (layout >= 0) {
    // A forced layout: fewer ants per block where not all of them fit.  A
    // unit-demand instance whose tables and draws fit while the one ant's
    // bitmap is up to 300 bytes too much is built with the next layout (the
    // routes are the same) rather than refused.
    int ants = wpb;
    while (!fits(layout, ants) && ants > 1) --ants;
    const size_t words = rows > 2048 ? (rows + 31) / 32 : 0;
    if ((int)p.total > max_smem && wpb == 1 && iv.unit &&
        p.off_draw + 512u - 16u + 4u * words <= (size_t)max_smem)
      packed_or_global();
  } else if (!finish(kLayoutSmemWeights, elem, wpb)) {
    packed_or_global();
  }
  return p;
}

template <int L, int E>
static cudaError_t configure_t() {
  cudaError_t e = cudaFuncSetAttribute(k_construct<L, E, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       construct_max_smem());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_construct<L, E, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, construct_max_smem());
  return e;
}

template <int L>
static cudaError_t configure_l() {
  cudaError_t e = configure_t<L, 1>();
  if (e == cudaSuccess) e = configure_t<L, 2>();
  if (e == cudaSuccess) e = configure_t<L, 4>();
  if (e == cudaSuccess) e = configure_t<L, kElemBits>();
  if (e == cudaSuccess) e = configure_t<L, kElemUnitBits>();
  return e;
}

// Opts every construct instantiation into the full shared-memory carve-out;
// called once per device before any launch or graph capture.
cudaError_t prepare_construct_kernels() {
  cudaError_t e = configure_l<kLayoutSmemWeights>();
  if (e == cudaSuccess) e = configure_l<kLayoutSmemPacked>();
  if (e == cudaSuccess) e = configure_l<kLayoutGlobal>();
  return e;
}

template <int L, int E>
static cudaError_t launch_construct_le(const ConstructArgs &a, cudaStream_t s) {
  const int grid = (a.iv.m + a.plan.wpb - 1) / a.plan.wpb;
  const int threads = a.plan.wpb * 32;
  if (a.iv.depot_rule == kDepotRuleCudaRef) {
    if (!a.et.rdep) return cudaErrorInvalidValue;
    return launch_after(k_construct<L, E, true>, grid, threads, a.plan.total, s, a);
  }
  return launch_after(k_construct<L, E, false>, grid, threads, a.plan.total, s, a);
}

template <int L>
static cudaError_t launch_construct_l(const ConstructArgs &a, cudaStream_t s) {
  switch (a.plan.elem) {
    case 1: return launch_construct_le<L, 1>(a, s);
    case 2: return launch_construct_le<L, 2>(a, s);
    case 4: return launch_construct_le<L, 4>(a, s);
    case kElemBits: return launch_construct_le<L, kElemBits>(a, s);
    case kElemUnitBits: return launch_construct_le<L, kElemUnitBits>(a, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_construct(const InstanceView &iv, const EpochTables &et,
                             const AntBuffers &ab, const SmemPlan &plan,
                             DevState *st, uint32_t seed, uint32_t epoch,
                             uint32_t stream_id, int use_state_epoch,
                             cudaStream_t s, const uint32_t *draw_src,
                             uint32_t draw_per_ant) {
  ConstructArgs a;
  a.draw_src = draw_src;
  a.draw_per_ant = draw_per_ant;
  a.iv = iv;
  a.et = et;
  a.ab = ab;
  a.plan = plan;
  a.st = st;
  a.seed = seed;
  a.epoch = epoch;
  a.stream = stream_id;
  a.use_state_epoch = use_state_epoch;
  if ((int)plan.total > construct_max_smem()) return cudaErrorInvalidValue;
  switch (plan.layout) {
    case kLayoutSmemWeights: return launch_construct_l<kLayoutSmemWeights>(a, s);
    case kLayoutSmemPacked: return launch_construct_l<kLayoutSmemPacked>(a, s);
    case kLayoutGlobal: return launch_construct_l<kLayoutGlobal>(a, s);
  }
  return cudaErrorInvalidValue;
}

// ===========================================================================
// Iteration best, global best and stop rules
// ===========================================================================

// is_significant_improvement, src/cuda/aco_cuda.cu:83-94.
__device__ __forceinline__ bool significant(double prev, double next,
                                            double min_rel) {
  if (prev >= DBL_MAX || next >= DBL_MAX) return next < prev;
  if (next >= __dsub_rn(prev, 1e-9)) return false;
  double gain = __dsub_rn(prev, next);
  double rel = __ddiv_rn(gain, fmax(prev, 1e-9));
  return __dadd_rn(rel, 1e-9) >= min_rel;
}

// Epoch bookkeeping of src/cuda/aco_cuda.cu:349-399 and the stop rules
// checked at the start of the next epoch (:333-339), given the iteration's
// best feasible ant (found, cost bc, ant ba) and its ant-steps.  Returns
// whether the global best improved.
__device__ int epoch_bookkeeping(DevState *st, bool found, double bc, int ba,
                                 unsigned long long steps, EpochRec *log) {
  int improved = 0;
  st->found = found ? 1 : 0;
  st->total_steps += steps;
  if (found) {
    st->iter_best = bc;
    st->best_ant = ba;
    if (bc < st->global_best) {
      improved = 1;
      if (significant(st->global_best, bc, st->min_rel)) st->iter_since_best = 0;
      else st->iter_since_best += 1;
      st->global_best = bc;
    } else {
      st->iter_since_best += 1;
    }
    st->dep_iter = __fdiv_rn(0.3f * st->Qs, (float)bc);
    st->dep_global = __fdiv_rn(0.7f * st->Qs, (float)st->global_best);
  } else {
    st->iter_since_best += 1;
  }
  st->improved = improved;
  st->epoch += 1;
  const unsigned long long now = global_timer_ns();
  const unsigned long long elapsed = now > st->start_ns ? now - st->start_ns : 0ull;
  EpochRec rec;
  rec.epoch = st->epoch;
  rec.iter_since_best = st->iter_since_best;
  rec.improved = improved;
  rec.found = found ? 1 : 0;
  rec.global_best = st->global_best;
  rec.elapsed_ns = elapsed;
  if (log) log[st->log_count % kLogCap] = rec;
  st->log_count += 1;
  int flags = st->stop_flags;
  if (st->stagnation > 0 && st->iter_since_best >= st->stagnation) flags |= kStopStagnation;
  if (st->fixed_epochs > 0 && st->epoch >= st->fixed_epochs) flags |= kStopFixed;
  if (st->timeout_ns > 0ull && elapsed > st->timeout_ns) flags |= kStopTimeout;
  if (st->run_limit > 0 && st->epoch >= st->run_limit) flags |= kStopRunLimit;
  st->stop_flags = flags;
  return improved;
}

// The device state staged in shared memory by one block: one coalesced read,
// the bookkeeping on the copy, one write-back before the block ends.
__device__ __forceinline__ void state_load(DevState *s, const DevState *g) {
  static_assert(sizeof(DevState) % sizeof(int) == 0, "DevState is whole words");
  constexpr int kWords = (int)(sizeof(DevState) / sizeof(int));
  for (int i = threadIdx.x; i < kWords; i += blockDim.x)
    reinterpret_cast<int *>(s)[i] = reinterpret_cast<const volatile int *>(g)[i];
  __syncthreads();
}
__device__ __forceinline__ void state_store(DevState *g, const DevState *s) {
  constexpr int kWords = (int)(sizeof(DevState) / sizeof(int));
  for (int i = threadIdx.x; i < kWords; i += blockDim.x)
    reinterpret_cast<int *>(g)[i] = reinterpret_cast<const int *>(s)[i];
}

constexpr int kEvapUnroll = 4;
constexpr int kEvapThreads = 512;

// Folds (oc, oa) into the running best (bc, ba): least cost, then lowest
// ant (the first minimum of select_iter_best_host, src/cuda/aco_cuda.cu:96-126).
__device__ __forceinline__ void best_fold(double &bc, int &ba, double oc, int oa) {
  if (oa != INT_MAX && (ba == INT_MAX || oc < bc || (oc == bc && oa < ba))) {
    bc = oc;
    ba = oa;
  }
}

__device__ __forceinline__ void warp_best(double &bc, int &ba, unsigned long long &steps) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double oc = __shfl_down_sync(kFull, bc, o);
    const int oa = __shfl_down_sync(kFull, ba, o);
    steps += __shfl_down_sync(kFull, steps, o);
    best_fold(bc, ba, oc, oa);
  }
}

// Iteration best of the m ants (INT_MAX: none feasible) and their
// ant-steps, over one block; every thread calls it, lane 0 of warp 0 holds
// the result.  The s_* scratch holds one entry per warp.
__device__ __forceinline__ void block_iter_best(const AntBuffers &ab, int m, double *s_cost,
                                                int *s_ant, unsigned long long *s_steps,
                                                double &bc, int &ba, unsigned long long &steps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  bc = DBL_MAX;
  ba = INT_MAX;
  steps = 0;
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    steps += (unsigned long long)ab.steps[i];
    if (ab.feasible[i]) {
      const double c = ab.cost[i];
      if (ba == INT_MAX || c < bc) {  // ascending i: first minimum kept
        bc = c;
        ba = i;
      }
    }
  }
  warp_best(bc, ba, steps);
  if (lane == 0) {
    s_cost[warp] = bc;
    s_ant[warp] = ba;
    s_steps[warp] = steps;
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    bc = (lane < nw) ? s_cost[lane] : DBL_MAX;
    ba = (lane < nw) ? s_ant[lane] : INT_MAX;
    steps = (lane < nw) ? s_steps[lane] : 0ull;
    warp_best(bc, ba, steps);
  }
}

// The pipelined epoch's iteration best, bookkeeping and both deposits over a
// cluster of kBestCluster blocks, so that the deposits' scattered pheromone
// reads and writes are issued from as many SMs.  Every block finds the same
// iteration best and, from the same state snapshot, the same deposit
// amounts; block 0 alone keeps the bookkeeping (state, log, global-best
// copy).  The cluster barrier puts the iteration-best deposit before the
// global-best one.
constexpr int kBestCluster = 8;
constexpr int kBestThreads = 256;

// Deposit of a complete solution (n + 2K entries) over gthreads threads, this
// one gtid: one arc (p, q) of consecutive entries per thread, both cells
// loaded together; the arcs of different customers' pairs touch different
// cells, but the two arcs of a one-customer route [0 p 0] share theirs and go
// to one thread in order.  (0, 0) pairs are route boundaries and empty
// routes; the empty routes' own cell (0, 0) is raised once per empty route by
// the thread with gtid 0's warp.
__device__ __forceinline__ void deposit_pair(const PheromoneView &pv, size_t stride, int u, int c,
                                             float dep) {
  uint8_t *fwd = pv.tau + (size_t)u * stride + c, *rev = pv.tau + (size_t)c * stride + u;
  const uint8_t old = ld_cg_u8(fwd), oldr = ld_cg_u8(rev);
  const uint8_t nq = quant(dequant(old, pv.log_min, pv.log_step) + dep, pv.log_min, pv.log_step,
                           pv.q_min, pv.q_max);
  if (nq > old) st_cg_u8(fwd, nq);
  if (nq > oldr) st_cg_u8(rev, nq);
}

__device__ __forceinline__ void deposit_complete(const PheromoneView &pv, size_t stride,
                                                 const int *nodes, const int *lens, int n, int K,
                                                 float dep, int gtid, int gthreads) {
  const int total = n + 2 * K;
  for (int j = 1 + gtid; j < total; j += gthreads) {
    const int p = nodes[j - 1], q = nodes[j];
    const int before = j >= 2 ? nodes[j - 2] : 0, after = j + 1 < total ? nodes[j + 1] : 0;
    if (p == 0 && q == 0) continue;
    if (q == 0 && before == 0) continue;  // second arc of [0 p 0]
    deposit_pair(pv, stride, p, q, dep);
    if (p == 0 && after == 0) deposit_pair(pv, stride, q, 0, dep);
  }
  if (gtid < 32) {
    int empty = 0;
    for (int b = 0; b < K; b += 32)
      empty += __popc(__ballot_sync(kFull, b + gtid < K && lens[b + gtid] == 2));
    if (gtid == 0 && empty > 0) {
      const uint8_t old = ld_cg_u8(pv.tau);
      uint8_t q = old;
      for (int i = 0; i < empty; ++i) {
        const uint8_t nq = quant(dequant(q, pv.log_min, pv.log_step) + dep, pv.log_min,
                                 pv.log_step, pv.q_min, pv.q_max);
        if (nq <= q) break;  // and so would every further one be
        q = nq;
      }
      if (q > old) st_cg_u8(pv.tau, q);
    }
  }
}

// The epoch's two deposits over the cluster, into the buffer evaporated
// beside the construction: the iteration best, a cluster barrier (its stores
// before the next deposit's loads, release / acquire at cluster scope), the
// global best; then block 0 switches the buffer and writes the state back.
__device__ __forceinline__ void cluster_deposits(cooperative_groups::cluster_group &cluster,
                                                 int rank, const InstanceView &iv,
                                                 const PheromoneView &pv, uint8_t *tau_alt,
                                                 DevState *s_st, DevState *st,
                                                 const int *it_nodes, const int *it_lens,
                                                 const int *gb_nodes, const int *gb_lens) {
  const bool sel = s_st->tau_sel != 0;
  PheromoneView pd = pv;
  pd.tau = sel ? pv.tau : tau_alt;  // the evaporated copy
  const size_t stride_n = (size_t)iv.n + 1;
  const int gt = rank * kBestThreads + (int)threadIdx.x, gn = kBestCluster * kBestThreads;
  deposit_complete(pd, stride_n, it_nodes, it_lens, iv.n, iv.K, s_st->dep_iter, gt, gn);
  cluster.sync();
  deposit_complete(pd, stride_n, gb_nodes, gb_lens, iv.n, iv.K, s_st->dep_global, gt, gn);
  if (rank == 0) {
    __syncthreads();
    if (threadIdx.x == 0) s_st->tau_sel = sel ? 0 : 1;
    __syncthreads();
    state_store(st, s_st);
  }
}

__global__ void __cluster_dims__(kBestCluster, 1, 1) __launch_bounds__(kBestThreads)
    k_best_cluster(InstanceView iv, AntBuffers ab, DevState *st, int *gbest_nodes,
                   int *gbest_lens, EpochRec *log, PheromoneView pv, uint8_t *tau_alt) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  __shared__ DevState s_st;
  __shared__ double s_cost[kBestThreads / 32];
  __shared__ int s_ant[kBestThreads / 32];
  __shared__ unsigned long long s_steps[kBestThreads / 32];
  __shared__ int s_improved, s_best;
  let_next_start();
  state_load(&s_st, st);
  double bc;
  int ba;
  unsigned long long steps;
  block_iter_best(ab, iv.m, s_cost, s_ant, s_steps, bc, ba, steps);
  if (s_st.skip) return;  // the same in every block: nothing is written
  if (threadIdx.x == 0) {
    // Each block updates its own copy; only block 0's copy and log entry are
    // kept (the others differ at most in the elapsed-time fields).
    s_improved = epoch_bookkeeping(&s_st, ba != INT_MAX, bc, ba, steps, rank == 0 ? log : nullptr);
    s_best = ba;
  }
  __syncthreads();
  const int R = iv.route_stride;
  if (rank == 0 && s_improved) {
    // New global best: keep a copy (aco_cuda.cu:367-380).
    const int *src = ab.routes + (size_t)s_best * R;
    const int *sl = ab.lens + (size_t)s_best * iv.K;
    int total = 0;
    for (int v = 0; v < iv.K; ++v) total += sl[v];
    for (int t = threadIdx.x; t < total; t += blockDim.x) gbest_nodes[t] = src[t];
    for (int v = threadIdx.x; v < iv.K; v += blockDim.x) gbest_lens[v] = sl[v];
  }
  if (s_best == INT_MAX) {
    // No feasible ant: no evaporation, no deposit; every block has read the
    // state before block 0 writes it back.
    cluster.sync();
    if (rank == 0) state_store(st, &s_st);
    return;
  }
  const int *it_nodes = ab.routes + (size_t)s_best * R;
  const int *it_lens = ab.lens + (size_t)s_best * iv.K;
  // The global best is this epoch's iteration best when it improved (the
  // copy block 0 makes holds the same routes).
  cluster_deposits(cluster, rank, iv, pv, tau_alt, &s_st, st, it_nodes, it_lens,
                   s_improved ? it_nodes : gbest_nodes, s_improved ? it_lens : gbest_lens);
}

cudaError_t launch_best_deposit(const InstanceView &iv, const AntBuffers &ab,
                                const PheromoneView &pv, uint8_t *tau_alt, DevState *st,
                                int *gbest_nodes, int *gbest_lens, EpochRec *log,
                                cudaStream_t s) {
  k_best_cluster<<<kBestCluster, kBestThreads, 0, s>>>(iv, ab, st, gbest_nodes, gbest_lens, log,
                                                       pv, tau_alt);
  return cudaGetLastError();
}

// Evaporation of the current pheromone buffer into the other one, run beside
// the construction (which reads only the weights): 16 bytes per thread,
// max(q, q_min + delta) - delta.
__global__ void __launch_bounds__(kEvapThreads) k_evaporate_to(PheromoneView pv,
                                                               uint8_t *tau_alt, DevState *st) {
  if (*(volatile int *)&st->skip) return;
  const bool sel = *(volatile int *)&st->tau_sel != 0;
  const uint8_t *src = sel ? tau_alt : pv.tau;
  uint8_t *dst = sel ? pv.tau : tau_alt;
  evap_sweep<kEvapUnroll>(src, dst, pv.total, pv.q_min, pv.delta);
}

// Blocks of an evaporation sweep over `total` bytes: one per kEvapUnroll *
// kEvapThreads vectors, at most one wave (the blocks resident on all SMs at
// once), so that large matrices are swept by a grid-stride loop: a block
// waits for the state's flags before its first load, which a block per tile
// would do for every tile (n=16000: 88 against 155 us).
int evap_grid_for(unsigned long long total, int num_sms) {
  static int resident = 0;
  if (resident == 0) {
    int r = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_evaporate_to, kEvapThreads, 0) !=
            cudaSuccess ||
        r < 1)
      r = 1;
    resident = r;
  }
  const unsigned long long per_block = (unsigned long long)kEvapUnroll * kEvapThreads;
  unsigned long long g = (total / 16 + per_block - 1) / per_block;
  const unsigned long long cap =
      (unsigned long long)(num_sms > 0 ? num_sms : 148) * (unsigned long long)resident;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

cudaError_t launch_evaporate_to(const PheromoneView &pv, uint8_t *tau_alt, DevState *st,
                                int grid, cudaStream_t s) {
  k_evaporate_to<<<grid, kEvapThreads, 0, s>>>(pv, tau_alt, st);
  return cudaGetLastError();
}

__global__ void k_set_run_limit(DevState *st, int limit) {
  st->run_limit = limit;
  st->stop_flags &= ~kStopRunLimit;
  if (limit > 0 && st->epoch >= limit) st->stop_flags |= kStopRunLimit;
}

cudaError_t launch_set_run_limit(DevState *st, int limit, cudaStream_t s) {
  k_set_run_limit<<<1, 1, 0, s>>>(st, limit);
  return cudaGetLastError();
}

// ===========================================================================
// Evaporation + deposit
// ===========================================================================

struct EvapArgs {
  InstanceView iv;
  PheromoneView pv;
  AntBuffers ab;
  const int *gbest_nodes;
  const int *gbest_lens;
  unsigned int *counter;
  int best_ant;
  float dep_iter, dep_global;
};

__global__ void __launch_bounds__(kEvapThreads) k_evap_deposit(EvapArgs a) {
  const PheromoneView &pv = a.pv;
  evap_sweep<kEvapUnroll>(pv.tau, pv.tau, pv.total, pv.q_min, pv.delta);
  // The last block to finish the sweep deposits (threadfence reduction).
  __shared__ int s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned ticket = atomicAdd(a.counter, 1u);
    s_last = (ticket == gridDim.x - 1) ? 1 : 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const size_t stride_n = (size_t)a.iv.n + 1;
  const int best = a.best_ant;
  const float dep_i = a.dep_iter, dep_g = a.dep_global;
  extern __shared__ int s_off[];
  int *offs = (a.iv.K <= kDepositSmemRoutes) ? s_off : nullptr;
  deposit_solution(pv, stride_n, CompactNodes{a.ab.routes + (size_t)best * a.iv.route_stride},
                   a.ab.lens + (size_t)best * a.iv.K, a.iv.K, dep_i, offs);
  __syncthreads();
  if (a.gbest_nodes) {
    deposit_solution(pv, stride_n, CompactNodes{a.gbest_nodes}, a.gbest_lens, a.iv.K, dep_g, offs);
  }
  if (threadIdx.x == 0) *a.counter = 0u;
}

// In place, with the ant and the amounts given by the caller.
cudaError_t launch_evap_deposit_explicit(const InstanceView &iv,
                                         const PheromoneView &pv,
                                         const AntBuffers &ab, int best_ant,
                                         float dep_iter,
                                         const int *gbest_nodes,
                                         const int *gbest_lens,
                                         float dep_global,
                                         unsigned int *counter, int grid,
                                         cudaStream_t s) {
  EvapArgs a;
  a.iv = iv;
  a.pv = pv;
  a.ab = ab;
  a.gbest_nodes = gbest_nodes;
  a.gbest_lens = gbest_lens;
  a.counter = counter;
  a.best_ant = best_ant;
  a.dep_iter = dep_iter;
  a.dep_global = dep_global;
  const size_t smem = iv.K <= kDepositSmemRoutes ? sizeof(int) * (iv.K + 1) : 0;
  k_evap_deposit<<<grid, kEvapThreads, smem, s>>>(a);
  return cudaGetLastError();
}

// ===========================================================================
// Colony split over several devices: local best packet, exchange, winner
// ===========================================================================

// Packet of one device's iteration best (int32 words):
//   [0,1] cost (FP64 bits; DBL_MAX when no feasible ant)  [2] found
//   [3] global ant id  [4,5] ant-steps of all local ants  [6, 6+K) lengths
//   [6+K, 6+K+n+2K) compact route.
__host__ __device__ inline int shard_packet_ints(int n, int K) {
  return (6 + K + n + 2 * K + 3) & ~3;
}

__global__ void __launch_bounds__(1024) k_shard_pack(InstanceView iv, AntBuffers ab,
                                                     DevState *st, int *send) {
  __shared__ double s_cost[32];
  __shared__ int s_ant[32];
  __shared__ unsigned long long s_steps[32];
  __shared__ int s_best;
  const bool skip = *(volatile int *)&st->skip;
  double bc;
  int ba;
  unsigned long long steps;
  block_iter_best(ab, skip ? 0 : iv.m, s_cost, s_ant, s_steps, bc, ba, steps);
  if (threadIdx.x == 0) {
    const unsigned long long cb = (unsigned long long)__double_as_longlong(bc);
    send[0] = (int)(cb & 0xffffffffu);
    send[1] = (int)(cb >> 32);
    send[2] = (ba != INT_MAX) ? 1 : 0;
    send[3] = (ba != INT_MAX) ? ba + iv.ant_base : INT_MAX;
    send[4] = (int)(steps & 0xffffffffu);
    send[5] = (int)(steps >> 32);
    s_best = ba;
  }
  __syncthreads();
  if (s_best != INT_MAX) {
    const int *src = ab.routes + (size_t)s_best * iv.route_stride;
    const int *sl = ab.lens + (size_t)s_best * iv.K;
    for (int v = threadIdx.x; v < iv.K; v += blockDim.x) send[6 + v] = sl[v];
    int total = 0;
    for (int v = 0; v < iv.K; ++v) total += sl[v];
    for (int t = threadIdx.x; t < total; t += blockDim.x) send[6 + iv.K + t] = src[t];
  }
}

// Winner over the gathered packets (lowest cost, then lowest global ant:
// the first minimum a single device holding every ant would find), then the
// same bookkeeping as k_best_cluster; its route goes to iter_nodes/iter_lens and,
// on improvement, to the global best; then both deposits into the
// evaporated pheromone buffer and the buffer switch.
__global__ void __cluster_dims__(kBestCluster, 1, 1) __launch_bounds__(kBestThreads)
    k_shard_select(InstanceView iv, DevState *st, const int *recv, int world, int *iter_nodes,
                   int *iter_lens, int *gbest_nodes, int *gbest_lens, EpochRec *log,
                   PheromoneView pv, uint8_t *tau_alt) {
  // A cluster like k_best_cluster: every block selects the same winner and
  // deposit amounts from the same packets and state snapshot, block 0 keeps
  // the bookkeeping and the copies, the deposits' arcs are shared out over
  // the cluster with a barrier between the two deposits.
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  __shared__ DevState s_st;
  __shared__ int s_src, s_improved;
  state_load(&s_st, st);
  if (s_st.skip) return;  // the same in every block: nothing is written
  const int P = shard_packet_ints(iv.n, iv.K);
  if (threadIdx.x == 0) {
    double bc = DBL_MAX;
    int ba = INT_MAX, src = -1;
    unsigned long long steps = 0;
    for (int r = 0; r < world; ++r) {
      const int *pk = recv + (size_t)r * P;
      steps += (unsigned long long)(unsigned)pk[4] | ((unsigned long long)(unsigned)pk[5] << 32);
      if (!pk[2]) continue;
      const double c = __longlong_as_double(
          (long long)((unsigned long long)(unsigned)pk[0] | ((unsigned long long)(unsigned)pk[1] << 32)));
      const int ga = pk[3];
      if (src < 0 || c < bc || (c == bc && ga < ba)) {
        bc = c;
        ba = ga;
        src = r;
      }
    }
    s_improved = epoch_bookkeeping(&s_st, src >= 0, bc, ba, steps, rank == 0 ? log : nullptr);
    s_src = src;
  }
  __syncthreads();
  if (s_src < 0) {
    // No feasible ant anywhere: no evaporation, no deposit; every block has
    // read the state before block 0 writes it back.
    cluster.sync();
    if (rank == 0) state_store(st, &s_st);
    return;
  }
  const int *pk = recv + (size_t)s_src * P;
  const int *w_lens = pk + 6;
  const int *w_nodes = pk + 6 + iv.K;
  if (rank == 0) {
    int total = 0;
    for (int v = 0; v < iv.K; ++v) total += w_lens[v];
    for (int v = threadIdx.x; v < iv.K; v += blockDim.x) {
      iter_lens[v] = w_lens[v];
      if (s_improved) gbest_lens[v] = w_lens[v];
    }
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
      iter_nodes[t] = w_nodes[t];
      if (s_improved) gbest_nodes[t] = w_nodes[t];
    }
  }
  // The deposits read the winner straight from its packet.
  cluster_deposits(cluster, rank, iv, pv, tau_alt, &s_st, st, w_nodes, w_lens,
                   s_improved ? w_nodes : gbest_nodes, s_improved ? w_lens : gbest_lens);
}

int shard_packet_size(int n, int K) { return shard_packet_ints(n, K); }

cudaError_t launch_shard_pack(const InstanceView &iv, const AntBuffers &ab, DevState *st,
                              int *send, cudaStream_t s) {
  k_shard_pack<<<1, 1024, 0, s>>>(iv, ab, st, send);
  return cudaGetLastError();
}

cudaError_t launch_shard_select(const InstanceView &iv, DevState *st, const int *recv,
                                int world, int *iter_nodes, int *iter_lens,
                                int *gbest_nodes, int *gbest_lens, EpochRec *log,
                                const PheromoneView &pv, uint8_t *tau_alt, cudaStream_t s) {
  k_shard_select<<<kBestCluster, kBestThreads, 0, s>>>(iv, st, recv, world, iter_nodes,
                                                          iter_lens, gbest_nodes, gbest_lens,
                                                          log, pv, tau_alt);
  return cudaGetLastError();
}

}  // namespace acob200
