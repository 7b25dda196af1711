// aco_noalloc.cu -- pheromone evaporation + deposit that allocates nothing.
//
// Some callers cannot allocate device memory once they are running: a host
// application that reserves all device memory up front and hands plugins
// only the buffers it owns (a framework with its own caching allocator, a
// solver service with a fixed memory budget), or a real-time loop that must
// not call cudaMalloc/cudaFree because they can synchronise the device and
// can fail under memory pressure.  For them this file offers
// aco_b200_evaporate_deposit_noalloc: the caller passes every input and
// output as a device pointer, and the kernels' scratch is shared memory.
#include "aco_internal.cuh"

extern "C" {
#include "aco.h"
#include "aco_b200.h"
}

#include <cooperative_groups.h>

#include <cmath>
#include <cstdio>

using namespace acob200;

// Largest number of routes per solution: their offsets are kept in a block's
// shared memory.
constexpr int kNoAllocMaxRoutes = 4096;

namespace {

constexpr int kDepositThreads = 256;

// A block per tile: with one resident wave striding over the matrix, reads
// and writes spread over all of it all the time (n=16000, in place: 90.6 us,
// 5.65 TB/s, against 77.3 us, 6.62 TB/s).
constexpr int kSweepUnroll = 2;
constexpr int kSweepThreads = 256;

__global__ void __launch_bounds__(kSweepThreads) k_noalloc_sweep(PheromoneView pv) {
  evap_sweep<kSweepUnroll>(pv.tau, pv.tau, pv.total, pv.q_min, pv.delta);
}

// One solution's deposit, its arcs one per thread over the grid: at large n
// every arc waits for its cells' way from HBM, and one block walking them all
// after the sweep took longer than the sweep (n=16000: 100 us; these launches
// take 3 us each behind it).
__global__ void __launch_bounds__(kDepositThreads)
    k_noalloc_deposit(PheromoneView pv, int n, int K, const int *nodes, const int *lens, float dep) {
  extern __shared__ int s_off[];
  let_next_start();
  wait_for_previous();
  deposit_solution(pv, (size_t)n + 1, CompactNodes{nodes}, lens, K, dep, s_off,
                   (int)(blockIdx.x * blockDim.x + threadIdx.x), (int)(gridDim.x * blockDim.x));
}

// Small matrices with few routes: the sweep and both deposits in one launch, a
// cluster of blocks with its barrier in between.  Three launches cost the host
// 12.6 us, this one 8.4 (one kernel whose last block deposits, with its scratch
// cleared by a memset, took 9.6): n=100 K=5 8.4 us per call, 12.8 with three
// launches; n=500 K=1 10.8 and 12.8.  Beyond, eight SMs sweep and deposit too
// slowly (n=1000 K=1 14.9 and 12.7, n=512 K=16 14.5 and 12.7, n=50 K=50 39.0
// and 37.0).
constexpr int kSmallCluster = 8;
constexpr int kSmallThreads = 512;
inline bool small_update(int n, int K) { return K <= 16 && n <= 640 - 16 * K; }

__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(kSmallThreads)
    k_noalloc_small(PheromoneView pv, int n, int K, const int *it_nodes, const int *it_lens,
                    float dep_it, const int *gb_nodes, const int *gb_lens, float dep_gb) {
  extern __shared__ int s_off[];
  const auto cluster = cooperative_groups::this_cluster();
  const int gt = (int)(blockIdx.x * blockDim.x + threadIdx.x), gn = kSmallCluster * kSmallThreads;
  evap_sweep<kSweepUnroll>(pv.tau, pv.tau, pv.total, pv.q_min, pv.delta);
  cluster.sync();
  deposit_solution(pv, (size_t)n + 1, CompactNodes{it_nodes}, it_lens, K, dep_it, s_off, gt, gn);
  if (!gb_nodes) return;
  cluster.sync();
  deposit_solution(pv, (size_t)n + 1, CompactNodes{gb_nodes}, gb_lens, K, dep_gb, s_off, gt, gn);
}

}  // namespace

extern "C" ACO_API int aco_b200_evaporate_deposit_noalloc(
    uint8_t *d_tau, int n, int K, const int *d_iter_nodes, const int *d_iter_lens,
    float dep_iter, const int *d_gbest_nodes, const int *d_gbest_lens, float dep_global,
    double rho, void *stream) {
  if (!d_tau || !d_iter_nodes || !d_iter_lens || n < 1 || K < 1 ||
      (d_gbest_nodes == nullptr) != (d_gbest_lens == nullptr) || !(rho > 0.0 && rho < 1.0)) {
    fprintf(stderr, "aco_b200_evaporate_deposit_noalloc: invalid arguments\n");
    return ACO_ERR_INVALID_INPUT;
  }
  if (((uintptr_t)d_tau & 15u) != 0u) {
    fprintf(stderr, "aco_b200_evaporate_deposit_noalloc: d_tau must be 16-byte aligned\n");
    return ACO_ERR_INVALID_INPUT;
  }
  if (K > kNoAllocMaxRoutes) {
    fprintf(stderr,
            "aco_b200_evaporate_deposit_noalloc: K=%d routes exceed the limit "
            "(at most %d routes per solution)\n",
            K, kNoAllocMaxRoutes);
    return ACO_ERR_INVALID_INPUT;
  }
  // Quantization constants of the reference (src/cuda/aco_cuda.cu:209-215).
  const float lmin = logf(0.0001f);
  const float lmax = logf(100.0f);
  const float step = (lmax - lmin) / 255.0f;
  const float log_rho = logf(1.0f - (float)rho);
  PheromoneView pv;
  pv.tau = d_tau;
  pv.total = (unsigned long long)(n + 1) * (unsigned long long)(n + 1);
  pv.log_min = lmin;
  pv.log_step = step;
  pv.q_min = 0;
  pv.q_max = 255;
  pv.delta = (uint8_t)fmaxf(1.0f, roundf(-log_rho / step));
  pv.pad = 0;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t smem = sizeof(int) * (size_t)(K + 1);
  if (small_update(n, K)) {
    k_noalloc_small<<<kSmallCluster, kSmallThreads, smem, s>>>(
        pv, n, K, d_iter_nodes, d_iter_lens, dep_iter, d_gbest_nodes, d_gbest_lens, dep_global);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      fprintf(stderr, "aco_b200_evaporate_deposit_noalloc: launch: %s\n", cudaGetErrorString(e));
      return ACO_ERR_BACKEND;
    }
    return ACO_OK;
  }
  const unsigned long long tile = (unsigned long long)kSweepUnroll * kSweepThreads;
  const unsigned long long tiles = (pv.total / 16 + tile - 1) / tile;
  k_noalloc_sweep<<<(unsigned)(tiles < 1 ? 1 : tiles), kSweepThreads, 0, s>>>(pv);
  cudaError_t e = cudaGetLastError();
  const int grid = (n + 2 * K + kDepositThreads - 1) / kDepositThreads;
  if (e == cudaSuccess)
    e = launch_after(k_noalloc_deposit, grid, kDepositThreads, smem, s, pv, n, K, d_iter_nodes,
                     d_iter_lens, dep_iter);
  if (e == cudaSuccess && d_gbest_nodes)
    e = launch_after(k_noalloc_deposit, grid, kDepositThreads, smem, s, pv, n, K, d_gbest_nodes,
                     d_gbest_lens, dep_global);
  if (e != cudaSuccess) {
    fprintf(stderr, "aco_b200_evaporate_deposit_noalloc: launch: %s\n", cudaGetErrorString(e));
    return ACO_ERR_BACKEND;
  }
  return ACO_OK;
}
