// aco_prior.cu -- learned heuristic prior for the candidate edges.
//
// The plain path weighs candidate c of node i by eta^beta = d(i,c)^-beta,
// entered as integer levels L (16 per octave) in the selection weights
// (k_weights).  The learned prior replaces those levels with
//     L_t = round(gamma * (s_max - s_t) * 16 / ln 2),   s = MLP(features),
// i.e. a weight proportional to exp(gamma * s), so the construction stays
// the same exact integer roulette; the plain levels remain the fallback.
//
//   features  k_prior_features: 8 values per candidate edge, computed in
//             FP32 and stored as BF16 ([row][32 slots][8], 16 bytes/edge)
//   MLP       8 -> 64 -> 64 -> 1, ReLU, BF16 operands, FP32 accumulation on
//             the tcgen05 tensor cores (k_prior_mlp): a 128-edge tile
//             (4 rows x 32 slots) per step; forward for inference, forward
//             + backward for training
//   loss      softmax cross-entropy over each row's valid slots against the
//             successor taken by an elite route
//   optimiser Adam (k_prior_reduce)
//
// Layer 1 carries its bias as the weight of a constant-one input (input 8
// of the 16-wide K of the first MMA), so one GEMM
//     [dZ2^T ; dZ1^T] (128 x E) * [H1^T ; X^T]^T (E x 80)
// accumulated in tensor memory over a block's tiles yields dW2 (rows 0-63,
// columns 0-63), db2 (column 72), dW1 and db1 (rows 64-127, columns 64-72).
#include "aco_internal.cuh"
#include "aco_prior_internal.h"
#include "umma.cuh"

#include <cuda_bf16.h>

extern "C" {
#include "aco.h"
#include "aco_b200.h"
}

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

namespace acob200 {
namespace prior {

// Parameter vector (FP32): W1[64][8], b1[64], W2[64][64], b2[64], w3[64], b3.
constexpr int kW1 = 0, kB1 = 512, kW2 = 576, kB2 = 4672, kW3 = 4736, kB3 = 4800;
constexpr int kParams = 4801;
constexpr int kGradStride = 4808;  // partial-gradient row: kParams values, then the loss
static_assert(kParams == ACO_B200_PRIOR_PARAMS, "parameter count");

constexpr int kSlots = 32;      // candidate slots per row (k <= 32); a tile is 4 rows
constexpr uint32_t kPolls = 1u << 24;

// Shared-memory layout of k_prior_mlp (bytes; operand tiles in 8 x 8 core
// matrices, see umma.cuh).  Every tile is stored once, rows = edges (units for
// the weights): the products that need its transpose read it MN-major.  H1 and
// the inputs are neighbours, and so are dZ2 and dZ1: each pair is one operand
// of the weight-gradient product.  Transposed copies of H1, the inputs, dZ2,
// dZ1 and W2 took 200 two-byte stores per edge and 30 KB more: 3.07 ms for 56
// steps of 4096 examples, 2.82 ms without them.
constexpr uint32_t kSB1 = 0;                         // W1|b1   64 x 16
constexpr uint32_t kSB2 = kSB1 + 64 * 16 * 2;         // W2      64 x 64 [o][j]
constexpr uint32_t kSA2 = kSB2 + 64 * 64 * 2;         // H1      128 x 64
constexpr uint32_t kSA1 = kSA2 + 128 * 64 * 2;        // X       128 x 16
constexpr uint32_t kSHX = 128 * (64 + 16) * 2;         // H1 and X, of alternate tiles
constexpr uint32_t kSdZ2 = kSA2 + 2 * kSHX;           // dZ2     128 x 64
constexpr uint32_t kSdZ1 = kSdZ2 + 128 * 64 * 2;      // dZ1     128 x 64
constexpr uint32_t kSF32 = kSdZ1 + 128 * 64 * 2;      // b2[64], w3[64]
constexpr uint32_t kSRed = kSF32 + 128 * 4;           // 4 warps x 65 partial sums
constexpr uint32_t kSBar = kSRed + 4 * 65 * 4 + 48;    // mbarrier, TMEM base
constexpr uint32_t kSmemTrain = kSBar + 64;
constexpr uint32_t kSmemForward = kSmemTrain;         // same layout, training parts unused

// Tensor-memory columns: Z1 0-63, Z2 64-127, dW 128-207.  dH1 goes into
// Z2's columns: Z2 is read for the last time (the dZ2 epilogue) before the
// dH1 MMA is issued.  Training thus fits 256 columns, half of an SM's
// tensor memory, and two training blocks share an SM.
constexpr uint32_t kColZ1 = 0, kColZ2 = 64, kColDH1 = 64, kColDW = 128;

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ float warp_min(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(kFull, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

__device__ __forceinline__ void st_bf16(unsigned char *base, uint32_t off, float v) {
  *reinterpret_cast<__nv_bfloat16 *>(base + off) = __float2bfloat16_rn(v);
}

// --------------------------------------------------------------------------
// Instance-level helpers and features
// --------------------------------------------------------------------------

// Largest depot distance of every instance (feature scale): instance s owns
// rows seg_off[s] .. seg_off[s] + seg_n[s] of the coordinates; a block each.
__global__ void __launch_bounds__(256) k_depot_radius(const float2 *coords, const long long *seg_off,
                                                      const int *seg_n, int one_n, float *out) {
  __shared__ float s[8];
  if (seg_off) coords += seg_off[blockIdx.x];
  const int n = seg_n ? seg_n[blockIdx.x] : one_n;
  const float2 p0 = coords[0];
  float r = 0.f;
  for (int j = 1 + threadIdx.x; j <= n; j += blockDim.x) {
    const float dx = coords[j].x - p0.x, dy = coords[j].y - p0.y;
    r = fmaxf(r, sqrtf(dx * dx + dy * dy));
  }
  r = warp_max(r);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = r;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = fmaxf(r, s[w]);
    out[blockIdx.x] = r;
  }
}

// k-nearest candidate lists (k <= 32, empty slots 0), the same lists as the
// solver's (ties to the lower index).
__global__ void __launch_bounds__(256) k_prior_knn(const float2 *coords, int n, int k,
                                                   uint16_t *cand) {
  __shared__ unsigned long long s_buf[8][64];
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i <= n; i += warps) {
    const unsigned long long key = warp_knn(coords, n, k, i, lane, s_buf[threadIdx.x >> 5]);
    if (lane < k) cand[(size_t)i * k + lane] = (uint16_t)((key == ~0ull) ? 0 : (key & 0xffffffffu));
  }
}

// Features of candidate slot t (lane) of row i, c = cand[i][t]:
//   0  d(i,c) / largest candidate distance of the row
//   1  nearest candidate distance of the row / d(i,c)
//   2  t / 31 (rank in the row)
//   3  d(c,0) / R      (R = largest depot distance of the instance)
//   4  d(i,0) / R
//   5  demand(c) / capacity
//   6  cos of the angle between c - i and 0 - i (0 for the depot row)
//   7  1 if i is among c's candidates, else 0
// Empty slots get zeros; kv[i] = number of non-empty slots (a prefix).
// A warp per row, of one instance (seg_off null: rows 0 .. one_n) or of many
// packed one after another (rows first .. first + rows - 1 of all; feat and kv
// start at row `first`).
struct FeatureArgs {
  const float2 *coords;
  const int *demand;
  const uint16_t *cand;      // [rows][k]
  const float *radius;       // per instance
  const int *cap;            // capacity of instance s at cap[s cap_step] (seg_off given)
  int cap_step;
  float inv_cap;             // of the one instance
  const long long *seg_off;
  const int *seg_n;
  int count, one_n, k;
  long long first, rows;
  uint4 *feat;
  uint8_t *kv;
};

__global__ void __launch_bounds__(256) k_prior_features(FeatureArgs a) {
  const int lane = threadIdx.x & 31, k = a.k;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long g = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < a.rows;
       g += warps) {
    const long long row = a.first + g;
    int seg = 0;
    long long off = 0;
    if (a.seg_off) {
      int hi = a.count;  // last instance with seg_off <= row
      while (hi - seg > 1) {
        const int mid = (seg + hi) >> 1;
        if (__ldg(a.seg_off + mid) <= row) seg = mid; else hi = mid;
      }
      off = __ldg(a.seg_off + seg);
    }
    const float2 *coords = a.coords + off;
    const int *demand = a.demand + off;
    const uint16_t *cand = a.cand + off * k;
    const int i = (int)(row - off);
    const float inv_cap = a.seg_off ? 1.0f / (float)a.cap[(long long)seg * a.cap_step] : a.inv_cap;
    const float2 p0 = coords[0];
    const float inv_r = 1.0f / fmaxf(a.radius[seg], 1e-6f);
    const float2 pi = coords[i];
    const int c = (lane < k) ? (int)cand[(size_t)i * k + lane] : 0;
    const bool valid = c > 0;
    const float2 pc = valid ? coords[c] : pi;
    const float dx = pc.x - pi.x, dy = pc.y - pi.y;
    const float d = sqrtf(dx * dx + dy * dy);
    const float dmin = warp_min(valid ? d : FLT_MAX);
    const float dmax = warp_max(valid ? d : 0.f);
    const float ax = p0.x - pi.x, ay = p0.y - pi.y;
    const float di0 = sqrtf(ax * ax + ay * ay);
    const float bx = p0.x - pc.x, by = p0.y - pc.y;
    const float dc0 = sqrtf(bx * bx + by * by);
    float f[8];
    f[0] = d / fmaxf(dmax, 1e-6f);
    f[1] = dmin / fmaxf(d, 1e-6f);
    f[2] = (float)lane * (1.0f / 31.0f);
    f[3] = dc0 * inv_r;
    f[4] = di0 * inv_r;
    f[5] = (float)(valid ? demand[c] : 0) * inv_cap;
    f[6] = (i == 0) ? 0.f : (dx * ax + dy * ay) / fmaxf(d * di0, 1e-6f);
    int mutual = 0;
    if (valid)
      for (int s = 0; s < k; ++s) mutual |= (cand[(size_t)c * k + s] == i) ? 1 : 0;
    f[7] = (float)mutual;
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    if (valid) {
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t lo = __bfloat16_as_ushort(__float2bfloat16_rn(f[2 * q]));
        const uint32_t hi = __bfloat16_as_ushort(__float2bfloat16_rn(f[2 * q + 1]));
        w[q] = lo | (hi << 16);
      }
      out = make_uint4(w[0], w[1], w[2], w[3]);
    }
    a.feat[(size_t)g * kSlots + lane] = out;
    const unsigned vm = __ballot_sync(kFull, valid);
    if (lane == 0) a.kv[g] = (uint8_t)__popc(vm);
  }
}

// Slot of each elite successor in its row's candidate list (-1: absent).
__global__ void k_prior_slots(const int2 *pairs, long long count, const uint16_t *cand, int k,
                              int *slot) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= count) return;
  const int2 pr = pairs[p];
  int s = -1;
  for (int t = 0; t < k; ++t)
    if ((int)cand[(size_t)pr.x * k + t] == pr.y) {
      s = t;
      break;
    }
  slot[p] = s;
}

// --------------------------------------------------------------------------
// MLP on the tensor cores
// --------------------------------------------------------------------------

struct MlpArgs {
  const float *params;   // kParams FP32
  const uint4 *feat;     // [rows][32] edges, 8 BF16 each
  const uint8_t *kv;     // non-empty slots per row
  int tiles;
  // forward
  long long rows;
  float *scores;         // [rows][32]
  // training
  const int2 *examples;  // {feature row, target slot}
  const int *order;      // example ids of this minibatch
  int count;
  float inv_count;
  float *gpart;          // [grid][kGradStride] per-block partial gradients
  int *error;
};

// The feature row of one warp's edges in a tile (beyond the last tile or
// example: row 0, not live) and, in training, its target slot.
struct RowRef {
  long long row;
  int tgt;
  bool live;
};

template <bool TRAIN>
__device__ __forceinline__ RowRef row_ref(const MlpArgs &a, int tile, int warp) {
  RowRef r;
  if (TRAIN) {
    const int ex = tile * 4 + warp;
    r.live = ex < a.count;
    const int2 e2 = r.live ? a.examples[a.order[ex]] : make_int2(0, -1);
    r.row = e2.x;
    r.tgt = e2.y;
  } else {
    r.row = (long long)tile * 4 + warp;
    r.live = r.row < a.rows;
    if (!r.live) r.row = 0;
    r.tgt = -1;
  }
  return r;
}

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) |
         ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16);
}

// Four values of a table in shared memory, read where they are used: kept in
// registers over the tiles, b2 and w3 alone would take 128 of them.
__device__ __forceinline__ float4 lds4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}

// The same value, as one that is not known to stay the same: what is computed
// from it is computed where it is used, by the thread that issues the MMAs,
// instead of in registers of every thread over the tiles.
__device__ __forceinline__ uint32_t fresh(uint32_t v) {
  asm volatile("" : "+r"(v));
  return v;
}

template <bool TRAIN>
__global__ void __launch_bounds__(128, 2) k_prior_mlp(MlpArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char *sB1 = smem + kSB1, *sB2 = smem + kSB2;
  unsigned char *sdZ2 = smem + kSdZ2, *sdZ1 = smem + kSdZ1;
  float *s_b2 = reinterpret_cast<float *>(smem + kSF32);
  float *s_w3 = s_b2 + 64;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kSBar);
  uint32_t *s_tmem = reinterpret_cast<uint32_t *>(smem + kSBar + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr uint32_t kCols = TRAIN ? 256u : 128u;

  let_next_start();
  if (warp == 0) {
    umma::tmem_alloc(s_tmem, kCols);
    umma::tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  // Constant input 8 = 1 (layer-1 bias), inputs 9-15 = 0, for every edge.
#pragma unroll
  for (int b = 0; b < 2; ++b)
    *reinterpret_cast<uint4 *>(smem + kSA1 + b * kSHX + umma::kmajor_offset(tid, 8, 128)) =
        make_uint4(0x3F80u, 0u, 0u, 0u);
  // The first tile's rows: features and examples are fixed, so they are on
  // their way before this launch waits for the parameters' update.
  int tile = blockIdx.x;
  // now: the tile worked on; next: the one whose inputs are in fv (n_slots of
  // them); after: where the rows of the one behind it are.
  RowRef now = row_ref<TRAIN>(a, tile, warp), next = now;
  RowRef after = row_ref<TRAIN>(a, tile + gridDim.x, warp);
  int slots = 0, n_slots = next.live ? (int)a.kv[next.row] : 0;
  uint4 fv = a.feat[next.row * kSlots + lane];
  // The inputs of `next` into buffer b, and the request for those behind them.
  auto take_inputs = [&](uint32_t b) {
    *reinterpret_cast<uint4 *>(smem + kSA1 + b * kSHX + umma::kmajor_offset(tid, 0, 128)) =
        next.live && lane < n_slots ? fv : make_uint4(0u, 0u, 0u, 0u);
    now = next;
    slots = n_slots;
    next = after;
    n_slots = next.live ? (int)a.kv[next.row] : 0;
    fv = a.feat[next.row * kSlots + lane];
  };
  wait_for_previous();
  // Weights into their operand layouts (BF16), 8 along K at a time (16-byte
  // stores); biases of layers 2-3 in FP32.  All of them are asked for before
  // the first store, which the loads behind it could not be moved ahead of.
  const float *P = a.params;
  float w1[8];
  float4 w2[4][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int o = (tid + 128 * i) >> 4, f = tid & 15;
    w1[i] = f < 8 ? P[kW1 + o * 8 + f] : (f == 8 ? P[kB1 + o] : 0.f);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 *p = reinterpret_cast<const float4 *>(P + kW2) + 2 * (tid + 128 * i);
    w2[i][0] = p[0];
    w2[i][1] = p[1];
  }
  const float b2w3 = tid < 64 ? P[kB2 + tid] : P[kW3 + tid - 64], b3 = P[kB3];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    st_bf16(sB1, umma::kmajor_offset((tid + 128 * i) >> 4, tid & 15, 64), w1[i]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int o = (tid + 128 * i) >> 3, j = (tid & 7) * 8;
    const float4 lo = w2[i][0], hi = w2[i][1];
    *reinterpret_cast<uint4 *>(sB2 + umma::kmajor_offset(o, j, 64)) =
        make_uint4(bf16_pair(lo.x, lo.y), bf16_pair(lo.z, lo.w), bf16_pair(hi.x, hi.y),
                   bf16_pair(hi.z, hi.w));
  }
  s_b2[tid] = b2w3;  // b2, then w3
  umma::fence_async_smem();
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tm = *s_tmem;
  const uint32_t tl = tm + ((uint32_t)(warp * 32) << 16);  // this warp's lanes

  const uint32_t lbo128 = umma::kmajor_lbo(128), lbo64 = umma::kmajor_lbo(64);
  const uint32_t idesc64 = umma::idesc_bf16_f32(128, 64);
  // dH1 = dZ2 W2: W2 read along its rows; dW = [dZ2 dZ1]^T [H1 X]: both read
  // along their rows.
  const uint32_t idesc64t = idesc64 | umma::kTransposeB;
  const uint32_t idesc80t =
      umma::idesc_bf16_f32(128, 80) | umma::kTransposeA | umma::kTransposeB;
  const uint32_t aA1 = umma::smem_u32(smem + kSA1), aA2 = umma::smem_u32(smem + kSA2),
                 adZ2 = umma::smem_u32(sdZ2), aB1 = umma::smem_u32(sB1),
                 aB2 = umma::smem_u32(sB2), ab2 = umma::smem_u32(s_b2),
                 aw3 = umma::smem_u32(s_w3);

  float acc_w3[64];
#pragma unroll
  for (int j = 0; j < 64; ++j) acc_w3[j] = 0.f;
  float acc_loss = 0.f;
  uint32_t phase = 0;
  bool ok = true;
  int done = 0;

  // Z1 = X W1^T (+ b1 through the constant input)
  auto issue_z1 = [&](uint32_t b) {
    umma::mma_bf16(tm + kColZ1, umma::smem_desc(fresh(aA1 + b * kSHX), lbo128, 128),
                   umma::smem_desc(fresh(aB1), lbo64, 128), idesc64, 0u);
  };
  // Every thread waits for the group committed last; a wait that gives up is
  // noticed at the next barrier, which every thread still reaches.
  auto wait_group = [&]() {
    ok = mbar_wait_bounded(bar, phase, kPolls) && ok;
    phase ^= 1u;
    __syncwarp();
    umma::fence_after_sync();
  };
  auto operands_ready = [&]() {
    umma::fence_async_smem();
    umma::fence_before_sync();
    ok = __syncthreads_and(ok);
    return ok;
  };

  // The tensor cores' work of a tile hides behind its neighbours': a commit
  // covers every MMA that the thread issued before it.  Inference issues the next tile's Z1 with
  // this tile's Z2 (one wait per tile); training issues it with dH1, and does
  // not wait for dW, which ends before the next tile's Z2 (two waits per tile).
  // A stage reads its accumulator in one go: sixteen loads of 16 columns with a
  // wait behind each were most of a tile's latency (with four waits per tile
  // 25.7 us for 4096 examples, now 22.8: 8 us in all for the launch, the
  // weights and the partial sums, then 3.7 us for two tiles per SM, twice
  // what their instructions take to issue).  Two threads per edge, each with
  // half the units, took 26 us.
  if (tile < a.tiles) {
    take_inputs(0u);
    after = row_ref<TRAIN>(a, tile + 2 * gridDim.x, warp);
    operands_ready();
    if (tid == 0) {
      umma::fence_after_sync();
      issue_z1(0u);
      umma::commit(bar);
    }
    wait_group();
  }
  for (; tile < a.tiles; tile += gridDim.x) {
    const uint32_t buf = (uint32_t)done & 1u;
    unsigned char *sA2 = smem + kSA2 + buf * kSHX;
    const bool more = tile + (int)gridDim.x < a.tiles;
    const bool live = now.live, valid = live && lane < slots;
    const long long row = now.row;
    const int tgt = now.tgt;
    uint32_t pos_z1[2] = {0u, 0u};  // TRAIN: units with Z1 > 0
    if (!TRAIN) {
      take_inputs(buf ^ 1u);
      after = row_ref<TRAIN>(a, tile + 3 * gridDim.x, warp);
    }
    // H1 = relu(Z1) -> BF16 operand
    float z[64];
    umma::tmem_ld64(tl + kColZ1, z);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t w[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float lo = z[16 * q + 2 * i], hi = z[16 * q + 2 * i + 1];
        w[i] = bf16_pair(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
        if (TRAIN) {
          const int at = 16 * (q & 1) + 2 * i;
          pos_z1[q >> 1] |= (lo > 0.f ? 1u << at : 0u) | (hi > 0.f ? 2u << at : 0u);
        }
      }
      *reinterpret_cast<uint4 *>(sA2 + umma::kmajor_offset(tid, 16 * q, 128)) =
          make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4 *>(sA2 + umma::kmajor_offset(tid, 16 * q + 8, 128)) =
          make_uint4(w[4], w[5], w[6], w[7]);
    }
    if (!operands_ready()) break;
    // Z2 = H1 W2^T
    if (tid == 0) {
      umma::fence_after_sync();
      const uint64_t da = umma::smem_desc(fresh(aA2 + buf * kSHX), lbo128, 128);
      const uint64_t db = umma::smem_desc(fresh(aB2), lbo64, 128);
#pragma unroll
      for (int s = 0; s < 4; ++s)
        umma::mma_bf16(tm + kColZ2, da + 2 * s * (lbo128 >> 4), db + 2 * s * (lbo64 >> 4), idesc64,
                       s > 0 ? 1u : 0u);
      if (!TRAIN && more) issue_z1(buf ^ 1u);
      umma::commit(bar);
    }
    wait_group();
    if (TRAIN) {
      take_inputs(buf ^ 1u);
      after = row_ref<TRAIN>(a, tile + 3 * gridDim.x, warp);
    }
    // s = b3 + w3 . relu(Z2 + b2)
    float sc = b3;
    umma::tmem_ld64(tl + kColZ2, z);
#pragma unroll
    for (int j = 0; j < 64; j += 4) {
      const float4 b2 = lds4(ab2 + 4 * j), w3 = lds4(aw3 + 4 * j);
      z[j] = fmaxf(z[j] + b2.x, 0.f);
      z[j + 1] = fmaxf(z[j + 1] + b2.y, 0.f);
      z[j + 2] = fmaxf(z[j + 2] + b2.z, 0.f);
      z[j + 3] = fmaxf(z[j + 3] + b2.w, 0.f);
      sc += w3.x * z[j];
      sc += w3.y * z[j + 1];
      sc += w3.z * z[j + 2];
      sc += w3.w * z[j + 3];
    }
    if (!TRAIN) {
      if (live) a.scores[row * kSlots + lane] = sc;
    } else {
      // Softmax cross-entropy over the row's non-empty slots (one warp).
      const float mx = warp_max(valid ? sc : -FLT_MAX);
      const float ex = valid ? expf(sc - mx) : 0.f;
      const float sum = warp_sum(ex);
      float g = 0.f;
      if (valid && tgt >= 0) {
        g = (ex / sum - (lane == tgt ? 1.f : 0.f)) * a.inv_count;
        if (lane == tgt) acc_loss += (mx + logf(sum) - sc) * a.inv_count;
      }
      // dZ2 = g w3 relu'(Z2 + b2): operand of dH1 and of dW.
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          const int j = 16 * q + 2 * i;
          const float4 w3 = lds4(aw3 + 4 * j);
#pragma unroll
          for (int h = 0; h < 4; ++h) acc_w3[j + h] += g * z[j + h];
          w[i] = bf16_pair(z[j] > 0.f ? g * w3.x : 0.f, z[j + 1] > 0.f ? g * w3.y : 0.f);
          w[i + 1] = bf16_pair(z[j + 2] > 0.f ? g * w3.z : 0.f, z[j + 3] > 0.f ? g * w3.w : 0.f);
        }
        *reinterpret_cast<uint4 *>(sdZ2 + umma::kmajor_offset(tid, 16 * q, 128)) =
            make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4 *>(sdZ2 + umma::kmajor_offset(tid, 16 * q + 8, 128)) =
            make_uint4(w[4], w[5], w[6], w[7]);
      }
      if (!operands_ready()) break;
      // dH1 = dZ2 W2
      if (tid == 0) {
        umma::fence_after_sync();
        const uint64_t da = umma::smem_desc(fresh(adZ2), lbo128, 128);
        const uint64_t db = umma::smem_desc(fresh(aB2), 128, lbo64);
#pragma unroll
        for (int s = 0; s < 4; ++s)
          umma::mma_bf16(tm + kColDH1, da + 2 * s * (lbo128 >> 4), db + 2 * s * (128 >> 4),
                         idesc64t, s > 0 ? 1u : 0u);
        if (more) issue_z1(buf ^ 1u);
        umma::commit(bar);
      }
      wait_group();
      // dZ1 = dH1 relu'(Z1)
      umma::tmem_ld64(tl + kColDH1, z);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t m = pos_z1[q >> 1] >> (16 * (q & 1) + 2 * i);
          w[i] = bf16_pair(m & 1u ? z[16 * q + 2 * i] : 0.f,
                           m & 2u ? z[16 * q + 2 * i + 1] : 0.f);
        }
        *reinterpret_cast<uint4 *>(sdZ1 + umma::kmajor_offset(tid, 16 * q, 128)) =
            make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4 *>(sdZ1 + umma::kmajor_offset(tid, 16 * q + 8, 128)) =
            make_uint4(w[4], w[5], w[6], w[7]);
      }
      if (!operands_ready()) break;
      // dW += [dZ2 dZ1]^T [H1 X], accumulated over this block's tiles
      if (tid == 0) {
        umma::fence_after_sync();
        const uint64_t da = umma::smem_desc(fresh(adZ2), 128, lbo128);
        const uint64_t db = umma::smem_desc(fresh(aA2 + buf * kSHX), 128, lbo128);
#pragma unroll
        for (int s = 0; s < 8; ++s)
          umma::mma_bf16(tm + kColDW, da + 2 * s * (128 >> 4), db + 2 * s * (128 >> 4), idesc80t,
                         (done > 0 || s > 0) ? 1u : 0u);
      }
    }
    ++done;
  }
  if (TRAIN && ok && done > 0) {
    if (tid == 0) umma::commit(bar);
    wait_group();
  }
  umma::fence_before_sync();
  ok = __syncthreads_and(ok);
  umma::fence_after_sync();

  if (!ok) {
    // A wait gave up: wait (bounded) for the group still in flight, and for
    // what was issued behind it, before the tensor memory is released.
    mbar_wait_bounded(bar, phase ^ 1u, kPolls);
    if (tid == 0) umma::commit(bar);
    mbar_wait_bounded(bar, phase, kPolls);
    if (tid == 0) atomicOr(a.error, kErrStageTimeout);
  } else if (TRAIN && done > 0) {
    // This block's partial gradient, row blockIdx.x of gpart (summed in a
    // fixed order by k_prior_reduce: training is bit-reproducible).
    float *out = a.gpart + (size_t)blockIdx.x * kGradStride;
    // W2, b2 (rows 0-63) and W1, b1 (rows 64-127) from tensor memory.
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      float d[16];
      umma::tmem_ld16(tl + kColDW + 16 * q, d);
      umma::tmem_wait_ld();
      if (q < 4) {
        if (warp < 2) {
          float4 *o4 = reinterpret_cast<float4 *>(out + kW2 + tid * 64 + 16 * q);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            o4[i] = make_float4(d[4 * i], d[4 * i + 1], d[4 * i + 2], d[4 * i + 3]);
        }
      } else if (warp < 2) {
        out[kB2 + tid] = d[8];
      } else {
        float4 *o4 = reinterpret_cast<float4 *>(out + kW1 + (tid - 64) * 8);
        o4[0] = make_float4(d[0], d[1], d[2], d[3]);
        o4[1] = make_float4(d[4], d[5], d[6], d[7]);
        out[kB1 + tid - 64] = d[8];
      }
    }
    // w3 and the loss: warp sums, then the four warps in order.  The 64 sums
    // by halving: at each step a lane keeps half of its values and adds the
    // partner's (the sums of a butterfly over all 32 lanes, with 62 shuffles
    // instead of 320); lane L ends with values 2 rev(L) and 2 rev(L) + 1.
    float *s_red = reinterpret_cast<float *>(smem + kSRed);
    int at = 0;
#pragma unroll
    for (int o = 16, half = 32; o > 0; o >>= 1, half >>= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (j < half) {
          const float keep = up ? acc_w3[j + half] : acc_w3[j];
          const float give = up ? acc_w3[j] : acc_w3[j + half];
          acc_w3[j] = keep + __shfl_xor_sync(kFull, give, o);
        }
      }
      at += up ? half : 0;
    }
    s_red[warp * 65 + at] = acc_w3[0];
    s_red[warp * 65 + at + 1] = acc_w3[1];
    const float vl = warp_sum(acc_loss);
    if (lane == 0) s_red[warp * 65 + 64] = vl;
    __syncthreads();
    if (tid < 65) {
      const float v = s_red[tid] + s_red[65 + tid] + s_red[130 + tid] + s_red[195 + tid];
      if (tid < 64) out[kW3 + tid] = v;
      else out[kParams] = v;  // loss
    }
    // b3 is not trained: a constant added to every score of a row changes
    // neither the softmax nor the levels, and its gradient is identically 0.
    if (tid == 0) out[kB3] = 0.f;
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tm, kCols);
}

// Sum of the blocks' partial gradients in block order, into grad or (params
// given) taken as Adam's step; the loss goes to *loss.  A block takes 32
// parameters: all its threads bring the rows' values to shared memory at once
// by asynchronous copies, one warp adds them in order, so that training stays
// bit-reproducible.  It is bound by the latency of those copies and of the
// 296 dependent adds: 5.8 us (9.4 with 16 loads in flight per thread and the
// moments asked for behind the sum; one thread per parameter loading row after
// row, and the step in a launch of its own, took 15 + 4 us).
constexpr int kReduceThreads = 256;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__global__ void __launch_bounds__(kReduceThreads)
    k_prior_reduce(const float *gpart, int blocks, float *grad, float *loss, float *params,
                   float *m, float *v, float lr, float bc1, float bc2) {
  extern __shared__ __align__(16) float s_part[];  // [blocks][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  let_next_start();
  wait_for_previous();
  for (int e = threadIdx.x; e < blocks * 8; e += kReduceThreads) {
    const int r = e >> 3, col = blockIdx.x * 32 + 4 * (e & 7);
    if (col < kGradStride)
      cp_async16(smem_addr(s_part + r * 32 + 4 * (e & 7)), gpart + (size_t)r * kGradStride + col);
  }
  const bool mine = warp == 0 && i <= kParams;
  const bool step = mine && i < kParams && params;
  const float m0 = step ? m[i] : 0.f, v0 = step ? v[i] : 0.f, p0 = step ? params[i] : 0.f;
  cp_async_wait();
  __syncthreads();
  if (!mine) return;
  float g = 0.f;
#pragma unroll 16
  for (int r = 0; r < blocks; ++r) g += s_part[r * 32 + lane];
  if (i == kParams) {
    *loss += g;
    return;
  }
  if (!params) {
    grad[i] = g;
    return;
  }
  const float mi = 0.9f * m0 + 0.1f * g;
  const float vi = 0.999f * v0 + 0.001f * g * g;
  m[i] = mi;
  v[i] = vi;
  params[i] = p0 - lr * (mi / bc1) / (sqrtf(vi / bc2) + 1e-8f);
}

// Levels from scores: warp per row, L = min(4095, round(scale (s_max - s))).
// residual: the learned level is added to the plain level already in lvl
// (weights proportional to eta^beta exp(gamma s)).
__global__ void k_prior_levels(const float *scores, const uint8_t *kv, int rows, int k,
                               float scale, int residual, uint16_t *lvl) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const bool valid = lane < (int)kv[row];
  const float s = scores[(size_t)row * kSlots + lane];
  const float mx = warp_max(valid ? s : -FLT_MAX);
  if (lane < k) {
    int L = kThresholds;
    if (valid) {
      L = (int)fminf((float)kThresholds, rintf(scale * (mx - s)));
      if (residual) L = min(kThresholds, L + (int)lvl[(size_t)row * k + lane]);
    }
    lvl[(size_t)row * k + lane] = (uint16_t)L;
  }
}

// --------------------------------------------------------------------------
// Host side
// --------------------------------------------------------------------------

bool configure_mlp() {
  static int state = 0;  // 0 unknown, 1 ok, -1 failed
  if (state == 0) {
    cudaError_t e1 = cudaFuncSetAttribute(k_prior_mlp<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kSmemTrain);
    cudaError_t e2 = cudaFuncSetAttribute(k_prior_mlp<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)kSmemForward);
    state = (e1 == cudaSuccess && e2 == cudaSuccess) ? 1 : -1;
  }
  return state == 1;
}

}  // namespace prior
}  // namespace acob200

using namespace acob200;
using namespace acob200::prior;

struct aco_b200_prior {
  int device = 0;
  int num_sms = 148;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  float *d_params = nullptr, *d_m = nullptr, *d_v = nullptr, *d_grad = nullptr, *d_loss = nullptr;
  float *d_gpart = nullptr;  // [2 num_sms][kGradStride] partial gradients
  int *d_error = nullptr;
  int adam_step = 0;
  // training set
  long long rows = 0;
  uint4 *d_feat = nullptr;
  uint8_t *d_kv = nullptr;
  int2 *d_examples = nullptr;
  long long n_examples = 0;
  int *d_order = nullptr;
  // scratch of apply (one instance)
  long long s_rows = 0;
  uint4 *d_sfeat = nullptr;
  uint8_t *d_skv = nullptr;
  float *d_sscores = nullptr;
  float *d_radius = nullptr;
  float *d_radii = nullptr;  // of n_radii instances
  int n_radii = 0;

  void free_dataset() {
    cudaFree(d_feat);
    cudaFree(d_kv);
    cudaFree(d_examples);
    cudaFree(d_order);
    d_feat = nullptr;
    d_kv = nullptr;
    d_examples = nullptr;
    d_order = nullptr;
    rows = n_examples = 0;
  }
  void free_scratch() {
    cudaFree(d_sfeat);
    cudaFree(d_skv);
    cudaFree(d_sscores);
    d_sfeat = nullptr;
    d_skv = nullptr;
    d_sscores = nullptr;
    s_rows = 0;
  }
  ~aco_b200_prior() {
    cudaSetDevice(device);
    free_dataset();
    free_scratch();
    void *p[] = {d_params, d_m, d_v, d_grad, d_loss, d_error, d_radius, d_radii, d_gpart};
    for (void *q : p)
      if (q) cudaFree(q);
    if (own_stream && stream) cudaStreamDestroy(stream);
  }
};

#define PTRY(call)                                                           \
  do {                                                                       \
    cudaError_t err__ = (call);                                              \
    if (err__ != cudaSuccess) {                                              \
      fprintf(stderr, "aco_b200 prior: CUDA error %s at %s:%d\n",            \
              cudaGetErrorString(err__), __FILE__, __LINE__);                \
      return err__ == cudaErrorMemoryAllocation ? ACO_ERR_ALLOCATION         \
                                                : ACO_ERR_BACKEND;           \
    }                                                                        \
  } while (0)

namespace acob200 {
namespace prior {

static int ensure_scratch(aco_b200_prior *p, long long rows) {
  if (rows <= p->s_rows) return ACO_OK;
  p->free_scratch();
  PTRY(cudaMalloc(&p->d_sfeat, (size_t)rows * kSlots * sizeof(uint4)));
  PTRY(cudaMalloc(&p->d_skv, (size_t)rows));
  PTRY(cudaMalloc(&p->d_sscores, (size_t)rows * kSlots * sizeof(float)));
  p->s_rows = rows;
  return ACO_OK;
}

static int launch_forward(aco_b200_prior *p, const uint4 *feat, const uint8_t *kv, long long rows,
                          float *scores, cudaStream_t s) {
  if (!configure_mlp()) return ACO_ERR_BACKEND;
  MlpArgs a = {};
  a.params = p->d_params;
  a.feat = feat;
  a.kv = kv;
  a.rows = rows;
  a.scores = scores;
  a.tiles = (int)((rows + 3) / 4);
  a.error = p->d_error;
  const int grid = std::max(1, std::min(a.tiles, p->num_sms * 2));
  k_prior_mlp<false><<<grid, 128, kSmemForward, s>>>(a);
  PTRY(cudaGetLastError());
  return ACO_OK;
}

static int launch_feature_rows(aco_b200_prior *p, const FeatureArgs &a, cudaStream_t s) {
  const long long blocks = std::min<long long>((a.rows + 7) / 8, (long long)p->num_sms * 8);
  k_prior_features<<<(unsigned)blocks, 256, 0, s>>>(a);
  PTRY(cudaGetLastError());
  return ACO_OK;
}

static int launch_features(aco_b200_prior *p, const float2 *coords, const int *demand,
                           long long cap, int n, int k, const uint16_t *cand, uint4 *feat,
                           uint8_t *kv, cudaStream_t s) {
  k_depot_radius<<<1, 256, 0, s>>>(coords, nullptr, nullptr, n, p->d_radius);
  PTRY(cudaGetLastError());
  FeatureArgs a = {};
  a.coords = coords;
  a.demand = demand;
  a.cand = cand;
  a.radius = p->d_radius;
  a.inv_cap = 1.0f / (float)cap;
  a.one_n = n;
  a.k = k;
  a.rows = (long long)n + 1;
  a.feat = feat;
  a.kv = kv;
  return launch_feature_rows(p, a, s);
}

int learned_levels(aco_b200_prior *p, const float2 *coords, const int *demand, long long cap,
                   int n, int k, const uint16_t *cand, uint16_t *lvl, float gamma,
                   int residual, cudaStream_t s) {
  if (!p || k < 1 || k > kSlots || n < 1) return ACO_ERR_INVALID_INPUT;
  const long long rows = (long long)n + 1;
  int rc = ensure_scratch(p, rows);
  if (rc) return rc;
  rc = launch_features(p, coords, demand, cap, n, k, cand, p->d_sfeat, p->d_skv, s);
  if (rc) return rc;
  rc = launch_forward(p, p->d_sfeat, p->d_skv, rows, p->d_sscores, s);
  if (rc) return rc;
  const float scale = gamma * (float)kLevelsPerOctave / logf(2.0f);
  k_prior_levels<<<(unsigned)((rows + 7) / 8), 256, 0, s>>>(p->d_sscores, p->d_skv, (int)rows, k,
                                                           scale, residual, lvl);
  PTRY(cudaGetLastError());
  return ACO_OK;
}

// Levels of many packed instances, kChunkRows rows at a time (the scratch of
// features and scores stays below 44 MB).  One instance after another, four
// launches each, a batch of 128 took 3.1 ms, bound by their launches.
int learned_levels_multi(aco_b200_prior *p, const float2 *coords, const int *demand,
                         const int *cap, int cap_step, const long long *seg_off, const int *seg_n,
                         int count, long long rows, int k, const uint16_t *cand, uint16_t *lvl,
                         float gamma, cudaStream_t s) {
  if (!p || k < 1 || k > kSlots || count < 1 || rows < 2) return ACO_ERR_INVALID_INPUT;
  constexpr long long kChunkRows = 65536;
  int rc = ensure_scratch(p, std::min(rows, kChunkRows));
  if (rc) return rc;
  if (count > p->n_radii) {
    if (p->d_radii) cudaFree(p->d_radii);
    p->d_radii = nullptr;
    p->n_radii = 0;
    PTRY(cudaMalloc(&p->d_radii, (size_t)count * sizeof(float)));
    p->n_radii = count;
  }
  k_depot_radius<<<count, 256, 0, s>>>(coords, seg_off, seg_n, 0, p->d_radii);
  PTRY(cudaGetLastError());
  const float scale = gamma * (float)kLevelsPerOctave / logf(2.0f);
  for (long long first = 0; first < rows; first += kChunkRows) {
    FeatureArgs a = {};
    a.coords = coords;
    a.demand = demand;
    a.cand = cand;
    a.radius = p->d_radii;
    a.cap = cap;
    a.cap_step = cap_step;
    a.seg_off = seg_off;
    a.seg_n = seg_n;
    a.count = count;
    a.k = k;
    a.first = first;
    a.rows = std::min(kChunkRows, rows - first);
    a.feat = p->d_sfeat;
    a.kv = p->d_skv;
    rc = launch_feature_rows(p, a, s);
    if (rc) return rc;
    rc = launch_forward(p, p->d_sfeat, p->d_skv, a.rows, p->d_sscores, s);
    if (rc) return rc;
    k_prior_levels<<<(unsigned)((a.rows + 7) / 8), 256, 0, s>>>(
        p->d_sscores, p->d_skv, (int)a.rows, k, scale, 0, lvl + first * k);
    PTRY(cudaGetLastError());
  }
  return ACO_OK;
}

}  // namespace prior
}  // namespace acob200

extern "C" {

int aco_b200_prior_create(aco_b200_prior **out, int device) {
  if (!out) return ACO_ERR_INVALID_INPUT;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) {
    fprintf(stderr, "aco_b200 prior: no CUDA device %d\n", device);
    return ACO_ERR_BACKEND;
  }
  aco_b200_prior *p = new aco_b200_prior();
  p->device = device;
  cudaSetDevice(device);
  cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete p;
    return ACO_ERR_BACKEND;
  }
  p->own_stream = true;
  const size_t pb = (kParams + 3) / 4 * 16;
  if (cudaMalloc(&p->d_params, pb) != cudaSuccess || cudaMalloc(&p->d_m, pb) != cudaSuccess ||
      cudaMalloc(&p->d_v, pb) != cudaSuccess || cudaMalloc(&p->d_grad, pb) != cudaSuccess ||
      cudaMalloc(&p->d_loss, 16) != cudaSuccess || cudaMalloc(&p->d_error, 16) != cudaSuccess ||
      cudaMalloc(&p->d_radius, 16) != cudaSuccess ||
      cudaMalloc(&p->d_gpart, (size_t)2 * p->num_sms * kGradStride * sizeof(float)) !=
          cudaSuccess) {
    delete p;
    return ACO_ERR_ALLOCATION;
  }
  cudaMemset(p->d_params, 0, pb);
  cudaMemset(p->d_m, 0, pb);
  cudaMemset(p->d_v, 0, pb);
  cudaMemset(p->d_grad, 0, pb);
  cudaMemset(p->d_loss, 0, 16);
  cudaMemset(p->d_error, 0, 16);
  if (!configure_mlp()) {
    fprintf(stderr, "aco_b200 prior: cannot configure the MLP kernels\n");
    delete p;
    return ACO_ERR_BACKEND;
  }
  *out = p;
  return ACO_OK;
}

int aco_b200_prior_destroy(aco_b200_prior *p) {
  delete p;
  return ACO_OK;
}

int aco_b200_prior_set_stream(aco_b200_prior *p, void *stream) {
  if (!p) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  if (p->own_stream && p->stream) cudaStreamDestroy(p->stream);
  p->own_stream = false;
  p->stream = (cudaStream_t)stream;
  if (!p->stream) {
    if (cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking) != cudaSuccess)
      return ACO_ERR_BACKEND;
    p->own_stream = true;
  }
  return ACO_OK;
}

int aco_b200_prior_init(aco_b200_prior *p, unsigned int seed) {
  if (!p) return ACO_ERR_INVALID_INPUT;
  // He-normal weights, zero biases (std::mt19937 + Box-Muller, so the
  // values are the same on every platform).
  std::mt19937 rng(seed);
  auto normal = [&rng]() {
    const double u1 = (rng() + 1.0) / 4294967297.0, u2 = (rng() + 1.0) / 4294967297.0;
    return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
  };
  std::vector<float> h(kParams, 0.f);
  for (int i = 0; i < 512; ++i) h[kW1 + i] = (float)(normal() * std::sqrt(2.0 / 8.0));
  for (int i = 0; i < 4096; ++i) h[kW2 + i] = (float)(normal() * std::sqrt(2.0 / 64.0));
  for (int i = 0; i < 64; ++i) h[kW3 + i] = (float)(normal() * std::sqrt(1.0 / 64.0));
  return aco_b200_prior_set_params(p, h.data(), kParams);
}

int aco_b200_prior_set_params(aco_b200_prior *p, const float *params, int count) {
  if (!p || !params || count != kParams) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  const size_t pb = (size_t)kParams * sizeof(float);
  PTRY(cudaMemcpy(p->d_params, params, pb, cudaMemcpyHostToDevice));
  PTRY(cudaMemset(p->d_m, 0, pb));
  PTRY(cudaMemset(p->d_v, 0, pb));
  PTRY(cudaMemset(p->d_grad, 0, pb));
  p->adam_step = 0;
  return ACO_OK;
}

int aco_b200_prior_get_params(aco_b200_prior *p, float *params, int count) {
  if (!p || !params || count != kParams) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  PTRY(cudaStreamSynchronize(p->stream));
  PTRY(cudaMemcpy(params, p->d_params, (size_t)kParams * sizeof(float), cudaMemcpyDeviceToHost));
  return ACO_OK;
}

int aco_b200_prior_load(aco_b200_prior *p, const char *path) {
  if (!p || !path) return ACO_ERR_INVALID_INPUT;
  FILE *f = fopen(path, "rb");
  if (!f) return ACO_ERR_INVALID_INPUT;
  std::vector<float> h(kParams);
  const size_t got = fread(h.data(), sizeof(float), kParams, f);
  const bool extra = fgetc(f) != EOF;
  fclose(f);
  if (got != (size_t)kParams || extra) return ACO_ERR_INVALID_INPUT;
  return aco_b200_prior_set_params(p, h.data(), kParams);
}

int aco_b200_prior_save(aco_b200_prior *p, const char *path) {
  if (!p || !path) return ACO_ERR_INVALID_INPUT;
  std::vector<float> h(kParams);
  int rc = aco_b200_prior_get_params(p, h.data(), kParams);
  if (rc) return rc;
  FILE *f = fopen(path, "wb");
  if (!f) return ACO_ERR_INVALID_INPUT;
  const size_t put = fwrite(h.data(), sizeof(float), kParams, f);
  fclose(f);
  return put == (size_t)kParams ? ACO_OK : ACO_ERR_BACKEND;
}

int aco_b200_prior_set_dataset(aco_b200_prior *p, const aco_b200_prior_dataset *d,
                               long long *n_examples) {
  if (!p || !d || d->count < 1 || !d->n || !d->K || !d->capacity || !d->x || !d->y || !d->nodes ||
      !d->lens)
    return ACO_ERR_INVALID_INPUT;
  const int k = d->cand_k > 0 ? d->cand_k : kSlots;
  if (k > kSlots) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  cudaStream_t s = p->stream;
  // Offsets and validation.
  std::vector<long long> node_off(d->count + 1, 0), route_off(d->count + 1, 0),
      len_off(d->count + 1, 0);
  for (int i = 0; i < d->count; ++i) {
    const int n = d->n[i], K = d->K[i];
    if (n < 2 || n > 65534 || K < 1 || d->capacity[i] < 1) return ACO_ERR_INVALID_INPUT;
    node_off[i + 1] = node_off[i] + n + 1;
    len_off[i + 1] = len_off[i] + K;
    long long tot = 0;
    for (int v = 0; v < K; ++v) {
      const int L = d->lens[len_off[i] + v];
      if (L < 2) return ACO_ERR_INVALID_INPUT;
      tot += L;
    }
    route_off[i + 1] = route_off[i] + tot;
  }
  const long long rows = node_off[d->count];
  // Elite successor pairs (row, successor): depot -> first customer, and
  // both directions of every customer-customer arc.
  std::vector<int2> pairs;
  for (int i = 0; i < d->count; ++i) {
    const int n = d->n[i];
    long long off = route_off[i];
    for (int v = 0; v < d->K[i]; ++v) {
      const int L = d->lens[len_off[i] + v];
      const int *r = d->nodes + off;
      if (r[0] != 0 || r[L - 1] != 0) return ACO_ERR_INVALID_INPUT;
      for (int t = 1; t + 1 < L; ++t)
        if (r[t] < 1 || r[t] > n) return ACO_ERR_INVALID_INPUT;
      if (L > 2) pairs.push_back(make_int2((int)(node_off[i] + 0), r[1]));
      for (int t = 1; t + 2 < L; ++t) {
        pairs.push_back(make_int2((int)(node_off[i] + r[t]), r[t + 1]));
        pairs.push_back(make_int2((int)(node_off[i] + r[t + 1]), r[t]));
      }
      off += L;
    }
  }
  if (rows > 0x7fffffffLL) return ACO_ERR_INVALID_INPUT;
  p->free_dataset();
  // Per-instance device work: coordinates, candidate lists, features.
  float2 *d_xy = nullptr;
  int *d_dem = nullptr;
  uint16_t *d_cand = nullptr;
  int2 *d_pairs = nullptr;
  int *d_slot = nullptr;
  int rc = ACO_OK;
  auto fail = [&](int code) {
    cudaFree(d_xy);
    cudaFree(d_dem);
    cudaFree(d_cand);
    cudaFree(d_pairs);
    cudaFree(d_slot);
    return code;
  };
  std::vector<float2> xy(rows);
  std::vector<int> dem(rows);
  for (int i = 0; i < d->count; ++i)
    for (long long j = node_off[i]; j < node_off[i + 1]; ++j) {
      xy[j] = make_float2(d->x[j], d->y[j]);
      dem[j] = d->demand ? d->demand[j] : (j == node_off[i] ? 0 : 1);
    }
  if (cudaMalloc(&d_xy, rows * sizeof(float2)) != cudaSuccess ||
      cudaMalloc(&d_dem, rows * sizeof(int)) != cudaSuccess ||
      cudaMalloc(&d_cand, rows * k * sizeof(uint16_t)) != cudaSuccess ||
      cudaMalloc(&p->d_feat, rows * kSlots * sizeof(uint4)) != cudaSuccess ||
      cudaMalloc(&p->d_kv, rows) != cudaSuccess)
    return fail(ACO_ERR_ALLOCATION);
  if (cudaMemcpyAsync(d_xy, xy.data(), rows * sizeof(float2), cudaMemcpyHostToDevice, s) ||
      cudaMemcpyAsync(d_dem, dem.data(), rows * sizeof(int), cudaMemcpyHostToDevice, s))
    return fail(ACO_ERR_BACKEND);
  for (int i = 0; i < d->count && rc == ACO_OK; ++i) {
    const int n = d->n[i];
    const int ki = std::min(k, n);
    // Candidate lists of length k (the instance's own list is shorter
    // only when n < k; empty slots stay 0).
    if (ki < k) cudaMemsetAsync(d_cand + node_off[i] * k, 0, (size_t)(n + 1) * k * sizeof(uint16_t), s);
    int blocks = std::min((n + 1 + 7) / 8, p->num_sms * 16);
    k_prior_knn<<<blocks, 256, 0, s>>>(d_xy + node_off[i], n, k, d_cand + node_off[i] * k);
    if (cudaGetLastError() != cudaSuccess) rc = ACO_ERR_BACKEND;
    if (rc == ACO_OK)
      rc = launch_features(p, d_xy + node_off[i], d_dem + node_off[i], d->capacity[i], n, k,
                           d_cand + node_off[i] * k, p->d_feat + node_off[i] * kSlots,
                           p->d_kv + node_off[i], s);
  }
  if (rc) return fail(rc);
  // Slots of the successors; pairs whose successor is not a candidate drop.
  const long long np = (long long)pairs.size();
  std::vector<int> slot(np);
  if (np > 0) {
    if (cudaMalloc(&d_pairs, np * sizeof(int2)) != cudaSuccess ||
        cudaMalloc(&d_slot, np * sizeof(int)) != cudaSuccess)
      return fail(ACO_ERR_ALLOCATION);
    if (cudaMemcpyAsync(d_pairs, pairs.data(), np * sizeof(int2), cudaMemcpyHostToDevice, s))
      return fail(ACO_ERR_BACKEND);
    k_prior_slots<<<(unsigned)((np + 255) / 256), 256, 0, s>>>(d_pairs, np, d_cand, k, d_slot);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(slot.data(), d_slot, np * sizeof(int), cudaMemcpyDeviceToHost, s) ||
        cudaStreamSynchronize(s))
      return fail(ACO_ERR_BACKEND);
  } else if (cudaStreamSynchronize(s)) {
    return fail(ACO_ERR_BACKEND);
  }
  std::vector<int2> ex;
  ex.reserve(np);
  for (long long q = 0; q < np; ++q)
    if (slot[q] >= 0) ex.push_back(make_int2(pairs[q].x, slot[q]));
  fail(ACO_OK);  // frees the temporaries
  p->rows = rows;
  p->n_examples = (long long)ex.size();
  if (p->n_examples > 0) {
    PTRY(cudaMalloc(&p->d_examples, ex.size() * sizeof(int2)));
    PTRY(cudaMalloc(&p->d_order, ex.size() * sizeof(int)));
    PTRY(cudaMemcpy(p->d_examples, ex.data(), ex.size() * sizeof(int2), cudaMemcpyHostToDevice));
  }
  if (n_examples) *n_examples = p->n_examples;
  return ACO_OK;
}

// Gradient of the mean loss over `count` examples listed at order: the
// tensor-core kernel writes one partial row per block, k_prior_reduce sums
// them and adds the loss to *d_loss; step > 0: Adam's step number `step` on
// the parameters, else the gradient into d_grad.  first: the launch follows
// copies (the examples' order), which it must not overtake.
static int run_gradient(aco_b200_prior *p, const int *order, int count, int step, float lr,
                        bool first, cudaStream_t s) {
  MlpArgs a = {};
  a.params = p->d_params;
  a.feat = p->d_feat;
  a.kv = p->d_kv;
  a.examples = p->d_examples;
  a.order = order;
  a.count = count;
  a.inv_count = 1.0f / (float)count;
  a.gpart = p->d_gpart;
  a.error = p->d_error;
  a.tiles = (count + 3) / 4;
  // Two training blocks per SM (256 tensor-memory columns and 84 KB of shared
  // memory each): one block's MMA runs while the other's epilogue does.
  const int grid = std::max(1, std::min(a.tiles, p->num_sms * 2));
  if (first) {
    k_prior_mlp<true><<<grid, 128, kSmemTrain, s>>>(a);
    PTRY(cudaGetLastError());
  } else {
    PTRY(launch_after(k_prior_mlp<true>, grid, 128, kSmemTrain, s, a));
  }
  const float bc1 = 1.0f - powf(0.9f, (float)step), bc2 = 1.0f - powf(0.999f, (float)step);
  PTRY(launch_after(k_prior_reduce, (kParams + 1 + 31) / 32, kReduceThreads,
                    (size_t)grid * 32 * sizeof(float), s, (const float *)p->d_gpart, grid, p->d_grad, p->d_loss,
                    step > 0 ? p->d_params : nullptr, p->d_m, p->d_v, lr, bc1, bc2));
  return ACO_OK;
}

static int check_error(aco_b200_prior *p) {
  int err = 0;
  PTRY(cudaMemcpy(&err, p->d_error, sizeof(int), cudaMemcpyDeviceToHost));
  if (err) {
    fprintf(stderr, "aco_b200 prior: device error flag 0x%x\n", err);
    return ACO_ERR_BACKEND;
  }
  return ACO_OK;
}

int aco_b200_prior_gradient(aco_b200_prior *p, const int *examples, int count, float *grad,
                            float *loss) {
  if (!p || !examples || count < 1 || !grad || p->n_examples < 1) return ACO_ERR_INVALID_INPUT;
  for (int i = 0; i < count; ++i)
    if (examples[i] < 0 || examples[i] >= p->n_examples) return ACO_ERR_INVALID_INPUT;
  if (count > p->n_examples) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  cudaStream_t s = p->stream;
  PTRY(cudaMemcpyAsync(p->d_order, examples, count * sizeof(int), cudaMemcpyHostToDevice, s));
  PTRY(cudaMemsetAsync(p->d_loss, 0, sizeof(float), s));
  int rc = run_gradient(p, p->d_order, count, 0, 0.f, true, s);
  if (rc) return rc;
  PTRY(cudaStreamSynchronize(s));
  rc = check_error(p);
  if (rc) return rc;
  PTRY(cudaMemcpy(grad, p->d_grad, kParams * sizeof(float), cudaMemcpyDeviceToHost));
  if (loss) PTRY(cudaMemcpy(loss, p->d_loss, sizeof(float), cudaMemcpyDeviceToHost));
  return ACO_OK;
}

int aco_b200_prior_train(aco_b200_prior *p, int epochs, int batch, float lr, unsigned int seed,
                         float *epoch_loss) {
  if (!p || epochs < 0 || batch < 4 || !(lr >= 0.f) || p->n_examples < 1)
    return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  cudaStream_t s = p->stream;
  const long long N = p->n_examples;
  std::vector<int> order(N);
  std::mt19937 rng(seed);
  for (int e = 0; e < epochs; ++e) {
    for (long long i = 0; i < N; ++i) order[i] = (int)i;
    for (long long i = N - 1; i > 0; --i) {
      const long long j = (long long)(rng() % (unsigned long long)(i + 1));
      std::swap(order[i], order[j]);
    }
    PTRY(cudaMemcpyAsync(p->d_order, order.data(), N * sizeof(int), cudaMemcpyHostToDevice, s));
    PTRY(cudaMemsetAsync(p->d_loss, 0, sizeof(float), s));
    int steps = 0;
    for (long long b0 = 0; b0 < N; b0 += batch, ++steps) {
      const int cnt = (int)std::min<long long>(batch, N - b0);
      p->adam_step += 1;
      int rc = run_gradient(p, p->d_order + b0, cnt, p->adam_step, lr, b0 == 0, s);
      if (rc) return rc;
    }
    float l = 0.f;
    PTRY(cudaMemcpyAsync(&l, p->d_loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    PTRY(cudaStreamSynchronize(s));
    int rc = check_error(p);
    if (rc) return rc;
    if (epoch_loss) epoch_loss[e] = steps > 0 ? l / (float)steps : 0.f;
  }
  return ACO_OK;
}

long long aco_b200_prior_num_examples(aco_b200_prior *p) { return p ? p->n_examples : -1; }

int aco_b200_prior_get_examples(aco_b200_prior *p, int *rows_slots, long long count) {
  if (!p || !rows_slots || count < 0 || count > p->n_examples) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  if (count == 0) return ACO_OK;
  PTRY(cudaMemcpy(rows_slots, p->d_examples, count * sizeof(int2), cudaMemcpyDeviceToHost));
  return ACO_OK;
}

int aco_b200_prior_get_rows(aco_b200_prior *p, long long first, int count, uint16_t *features,
                            uint8_t *kv, float *scores) {
  if (!p || first < 0 || count < 1 || first + count > p->rows) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(p->device);
  cudaStream_t s = p->stream;
  if (features)
    PTRY(cudaMemcpy(features, p->d_feat + first * kSlots, (size_t)count * kSlots * sizeof(uint4),
                    cudaMemcpyDeviceToHost));
  if (kv) PTRY(cudaMemcpy(kv, p->d_kv + first, (size_t)count, cudaMemcpyDeviceToHost));
  if (scores) {
    int rc = ensure_scratch(p, count);
    if (rc) return rc;
    rc = launch_forward(p, p->d_feat + first * kSlots, p->d_kv + first, count, p->d_sscores, s);
    if (rc) return rc;
    PTRY(cudaStreamSynchronize(s));
    rc = check_error(p);
    if (rc) return rc;
    PTRY(cudaMemcpy(scores, p->d_sscores, (size_t)count * kSlots * sizeof(float),
                    cudaMemcpyDeviceToHost));
  }
  return ACO_OK;
}

}  // extern "C"
