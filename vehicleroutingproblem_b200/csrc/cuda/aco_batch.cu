// aco_batch.cu -- many independent instances in one persistent launch.
//
// Each block pulls instances from a queue and runs every epoch of an
// instance by itself: per-epoch weights into shared memory, the ants'
// construction (4 or 8 lanes per ant, a whole colony at a time), iteration/
// global best and stop rules, evaporation and deposit on the candidate cells
// of the pheromone -- phases separated by __syncthreads only, so the whole
// batch is one launch with no grid-wide synchronisation and no host round
// trip.  Instance i is solved exactly as
// the single-instance path solves it with seed + i (same draws, same rules,
// same device math), which the tests check route for route.
#include "aco_internal.cuh"
#include "aco_prior_internal.h"

extern "C" {
#include "aco.h"
#include "aco_b200.h"
}

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <vector>

using namespace acob200;

namespace {

struct BatchInst {
  int n, K, cap, total_demand;
  long long node_off;   // coords / demand / rows (cand, lvl at node_off * k)
  long long route_off;  // m * (n + 2K) ints
  long long lens_off;   // m * K ints
  long long gbest_off;  // n + 2K ints
  long long gblens_off; // K ints
  long long rep_off;    // m * n ints (repair scratch)
};

struct BatchArgs {
  const BatchInst *inst;
  const int *order;          // queue order of instance ids
  int count;
  int m, k;
  int epochs, stagnation;
  double min_rel;
  float Qs, log_min, log_step;
  uint8_t delta, q_tau0, pad0, pad1;
  uint32_t seed;
  const float2 *coords;
  const int *demand;
  const uint16_t *cand, *lvl;
  const uint16_t *tier;      // [rows][kTierLen]: ranks k+1 .. k+64 (fallback)
  const int32_t *A;
  const uint32_t *lut;
  uint8_t *tau;              // [rows][2 kMaxCand] levels where they do not fit a block
  int *routes, *lens, *loads, *rep, *last;
  double *cost;
  int *feasible, *steps;
  int *gbest_nodes, *gbest_lens;
  double *out_cost;
  int *out_epochs;
  unsigned long long *out_steps;
  unsigned int *queue;       // work counter (scratch, zeroed before launch)
};

__host__ __device__ inline uint32_t pad16u(uint32_t b) { return (b + 15u) & ~15u; }

// Which launch shapes and instance sizes the entry points accept: a bound of
// their own (with batch_v_for's n <= 2046), the same whatever shared memory the
// launch takes (batch_shape).
inline uint32_t shape_bytes(int max_rows, int k, int ants_per_block, int threads, int max_K) {
  const uint32_t r = (uint32_t)max_rows;
  return 2u * pad16u(r * k * 2) + pad16u(r * k * 4) + pad16u(r * 8) + pad16u(r * 4) + 2048u +
         (uint32_t)ants_per_block * 512u + pad16u((uint32_t)(threads / 32) * 16 + 64) +
         pad16u((uint32_t)(max_K + 1) * 4) + 64u;
}

constexpr int kBatchThreads = 512;  // per block at most
constexpr int kSlotsPerLane = 4;    // candidates per lane

// The launch: an ant takes lpa lanes with 4 candidate slots each (rows are
// padded to S = 4 ceil(k/4) slots), `round` ants of an instance are built at
// a time.  Offsets are bytes of dynamic shared memory.
struct BatchShape {
  int lpa, S, elem, threads, round;
  int tau_smem;              // levels in shared memory (else BatchArgs::tau)
  uint32_t off_lut, off_cand, off_w, off_coords, off_tau, off_el0, off_el, off_draw, off_red;
  uint32_t el_bytes;         // one ant's elements or bitmap
  uint32_t el0_bytes;        // the elements of an unserved instance; with bitmaps, the demands
  uint32_t total;
};

BatchShape batch_shape(int max_rows, int max_n, int k, int elem, int round, bool tau_smem) {
  BatchShape s = {};
  s.lpa = k <= 16 ? 4 : 8;
  s.S = (k + 3) & ~3;
  s.elem = elem;
  s.round = round;
  s.threads = (round * s.lpa + 31) & ~31;
  if (s.threads < 128) s.threads = 128;
  s.tau_smem = tau_smem ? 1 : 0;
  s.el_bytes = unserved_bytes(max_n, elem);
  s.el0_bytes = elem_is_bits(elem) ? unserved_bytes(max_n, 4) : s.el_bytes;
  const uint32_t r = (uint32_t)max_rows, S = (uint32_t)s.S;
  uint32_t o = 16;  // zeros, for lanes without candidates
  o += 1024;        // tau levels
  s.off_lut = o; o += 1024;
  s.off_cand = o; o += pad16u(r * S * 2);
  s.off_w = o; o += r * S * 4;
  s.off_coords = o; o += pad16u(r * 8);
  s.off_tau = o; o += tau_smem ? pad16u(r * S * 2) : 0u;
  s.off_el0 = o; o += s.el0_bytes;
  s.off_el = o; o += (uint32_t)round * s.el_bytes;
  s.off_draw = o; o += (uint32_t)round * 32u * (uint32_t)s.lpa;
  // per warp: 32 words of scratch; then the reductions
  s.off_red = o; o += (uint32_t)(s.threads / 32) * (128u + 16u);
  s.total = o;
  return s;
}

// One instance's tables as its block sees them.
template <int E>
struct BatchTables {
  const uint16_t *cand;      // [rows][S]
  const uint32_t *w;         // [rows][S]
  const float2 *coords;
  const uint16_t *tier;      // [rows][kTierLen] or null
  int S;
};

// Smallest instance whose fallback looks in the tier lists before it scans
// every node: a scan by the whole warp takes n/64 loads and compares per lane
// against one row's way from L2 (512-instance batch, 100 epochs: 47.5 ms with
// the lists from n=64 or 256 on, 55.9 ms from 512 on; below 128 the scan is
// two batches).
constexpr int kBatchTierMinCustomers = 128;

// Nearest eligible customer of one ant by the scan of every node, made by the
// whole warp (all arguments but lane are the warp's).  0 if none.
template <int E>
__device__ __noinline__ int coop_scan(const float2 *coords, Unserved<E> us, int n, int cur,
                                      uint32_t lim, int lane) {
  uint32_t best_h;
  const float2 pc = coords[cur];
  const uint32_t best_n = scan_pairs<false, E, 2>(coords, us, n, pc, lim, lane, &best_h);
  const uint32_t mh = __reduce_min_sync(kFull, best_h);
  const uint32_t mn = __reduce_min_sync(kFull, best_h == mh ? best_n : 0xffffffffu);
  return mh == 0xffffffffu ? 0 : (int)mn;
}

// The first eligible node of a tier row, which lane holds two ranks of; 0
// when the row lists every remaining customer and none is eligible, -1 when
// it is full and none is.
template <int E>
__device__ __forceinline__ int coop_tier(uint32_t two, const Unserved<E> &us, uint32_t lim) {
  const int n0 = (int)(two & 0xffffu), n1 = (int)(two >> 16);
  const bool ok0 = us.get(n0) <= lim, ok1 = us.get(n1) <= lim;
  const unsigned m = __ballot_sync(kFull, ok0 || ok1);
  const int at = m ? __ffs(m) - 1 : 31;
  const int node = __shfl_sync(kFull, m && ok0 ? n0 : n1, at);
  return m || node == 0 ? node : -1;
}

// Backward repair of one ant by the whole warp (aco_sequential.c:659-680, as
// in build_ant of aco_kernels.cu): from the last vehicle down, the nearest
// customers that fit are appended; then the compact route is laid out again
// in place.  left customers are unserved; returns how many of them were
// added.  With at most 32 of them each lane holds one (ascending), and no
// search looks at another node.
template <int E>
__device__ __noinline__ int coop_repair(const float2 *coords, Unserved<E> us, int n, int K,
                                        int cap, int pos, int left, int *route, int *lens,
                                        const int *loads, const int *last, int *rep,
                                        int *scratch, int lane) {
  const bool few = left <= 32;
  int mine = 0;
  uint32_t mdem = Unserved<E>::kVisited;
  float2 mp = make_float2(0.f, 0.f);
  if (few) {
    int found = 0;
    for (int b = 0; b <= n; b += 32) {
      const int node = min(b + lane, n);
      const bool open = b + lane <= n && us.get(node) != Unserved<E>::kVisited;
      const unsigned m = __ballot_sync(kFull, open);
      if (open) scratch[found + __popc(m & ((1u << lane) - 1u))] = node;
      found += __popc(m);
    }
    __syncwarp();
    if (lane < left) {
      mine = scratch[lane];
      mdem = us.get(mine);
      mp = coords[mine];
    }
    __syncwarp();
    rep = scratch;
  }
  int nrep = 0;
  const int top = (K - 1) & ~31;
  int cnt_top = 0, len_top = 0;
  for (int g = top; g >= 0; g -= 32) {
    const bool in = g + lane < K;
    const int len_l = in ? lens[g + lane] : 0, load_l = in ? loads[g + lane] : 0;
    const int last_l = in ? last[g + lane] : 0;
    int cnt_l = 0;
    for (int v = min(K - 1, g + 31); v >= g && left > 0; --v) {
      int cur = __shfl_sync(kFull, last_l, v & 31), load = __shfl_sync(kFull, load_l, v & 31);
      int cnt = 0;
      while (left > 0 && load < cap) {
        const uint32_t lim = us.limit(cap - load);
        int next;
        uint32_t dn;
        if (few) {
          const uint32_t h =
              mdem <= lim ? __float_as_uint(dist2f(coords[cur], mp)) : 0xffffffffu;
          const uint32_t mh = __reduce_min_sync(kFull, h);
          if (mh == 0xffffffffu) break;
          const int src = __ffs(__ballot_sync(kFull, h == mh)) - 1;
          next = __shfl_sync(kFull, mine, src);
          dn = __shfl_sync(kFull, mdem, src);
          if (lane == src) mdem = Unserved<E>::kVisited;
        } else {
          next = coop_scan<E>(coords, us, n, cur, lim, lane);
          if (next <= 0) break;
          dn = us.get(next);
          __syncwarp();
          us.mark(next);
          __syncwarp();
        }
        if (lane == 0) rep[nrep + cnt] = next;
        ++cnt;
        load += (int)dn;
        --left;
        cur = next;
      }
      if (lane == (v & 31)) cnt_l = cnt;
      nrep += cnt;
    }
    // The additions of a lower group wait in `last`, which it has read.
    if (g == top) {
      cnt_top = cnt_l;
      len_top = len_l;
    } else if (in) {
      const_cast<int *>(last)[g + lane] = cnt_l;
    }
  }
  __syncwarp();
  int off_total = pos, add_after = 0, shift = nrep;
  for (int g = top; g >= 0 && shift > 0; g -= 32) {
    const bool in = g + lane < K;
    const int len_l = g == top ? len_top : (in ? lens[g + lane] : 0);
    const int cnt_l = g == top ? cnt_top : (in ? last[g + lane] : 0);
    if (in && cnt_l > 0) lens[g + lane] = len_l + cnt_l;
    for (int v = min(K - 1, g + 31); v >= g && shift > 0; --v) {
      const int len_v = __shfl_sync(kFull, len_l, v & 31);
      const int cnt = __shfl_sync(kFull, cnt_l, v & 31);
      off_total -= len_v;
      shift -= cnt;  // now: additions of vehicles < v
      const int new_off = off_total + shift, main_len = len_v - 1;
      if (shift > 0) {
        // From the end, 256 entries at a time with their loads in flight.
        for (int t0 = (main_len - 1) & ~255; t0 >= 0; t0 -= 256) {
          int x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int t = t0 + 32 * i + lane;
            x[i] = t < main_len ? route[off_total + t] : 0;
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int t = t0 + 32 * i + lane;
            if (t < main_len) route[new_off + t] = x[i];
          }
          __syncwarp();
        }
      }
      for (int j = lane; j < cnt; j += 32) route[new_off + main_len + j] = rep[add_after + j];
      if (lane == 0) route[new_off + main_len + cnt] = 0;
      __syncwarp();
      add_after += cnt;
    }
  }
  return nrep;
}

// The 4 LPA draws from number d on of an ant into its ring of 8 LPA words
// (each in the upper 24 bits, or 1 for a draw of 0: see next_draws in
// aco_kernels.cu); lane l computes one Philox block.
template <int LPA>
__device__ __forceinline__ void ring_fill(uint32_t ring, uint32_t d, uint32_t seed, uint32_t epoch,
                                          uint32_t ant, int l) {
  uint32_t r[4];
  const uint32_t block = (d >> 2) + (uint32_t)l;
  philox4x32_10(block, ant, epoch, 0u, seed, kDrawKey1, r);
  constexpr uint32_t kMask = ~0u << (32 - kDrawBits);
  const uint32_t at = ring + ((16u * block) & (32u * LPA - 1u));
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(max(r[0] & kMask, 1u)),
               "r"(max(r[1] & kMask, 1u)), "r"(max(r[2] & kMask, 1u)), "r"(max(r[3] & kMask, 1u))
               : "memory");
}

// The ants of one warp, 32 / LPA at a time, in lockstep: the rules of
// build_ant in aco_kernels.cu (src/seq/aco_sequential.c:616-681 with the
// demand extension).  Each ant is LPA lanes with 4 candidates per lane (the
// first ones in its highest lane), so that a warp instruction serves 8 (4)
// ants and a step's sums take 2 (3) shuffles; what only one ant needs (the
// fallback, the repair) is done for it by the whole warp.  With one ant per
// 16 lanes and two ants drifting apart in a warp the step took 103 warp
// instructions per ant and the batch was bound by their issue (100 epochs of
// the 512-instance batch 110 ms); here it is about 95 for 8 ants, and as much
// again for their fallbacks, repairs and costs (40 ms, 2.2 instructions per
// cycle and SM at 16 warps).
template <int LPA, int E>
__device__ __forceinline__ void build_ants(const BatchArgs &a, const BatchShape &sh,
                                           const BatchInst &I, const BatchTables<E> &tb,
                                           unsigned char *smem, uint32_t seed, uint32_t epoch,
                                           int ant0, int ii) {
  constexpr int kApw = 32 / LPA;
  const int lane = threadIdx.x & 31, l = lane & (LPA - 1), seg = lane / LPA;
  const int warp = threadIdx.x >> 5;
  const int slot = warp * kApw + seg, ant = ant0 + slot;
  const bool valid = slot < sh.round && ant < a.m;
  if (!__any_sync(kFull, valid)) return;
  const unsigned seg_mask = ((LPA == 4 ? 0xfu : 0xffu) << (lane & ~(LPA - 1)));
  const int n = I.n, K = I.K, R = n + 2 * K, cap = I.cap, S = tb.S;
  const int use = valid ? ant : ant0;  // lanes without an ant read the first one's addresses
  int *route = a.routes + I.route_off + (long long)use * R;
  int *lens = a.lens + I.lens_off + (long long)use * K;
  int *loads = a.loads + I.lens_off + (long long)use * K;
  int *last = a.last + I.lens_off + (long long)use * K;
  Unserved<E> us;
  us.base = smem_addr(smem + sh.off_el) + (uint32_t)(valid ? slot : 0) * sh.el_bytes;
  us.chunks = sh.el_bytes / 16u;
  us.dem = nullptr;
  us.dem_s = smem_addr(smem + sh.off_el0);
  constexpr bool kBits = elem_is_bits(E);
  const uint32_t ring = smem_addr(smem + sh.off_draw) + (uint32_t)(valid ? slot : 0) * 32u * LPA;
  // The elements from the instance's, and the first draws.
  if (valid) {
    const uint32_t src = smem_addr(smem + sh.off_el0);
    if (kBits) us.init_bits(n, l, LPA);
    for (uint32_t o = 16u * (uint32_t)l; !kBits && o < sh.el_bytes; o += 16u * LPA) {
      uint32_t x[4];
      asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(src + o));
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(us.base + o), "r"(x[0]),
                   "r"(x[1]), "r"(x[2]), "r"(x[3]) : "memory");
    }
    ring_fill<LPA>(ring, 0u, seed, epoch, (uint32_t)ant, l);
    ring_fill<LPA>(ring, 4u * LPA, seed, epoch, (uint32_t)ant, l);
  }
  __syncwarp();

  // This lane's slots: 4 (LPA - 1 - l) ..  A lane past the row's end reads
  // zeros.
  const int s0 = kSlotsPerLane * (LPA - 1 - l);
  const bool has = s0 < S;
  const uint32_t cbase = has ? smem_addr(tb.cand) + 2u * s0 : smem_addr(smem);
  const uint32_t wbase = has ? smem_addr(tb.w) + 4u * s0 : smem_addr(smem);
  const uint32_t cstep = has ? 2u * S : 0u, wstep = has ? 4u * S : 0u;

  uint32_t d = 0, dbase = 0;  // draws spent; number of the ring's oldest
  int rem_dem = I.total_demand, pos = 0, v = 0, start = 0, cur = 0, room = 0, floor_room = 0;
  bool active = valid;
  // The route's last entries wait in the lanes (entry p in lane p mod LPA) and
  // leave LPA at a time: one entry per step per ant touched a line of its own
  // with every store (100 epochs of the 512-instance batch 47.8 -> 41.7 ms).
  int held = 0;
  auto put = [&](int node) {
    if (l == (pos & (LPA - 1))) held = node;
    ++pos;
    if ((pos & (LPA - 1)) == 0) route[pos - LPA + l] = held;
  };
  auto open_vehicle = [&]() {
    start = pos;
    put(0);
    cur = 0;
    room = cap;
    // "remaining demand > (K - v - 1) Q and load < Q" as one bound on the
    // room (see build_ant).
    const long long f = (long long)(K - v - 1) * cap - ((long long)rem_dem - cap);
    floor_room = f < 0 ? 0 : (f > INT_MAX ? INT_MAX : (int)f);
  };
  if (active) open_vehicle();

  uint32_t tick = 0;
  while (true) {
    bool closing = active && room <= floor_room;
    if (__any_sync(kFull, closing)) {
      while (closing) {
        if (l == 0) {
          lens[v] = pos + 1 - start;
          loads[v] = cap - room;
          last[v] = cur;
        }
        put(0);
        rem_dem -= cap - room;
        ++v;
        active = v < K;
        if (!active) break;
        open_vehicle();
        closing = room <= floor_room;
      }
      __syncwarp();
      if (!__any_sync(kFull, active)) break;
    }
    uint32_t c01, c23, w[4];
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];"
                 : "=r"(c01), "=r"(c23) : "r"(cbase + (uint32_t)cur * cstep));
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                 : "r"(wbase + (uint32_t)cur * wstep));
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(ring + ((4u * d) & (32u * LPA - 1u))));
    uint32_t c[4] = {c01 & 0xffffu, c01 >> 16, c23 & 0xffffu, c23 >> 16};
    uint32_t e[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e[i] = us.get((int)c[i]);
    const uint32_t lim = us.limit(room);
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = e[i] <= lim ? w[i] : 0u;
    const uint32_t p1 = w[0] + w[1], p2 = p1 + w[2], p3 = p2 + w[3];
    // Sum over the ant's lanes and over the lanes above this one (those hold
    // the candidates before this lane's).
    const uint32_t x1 = __shfl_xor_sync(kFull, p3, 1);
    const uint32_t t1 = p3 + x1;
    const uint32_t x2 = __shfl_xor_sync(kFull, t1, 2);
    uint32_t denom = t1 + x2;
    uint32_t before = ((l & 1) ? 0u : x1) + ((l & 2) ? 0u : x2);
    if (LPA == 8) {
      const uint32_t x4 = __shfl_xor_sync(kFull, denom, 4);
      denom += x4;
      before += (l & 4) ? 0u : x4;
    }
    // As in build_ant: the first candidate whose inclusive sum exceeds thr;
    // none for denom = 0.
    const uint32_t thr = (uint32_t)(((unsigned long long)r * denom - 1ull) >> 32);
    const unsigned msk = __ballot_sync(kFull, active && before + p3 > thr) & seg_mask;
    const uint32_t need = thr - before;  // in the lane chosen: before <= thr
    const bool b0 = w[0] > need, b1 = p1 > need, b2 = p2 > need;
    uint32_t cs = b0 ? c[0] : (b1 ? c[1] : (b2 ? c[2] : c[3]));
    uint32_t es = b0 ? e[0] : (b1 ? e[1] : (b2 ? e[2] : e[3]));
    const int src = 31 - __clz((int)msk);
    int next;
    uint32_t dn;
    if (E == 4 || kBits) {
      next = (int)__shfl_sync(kFull, cs, src);
      dn = __shfl_sync(kFull, es, src);
    } else {
      const uint32_t ce = __shfl_sync(kFull, cs | (es << 16), src);
      next = (int)(ce & 0xffffu);
      dn = ce >> 16;
    }
    bool take = msk != 0u;
    d += take ? 1u : 0u;  // only a roulette selection spends a draw
    unsigned none = __ballot_sync(kFull, active && !take && l == 0);
    if (none) {
      // The nearest eligible customer (the rule of nearest_eligible in
      // aco_kernels.cu), one ant after another by the whole warp.  An
      // eligible candidate whose weight is 0 would come before the tier row:
      // an ant that has one is left to the scan.  The other ants' lanes read
      // elements that this ant's lanes marked in earlier steps, and neither
      // shuffles nor ballots order memory.
      __syncwarp();
      const unsigned zero = __ballot_sync(
          kFull, e[0] <= lim || e[1] <= lim || e[2] <= lim || e[3] <= lim);
      do {
        const int b = __ffs(none) - 1;
        none &= none - 1u;
        const int fc = __shfl_sync(kFull, cur, b);
        const uint32_t fl = __shfl_sync(kFull, lim, b);
        Unserved<E> its = us;
        its.base = __shfl_sync(kFull, us.base, b);
        int nx = -1;
        if (tb.tier && ((zero >> b) & (LPA == 4 ? 0xfu : 0xffu)) == 0u) {
          const uint32_t two =
              __ldg(reinterpret_cast<const uint32_t *>(tb.tier + (size_t)fc * kTierLen) + lane);
          nx = coop_tier<E>(two, its, fl);
        }
        if (nx < 0) nx = coop_scan<E>(tb.coords, its, n, fc, fl, lane);
        if ((lane & ~(LPA - 1)) == b) {
          next = nx;
          take = nx > 0;
          if (take) dn = us.get(nx);
          else floor_room = INT_MAX;  // no customer fits: the route ends
        }
      } while (none);
      __syncwarp();  // the elements are read before they are marked
    }
    // The step, without a branch: an ant that takes none marks the depot,
    // which is marked from the start (not in a bitmap: lanes without an ant
    // would write back the first ant's word as it was).
    // A bitmap's word is read, changed and written by each of the ant's lanes: the
    // last step's writes come first.
    if (kBits) __syncwarp();
    if (!kBits) us.mark(take ? next : 0);
    else if (take) us.mark(next);
    held = take && l == (pos & (LPA - 1)) ? next : held;
    pos += take ? 1 : 0;
    if (take && (pos & (LPA - 1)) == 0) route[pos - LPA + l] = held;
    room -= take ? (int)dn : 0;
    cur = take ? next : cur;
    // Every 4 LPA steps each ant that has spent its ring's older half
    // replaces it: no ant can spend more than the other half until then.
    if (((++tick) & (4u * LPA - 1u)) == 0u) {
      __syncwarp();
      if (active && d - dbase >= 4u * LPA) {
        ring_fill<LPA>(ring, dbase + 8u * LPA, seed, epoch, (uint32_t)ant, l);
        dbase += 4u * LPA;
      }
      __syncwarp();
    }
  }

  if (valid && l < (pos & (LPA - 1))) route[(pos & ~(LPA - 1)) + l] = held;
  __syncwarp();  // routes, lengths and elements before other lanes read them
  int left = valid ? n - (pos - 2 * K) : 0;
  unsigned rm = __ballot_sync(kFull, left > 0 && l == 0);
  if (rm) {
    int *scratch = reinterpret_cast<int *>(smem + sh.off_red) + 32 * warp;
    do {
      const int b = __ffs(rm) - 1;
      rm &= rm - 1u;
      const int who = ant0 + warp * kApw + b / LPA;
      const long long lo = I.lens_off + (long long)who * K;
      Unserved<E> its = us;
      its.base = __shfl_sync(kFull, us.base, b);
      const int added = coop_repair<E>(
          tb.coords, its, n, K, cap, __shfl_sync(kFull, pos, b),
          __shfl_sync(kFull, left, b), a.routes + I.route_off + (long long)who * R, a.lens + lo,
          a.loads + lo, a.last + lo, a.rep + I.rep_off + (long long)who * n, scratch, lane);
      if ((lane & ~(LPA - 1)) == b) {
        pos += added;
        left -= added;
      }
      __syncwarp();
    } while (rm);
  }

  // FP64 cost in route order (boundary (0,0) pairs add +0.0), 4 LPA arcs at a
  // time: a lane forms 4 consecutive arcs and the ant's lanes add all of them
  // in order; the next ones' end points are loaded meanwhile.  An ant with
  // customers left has no cost anyone reads.
  const int arcs = valid && left == 0 ? pos - 1 : 0;
  double acc = 0.0;
  int nd[kSlotsPerLane + 1];
  auto load_nodes = [&](int b) {
#pragma unroll
    for (int i = 0; i <= kSlotsPerLane; ++i) {
      const int j = b + kSlotsPerLane * l + i;
      nd[i] = j <= arcs ? route[j] : 0;
    }
  };
  load_nodes(0);
  for (int b = 0; __any_sync(kFull, b < arcs); b += kSlotsPerLane * LPA) {
    double dj[kSlotsPerLane];
    float2 p = tb.coords[nd[0]];
#pragma unroll
    for (int i = 0; i < kSlotsPerLane; ++i) {
      const float2 q = tb.coords[nd[i + 1]];
      const double dx = __dsub_rn((double)p.x, (double)q.x);
      const double dy = __dsub_rn((double)p.y, (double)q.y);
      dj[i] = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
      p = q;
    }
    load_nodes(b + kSlotsPerLane * LPA);
#pragma unroll
    for (int i = 0; i < kSlotsPerLane; ++i) {
      const double s = __dsqrt_rn(dj[i] == 0.0 ? 1.0 : dj[i]);
      // Arcs past the end join node 0 to the depot or to itself: no length.
      dj[i] = dj[i] == 0.0 || b + kSlotsPerLane * l + i >= arcs ? 0.0 : s;
    }
#pragma unroll
    for (int t = 0; t < LPA; ++t)
#pragma unroll
      for (int i = 0; i < kSlotsPerLane; ++i)
        acc = __dadd_rn(acc, __shfl_sync(kFull, dj[i], t, LPA));
  }
  if (valid && l == 0) {
    const long long ai = (long long)ii * a.m + ant;
    a.cost[ai] = acc;
    a.feasible[ai] = left == 0 ? 1 : 0;
    a.steps[ai] = pos - K;
  }
}

// Slot of `node` (> 0) in a candidate row of S slots, or -1.
__device__ __forceinline__ int slot_of(const uint16_t *row, int S, int node) {
  int t = -1;
  for (int q = 0; q < S; q += 4) {
    const uint2 v = *reinterpret_cast<const uint2 *>(row + q);
    if ((int)(v.x & 0xffffu) == node) t = q;
    if ((int)(v.x >> 16) == node) t = q + 1;
    if ((int)(v.y & 0xffffu) == node) t = q + 2;
    if ((int)(v.y >> 16) == node) t = q + 3;
  }
  return t;
}

// Pheromone of an instance inside its block.  Only the levels of candidate
// cells are ever read (by the weights), and a deposit on arc (u, c) reads
// tau[u][c] and raises it and tau[c][u]; so the cells kept are those of the
// candidate pairs in both directions: fwd[i][t] = tau[i][cand[i][t]] and
// rev[i][t] = tau[cand[i][t]][i].  A cell that is in both (two mutual
// candidates) is written to both.  The full matrix would be (n+1)^2 bytes in
// L2, evaporated as a whole every epoch.
struct BatchTau {
  uint8_t *fwd, *rev;
  const uint16_t *cand;
  int S;
  float log_min, log_step;
  uint8_t q_min, q_max;
};

__device__ __forceinline__ void batch_deposit_arc(const BatchTau &t, int u, int c, float dep) {
  const int i = c > 0 ? slot_of(t.cand + u * t.S, t.S, c) : -1;  // c among u's candidates
  const int j = u > 0 ? slot_of(t.cand + c * t.S, t.S, u) : -1;  // u among c's
  if (i < 0 && j < 0) return;  // neither cell is ever read
  const int at_u = u * t.S + i, at_c = c * t.S + j;
  const uint8_t old = i >= 0 ? t.fwd[at_u] : t.rev[at_c];
  const uint8_t nq = quant(dequant(old, t.log_min, t.log_step) + dep, t.log_min, t.log_step,
                           t.q_min, t.q_max);
  if (nq > old) {
    if (i >= 0) t.fwd[at_u] = nq;
    if (j >= 0) t.rev[at_c] = nq;
  }
  const uint8_t oldr = j >= 0 ? t.fwd[at_c] : t.rev[at_u];
  if (nq > oldr) {
    if (j >= 0) t.fwd[at_c] = nq;
    if (i >= 0) t.rev[at_u] = nq;
  }
}

// Deposit of a complete solution (total = n + 2K compact entries) by the
// block: one arc per thread (the cells of different arcs differ), but the two
// arcs of a one-customer route, which share their cells, by one thread in
// order.  (0,0) pairs (empty routes, route boundaries) are no candidate cell.
__device__ __forceinline__ void batch_deposit(const BatchTau &t, const int *nodes, int total,
                                              float dep) {
  for (int j = 1 + (int)threadIdx.x; j < total; j += blockDim.x) {
    const int p = nodes[j - 1], q = nodes[j];
    if (p == 0 && q == 0) continue;
    if (q == 0 && nodes[j - 2] == 0) continue;  // second arc of [0 p 0]
    batch_deposit_arc(t, p, q, dep);
    if (p == 0 && nodes[j + 1] == 0) batch_deposit_arc(t, q, 0, dep);
  }
}

// is_significant_improvement, src/cuda/aco_cuda.cu:83-94.
__device__ __forceinline__ bool b_significant(double prev, double next, double min_rel) {
  if (prev >= DBL_MAX || next >= DBL_MAX) return next < prev;
  if (next >= __dsub_rn(prev, 1e-9)) return false;
  const double rel = __ddiv_rn(__dsub_rn(prev, next), fmax(prev, 1e-9));
  return __dadd_rn(rel, 1e-9) >= min_rel;
}

// Per-epoch weights of one instance (k_weights in aco_kernels.cu), LPA lanes
// per row.
template <int LPA>
__device__ __forceinline__ void batch_weights(const BatchArgs &a, const BatchInst &I,
                                              const uint16_t *cand, const uint8_t *fwd,
                                              const int32_t *A, const uint32_t *lut, uint32_t *w,
                                              int rows, int S) {
  const int l = threadIdx.x & (LPA - 1), seg = threadIdx.x / LPA, nseg = blockDim.x / LPA;
  const int s0 = kSlotsPerLane * l, k = a.k;
  const uint16_t *lvl = a.lvl + I.node_off * k;
#pragma unroll 2
  for (int r0 = 0; r0 < rows; r0 += nseg) {
    const int r = r0 + seg;
    const bool in = r < rows && s0 < S;
    uint2 cc = make_uint2(0u, 0u);
    uint32_t f = 0u;
    int lv[4] = {0, 0, 0, 0};
    if (in) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (s0 + i < k) lv[i] = (int)__ldg(lvl + (long long)r * k + s0 + i);
      cc = *reinterpret_cast<const uint2 *>(cand + r * S + s0);
      f = *reinterpret_cast<const uint32_t *>(fwd + r * S + s0);
    }
    const uint32_t c[4] = {cc.x & 0xffffu, cc.x >> 16, cc.y & 0xffffu, cc.y >> 16};
    int e[4], emax = INT_MIN;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      e[i] = c[i] ? A[(f >> (8 * i)) & 0xffu] - lv[i] : INT_MIN;
      emax = max(emax, e[i]);
    }
#pragma unroll
    for (int o = 1; o < LPA; o <<= 1) emax = max(emax, __shfl_xor_sync(kFull, emax, o));
    if (in) {
      uint32_t x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = c[i] ? lut[min(emax - e[i], kRelMax)] : 0u;
      *reinterpret_cast<uint4 *>(w + r * S + s0) = make_uint4(x[0], x[1], x[2], x[3]);
    }
  }
}

template <int LPA, int E>
__global__ void __launch_bounds__(kBatchThreads)
    k_batch_solve(const __grid_constant__ BatchArgs a, const __grid_constant__ BatchShape sh) {
  extern __shared__ __align__(16) unsigned char smem[];
  int32_t *s_A = reinterpret_cast<int32_t *>(smem + 16);
  uint32_t *s_lut = reinterpret_cast<uint32_t *>(smem + sh.off_lut);
  uint16_t *s_cand = reinterpret_cast<uint16_t *>(smem + sh.off_cand);
  uint32_t *s_w = reinterpret_cast<uint32_t *>(smem + sh.off_w);
  float2 *s_coords = reinterpret_cast<float2 *>(smem + sh.off_coords);
  double *s_redc = reinterpret_cast<double *>(smem + sh.off_red + (blockDim.x / 32) * 128);
  int *s_reda = reinterpret_cast<int *>(s_redc + blockDim.x / 32);
  __shared__ int s_inst, s_best, s_found, s_improved, s_stop;
  __shared__ double s_gbest;
  __shared__ int s_since;
  __shared__ float s_dep_i, s_dep_g;
  __shared__ unsigned long long s_steps;

  const int tid = threadIdx.x, nthr = blockDim.x;
  const int warp = tid >> 5, nwarps = nthr >> 5;
  const int S = sh.S;
  if (tid < 4) reinterpret_cast<uint32_t *>(smem)[tid] = 0u;
  for (int i = tid; i < 256; i += nthr) {
    s_A[i] = a.A[i];
    s_lut[i] = a.lut[i];
  }
  while (true) {
    __syncthreads();
    if (tid == 0) {
      const unsigned q = atomicAdd(a.queue, 1u);
      s_inst = (q < (unsigned)a.count) ? a.order[q] : -1;
    }
    __syncthreads();
    const int ii = s_inst;
    if (ii < 0) return;
    const BatchInst I = a.inst[ii];
    const int n = I.n, k = a.k, rows = n + 1, K = I.K;
    const uint32_t seed = a.seed + (uint32_t)ii;
    BatchTables<E> tb;
    tb.cand = s_cand;
    tb.w = s_w;
    tb.coords = s_coords;
    tb.tier = n >= kBatchTierMinCustomers ? a.tier + I.node_off * kTierLen : nullptr;
    tb.S = S;
    BatchTau bt;
    bt.fwd = sh.tau_smem ? smem + sh.off_tau : a.tau + I.node_off * 2 * kMaxCand;
    bt.rev = bt.fwd + rows * S;
    bt.cand = s_cand;
    bt.S = S;
    bt.log_min = a.log_min;
    bt.log_step = a.log_step;
    bt.q_min = 0;
    bt.q_max = 255;
    // Stage the instance: rows at stride S (empty slots 0), coordinates, the
    // elements of an unserved instance, the initial pheromone.
    for (int e = tid; e < rows * S; e += nthr) {
      const int r = e / S, t = e - r * S;
      s_cand[e] = t < k ? a.cand[(I.node_off + r) * k + t] : (uint16_t)0;
    }
    for (int e = tid; e < rows; e += nthr) s_coords[e] = a.coords[I.node_off + e];
    constexpr uint32_t kSize = elem_is_bits(E) ? 4u : (uint32_t)E;
    for (uint32_t e = tid; e < sh.el0_bytes / kSize; e += nthr) {
      const uint32_t x = e >= 1 && e <= (uint32_t)n ? (uint32_t)a.demand[I.node_off + e]
                                                    : Unserved<E>::kVisited;
      if (E == 1) smem[sh.off_el0 + e] = (unsigned char)x;
      else if (E == 2) reinterpret_cast<uint16_t *>(smem + sh.off_el0)[e] = (uint16_t)x;
      else reinterpret_cast<uint32_t *>(smem + sh.off_el0)[e] = x;
    }
    for (int e = tid; e < rows * S / 2; e += nthr)
      reinterpret_cast<uint32_t *>(bt.fwd)[e] = 0x01010101u * a.q_tau0;
    if (tid == 0) {
      s_gbest = DBL_MAX;
      s_since = 0;
      s_stop = 0;
      s_steps = 0ull;
    }
    __syncthreads();
    int epoch = 0;
    for (; epoch < a.epochs && !s_stop; ++epoch) {
      batch_weights<LPA>(a, I, s_cand, bt.fwd, s_A, s_lut, s_w, rows, S);
      __syncthreads();
      for (int a0 = 0; a0 < a.m; a0 += sh.round)
        build_ants<LPA, E>(a, sh, I, tb, smem, seed, (uint32_t)epoch, a0, ii);
      __syncthreads();
      // Iteration best: first minimum among feasible ants (k_best_cluster).
      {
        double bc = DBL_MAX;
        int ba = INT_MAX;
        unsigned long long st = 0;
        for (int i = tid; i < a.m; i += nthr) {
          const long long ai = (long long)ii * a.m + i;
          st += (unsigned long long)a.steps[ai];
          if (a.feasible[ai]) {
            const double c = a.cost[ai];
            if (ba == INT_MAX || c < bc) {
              bc = c;
              ba = i;
            }
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const double oc = __shfl_down_sync(kFull, bc, o);
          const int oa = __shfl_down_sync(kFull, ba, o);
          st += __shfl_down_sync(kFull, st, o);
          if (oa != INT_MAX && (ba == INT_MAX || oc < bc || (oc == bc && oa < ba))) {
            bc = oc;
            ba = oa;
          }
        }
        if ((tid & 31) == 0) {
          s_redc[warp] = bc;
          s_reda[warp] = ba;
          atomicAdd(&s_steps, st);
        }
        __syncthreads();
        if (tid == 0) {
          bc = DBL_MAX;
          ba = INT_MAX;
          for (int w = 0; w < nwarps; ++w) {
            const double oc = s_redc[w];
            const int oa = s_reda[w];
            if (oa != INT_MAX && (ba == INT_MAX || oc < bc || (oc == bc && oa < ba))) {
              bc = oc;
              ba = oa;
            }
          }
          const bool found = ba != INT_MAX;
          s_found = found;
          s_improved = 0;
          s_best = ba;
          if (found) {
            if (bc < s_gbest) {
              s_improved = 1;
              if (b_significant(s_gbest, bc, a.min_rel)) s_since = 0; else s_since += 1;
              s_gbest = bc;
            } else {
              s_since += 1;
            }
            s_dep_i = __fdiv_rn(0.3f * a.Qs, (float)bc);
            s_dep_g = __fdiv_rn(0.7f * a.Qs, (float)s_gbest);
          } else {
            s_since += 1;
          }
          if (a.stagnation > 0 && s_since >= a.stagnation) s_stop = 1;
        }
        __syncthreads();
      }
      const int total = n + 2 * K;  // entries of a feasible ant's routes
      const int *it_nodes = a.routes + I.route_off + (long long)s_best * total;
      if (s_improved) {
        const int *sl = a.lens + I.lens_off + (long long)s_best * K;
        for (int t = tid; t < total; t += nthr) a.gbest_nodes[I.gbest_off + t] = it_nodes[t];
        for (int v = tid; v < K; v += nthr) a.gbest_lens[I.gblens_off + v] = sl[v];
      }
      if (s_found) {
        // Evaporation max(q, delta) - delta (q_min = 0), then both deposits.
        const uint32_t delta4 = 0x01010101u * a.delta;
        for (int e = tid; e < rows * S / 2; e += nthr) {
          uint32_t *x = reinterpret_cast<uint32_t *>(bt.fwd) + e;
          *x = __vsub4(__vmaxu4(*x, delta4), delta4);
        }
        __syncthreads();
        batch_deposit(bt, it_nodes, total, s_dep_i);
        __syncthreads();
        batch_deposit(bt, a.gbest_nodes + I.gbest_off, total, s_dep_g);
        __syncthreads();
      }
    }
    if (tid == 0) {
      a.out_cost[ii] = s_gbest;
      a.out_epochs[ii] = epoch;
      a.out_steps[ii] = s_steps;
    }
  }
}

using BatchKernel = void (*)(BatchArgs, BatchShape);

template <int LPA>
BatchKernel batch_kernel_of(int elem) {
  switch (elem) {
    case 1: return k_batch_solve<LPA, 1>;
    case 2: return k_batch_solve<LPA, 2>;
    case 4: return k_batch_solve<LPA, 4>;
  }
  return k_batch_solve<LPA, kElemStagedBits>;
}

BatchKernel batch_kernel(int lpa, int elem) {
  return lpa == 4 ? batch_kernel_of<4>(elem) : batch_kernel_of<8>(elem);
}

// Opts the kernels into the largest dynamic shared memory their static
// shared variables leave free.
cudaError_t configure_batch() {
  for (int lpa : {4, 8})
    for (int elem : {1, 2, 4, kElemStagedBits}) {
      cudaFuncAttributes fa;
      const void *f = reinterpret_cast<const void *>(batch_kernel(lpa, elem));
      cudaError_t e = cudaFuncGetAttributes(&fa, f);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 construct_max_smem() - (int)fa.sharedSizeBytes);
      if (e != cudaSuccess) return e;
    }
  return cudaSuccess;
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------

struct aco_b200_batch {
  int device = 0, num_sms = 148;
  cudaStream_t stream = nullptr;
  bool own_stream = true;
  bool ready = false;
  int count = 0, m = 0, k = 0, epochs = 0, max_rows = 0, max_K = 0, max_n = 0, max_demand = 0;
  BatchArgs args = {};
  std::vector<BatchInst> inst;
  std::vector<int> sizes;  // work estimate per instance
  // Every device buffer is a 256-byte aligned slice of one allocation; a
  // set-up reuses it while the new batch fits, so solving a stream of
  // batches allocates once.
  unsigned char *arena = nullptr;
  size_t arena_cap = 0, arena_used = 0;
  bool sizing = false;
  aco_b200_batch_tuning tuning = {32, 16, 1};
  // The solve (queue reset + persistent launch) as a CUDA graph, kept while
  // the launch's arguments are unchanged.
  cudaGraphExec_t graph = nullptr;
  std::vector<unsigned char> graph_key;
  const float *d_thr = nullptr;  // eta thresholds (plain levels)
  const long long *d_seg_off = nullptr;  // first row of every instance
  const int *d_seg_n = nullptr;          // customers of every instance
  long long rows = 0;                    // sum of n + 1
  void drop_graph() {
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
    graph_key.clear();
  }
  void free_all() {
    drop_graph();
    if (arena) cudaFree(arena);
    arena = nullptr;
    arena_cap = arena_used = 0;
    ready = false;
  }
  template <typename T>
  void carve(T **p, size_t count) {
    size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
    if (bytes == 0) bytes = 256;
    *p = sizing ? nullptr : reinterpret_cast<T *>(arena + arena_used);
    arena_used += bytes;
  }
};

#define BTRY(call)                                                                     \
  do {                                                                                 \
    cudaError_t err__ = (call);                                                        \
    if (err__ != cudaSuccess) {                                                        \
      fprintf(stderr, "aco_b200_batch: CUDA error %s at %s:%d\n",                      \
              cudaGetErrorString(err__), __FILE__, __LINE__);                          \
      return err__ == cudaErrorMemoryAllocation ? ACO_ERR_ALLOCATION : ACO_ERR_BACKEND; \
    }                                                                                  \
  } while (0)

// Part of the accepted sizes: 32 nodes per lane and word, two words at most.
static int batch_v_for(int lanes, int max_rows) {
  const int words = (max_rows + 31) / 32;
  if (words <= lanes) return 1;
  if (words <= 2 * lanes) return 2;
  return 0;
}

// The launch for the batch: every ant of a colony at a time where a block's
// threads and shared memory allow, with bitmaps in place of the ants' elements
// where those leave no room; of the ways to do that, the one with the most
// blocks resident at once that the instances can use, and then with the
// pheromone levels in shared memory.
static bool choose_shape(const aco_b200_batch *b, BatchShape *out, int *grid) {
  const int lpa = b->k <= 16 ? 4 : 8;
  const int most = kBatchThreads / lpa;
  const int rounds = (b->m + most - 1) / most;
  const int useful = (b->count + b->num_sms - 1) / b->num_sms;  // blocks per SM with work
  int best = 0;
  for (int round = (b->m + rounds - 1) / rounds; round >= 1 && best == 0;
       round = round > 8 ? round * 3 / 4 : round - 1) {
    for (int elem : {demand_bytes(b->max_demand), kElemStagedBits}) {
      for (int tau_smem = 1; tau_smem >= 0; --tau_smem) {
        const BatchShape sh =
            batch_shape(b->max_rows, b->max_n, b->k, elem, round, tau_smem != 0);
        if ((int)sh.total + 64 > construct_max_smem()) continue;
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                &per_sm, reinterpret_cast<const void *>(batch_kernel(sh.lpa, elem)), sh.threads,
                sh.total) != cudaSuccess)
          return false;
        per_sm = std::min(per_sm, useful);
        if (per_sm > best) {
          best = per_sm;
          *out = sh;
        }
      }
      if (best > 0) break;
    }
  }
  *grid = std::min(best * b->num_sms, b->count);
  return best > 0;
}

extern "C" {

int aco_b200_batch_create(aco_b200_batch **out, int device) {
  if (!out) return ACO_ERR_INVALID_INPUT;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
    return ACO_ERR_BACKEND;
  aco_b200_batch *b = new aco_b200_batch();
  b->device = device;
  cudaSetDevice(device);
  cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, device);
  cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = configure_batch();
  if (e != cudaSuccess) {
    fprintf(stderr, "aco_b200_batch_create: %s\n", cudaGetErrorString(e));
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return ACO_ERR_BACKEND;
  }
  *out = b;
  return ACO_OK;
}

int aco_b200_batch_destroy(aco_b200_batch *b) {
  if (!b) return ACO_OK;
  cudaSetDevice(b->device);
  b->free_all();
  if (b->stream && b->own_stream) cudaStreamDestroy(b->stream);
  delete b;
  return ACO_OK;
}

int aco_b200_batch_set_stream(aco_b200_batch *b, void *cuda_stream) {
  if (!b) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  b->drop_graph();
  if (b->stream && b->own_stream) cudaStreamDestroy(b->stream);
  if (cuda_stream) {
    b->stream = (cudaStream_t)cuda_stream;
    b->own_stream = false;
  } else {
    BTRY(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    b->own_stream = true;
  }
  return ACO_OK;
}

int aco_b200_batch_setup(aco_b200_batch *b, const aco_b200_batch_problem *p) {
  if (!b || !p || p->count <= 0 || !p->n || !p->K || !p->capacity || !p->x || !p->y)
    return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  b->ready = false;
  const int count = p->count;
  int k = p->cand_k > 0 ? p->cand_k : 32;
  if (k > kMaxCand) k = kMaxCand;
  const int m = p->ants > 0 ? p->ants : 64;
  b->inst.assign(count, BatchInst{});
  b->sizes.assign(count, 0);
  long long node = 0, route = 0, lensn = 0, gb = 0, gbl = 0, rep = 0;
  int max_rows = 0, max_K = 0, max_n = 0, max_demand = 1;
  std::vector<float2> xy;
  std::vector<int> dem;
  std::vector<long long> seg_off(count);
  std::vector<int> seg_n(count);
  for (int i = 0; i < count; ++i) {
    const int n = p->n[i], K = p->K[i];
    const long long cap = p->capacity[i];
    if (n < 1 || K < 1 || cap < 1 || cap > 0x7fffffffLL || n < k) {
      fprintf(stderr, "aco_b200_batch: instance %d invalid (n=%d K=%d cap=%lld, k=%d)\n", i, n,
              K, cap, k);
      return ACO_ERR_INVALID_INPUT;
    }
    BatchInst &I = b->inst[i];
    I.n = n;
    I.K = K;
    I.cap = (int)cap;
    long long tot = 0;
    int mx = 1;
    for (int j = 0; j <= n; ++j) {
      const int d = p->demand ? p->demand[node + j] : (j ? 1 : 0);
      if ((j == 0 && d != 0) || (j > 0 && d < 1)) return ACO_ERR_INVALID_INPUT;
      if (j > 0) {
        tot += d;
        mx = d > mx ? d : mx;
      }
      xy.push_back(make_float2(p->x[node + j], p->y[node + j]));
      dem.push_back(d);
    }
    if (tot > 0x7fffffffLL) return ACO_ERR_INVALID_INPUT;
    I.total_demand = (int)tot;
    max_demand = std::max(max_demand, mx);
    I.node_off = node;
    seg_off[i] = node;
    seg_n[i] = n;
    I.route_off = route;
    I.lens_off = lensn;
    I.gbest_off = gb;
    I.gblens_off = gbl;
    I.rep_off = rep;
    node += n + 1;
    route += (long long)m * (n + 2 * K);
    lensn += (long long)m * K;
    gb += n + 2 * K;
    gbl += K;
    rep += (long long)m * n;
    max_rows = std::max(max_rows, n + 1);
    max_K = std::max(max_K, K);
    max_n = std::max(max_n, n);
    b->sizes[i] = (n + K) * m;
  }
  if (batch_v_for(16, max_rows) == 0 && batch_v_for(32, max_rows) == 0) {
    fprintf(stderr, "aco_b200_batch: n <= 2046 per instance\n");
    return ACO_ERR_INVALID_INPUT;
  }
  b->count = count;
  b->m = m;
  b->k = k;
  b->epochs = p->epochs;
  b->max_rows = max_rows;
  b->max_K = max_K;
  b->max_n = max_n;
  b->max_demand = max_demand;

  float lmin = logf(0.0001f), lmax = logf(100.0f);
  float step = (lmax - lmin) / 255.0f;
  const float log_rho = logf(1.0f - (float)p->rho);
  uint8_t delta = (uint8_t)fmaxf(1.0f, roundf(-log_rho / step));
  uint8_t q0 = (uint8_t)fmaxf(0.0f, fminf(255.0f, roundf((logf((float)p->tau0) - lmin) / step)));
  // Tables as in the single-instance set-up.
  std::vector<int32_t> A(256);
  std::vector<uint32_t> lut(256);
  std::vector<float> thr(kThresholds, INFINITY);
  const double ln2 = 0.69314718055994530942;
  for (int q = 0; q < 256; ++q)
    A[q] = (int32_t)std::floor(p->alpha * (double)q * (double)step * kLevelsPerOctave / ln2 + 0.5);
  for (int r = 0; r < kRelMax; ++r)
    lut[r] = (uint32_t)std::floor(8388608.0 * std::exp2(-(double)r / kLevelsPerOctave) + 0.5);
  lut[kRelMax] = 0u;
  if (p->beta > 0.0)
    for (int j = 1; j <= kThresholds; ++j) {
      const double t = std::exp2(2.0 * (double)j / (p->beta * kLevelsPerOctave));
      thr[j - 1] = (t > 3.0e38) ? INFINITY : (float)t;
    }

  BatchArgs &a = b->args;
  a = BatchArgs{};
  a.count = count;
  a.m = m;
  a.k = k;
  a.epochs = p->epochs;
  a.stagnation = p->stagnation_epochs > 0 ? p->stagnation_epochs : 0;
  a.min_rel = p->min_rel_improvement > 0.0 ? p->min_rel_improvement : 1e-3;
  a.Qs = (float)p->Q * 100.0f;
  a.log_min = lmin;
  a.log_step = step;
  a.delta = delta;
  a.q_tau0 = q0;
  a.seed = p->seed;
  BatchInst *d_inst;
  int *d_order;
  float2 *d_coords;
  int *d_dem;
  uint16_t *d_cand, *d_lvl, *d_tier;
  int32_t *d_A;
  uint32_t *d_lut;
  float *d_thr;
  long long *d_soff;
  int *d_sn;
  auto layout = [&]() {
    b->arena_used = 0;
    b->carve(&d_inst, count);
    b->carve(&d_order, count);
    b->carve(&d_coords, node);
    b->carve(&d_dem, node);
    // Candidate tables sized for the longest list, so that
    // aco_b200_batch_set_cand_k can rebuild them with any length in place.
    b->carve(&d_cand, node * kMaxCand);
    b->carve(&d_lvl, node * kMaxCand);
    b->carve(&d_tier, node * kTierLen);
    b->carve(&d_A, 256);
    b->carve(&d_lut, 256);
    b->carve(&d_thr, kThresholds);
    b->carve(&d_soff, count);
    b->carve(&d_sn, count);
    b->carve(&a.tau, node * 2 * kMaxCand);
    b->carve(&a.routes, route);
    b->carve(&a.lens, lensn);
    b->carve(&a.loads, lensn);
    b->carve(&a.last, lensn);
    b->carve(&a.rep, rep);
    b->carve(&a.cost, (long long)count * m);
    b->carve(&a.feasible, (long long)count * m);
    b->carve(&a.steps, (long long)count * m);
    b->carve(&a.gbest_nodes, gb);
    b->carve(&a.gbest_lens, gbl);
    b->carve(&a.out_cost, count);
    b->carve(&a.out_epochs, count);
    b->carve(&a.out_steps, count);
    b->carve(&a.queue, 1);
  };
  b->sizing = true;
  layout();
  b->sizing = false;
  const size_t need = b->arena_used;
  if (need > b->arena_cap) {
    b->free_all();
    BTRY(cudaMalloc((void **)&b->arena, need));
    b->arena_cap = need;
  }
  layout();
  cudaStream_t s = b->stream;
  BTRY(cudaMemsetAsync(b->arena, 0, need, s));
  BTRY(cudaMemcpyAsync(d_inst, b->inst.data(), sizeof(BatchInst) * count, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_coords, xy.data(), sizeof(float2) * node, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_dem, dem.data(), sizeof(int) * node, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_A, A.data(), 1024, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_lut, lut.data(), 1024, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_thr, thr.data(), sizeof(float) * kThresholds, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_soff, seg_off.data(), sizeof(long long) * count, cudaMemcpyHostToDevice, s));
  BTRY(cudaMemcpyAsync(d_sn, seg_n.data(), sizeof(int) * count, cudaMemcpyHostToDevice, s));
  BTRY(launch_knn_levels_multi(d_coords, d_soff, d_sn, count, node, k, d_thr, kThresholds, d_cand,
                               d_lvl, d_tier, s));
  b->d_seg_off = d_soff;
  b->d_seg_n = d_sn;
  b->rows = node;
  b->d_thr = d_thr;
  a.inst = d_inst;
  a.order = d_order;
  a.coords = d_coords;
  a.demand = d_dem;
  a.cand = d_cand;
  a.lvl = d_lvl;
  a.tier = d_tier;
  a.A = d_A;
  a.lut = d_lut;
  BTRY(cudaStreamSynchronize(s));
  b->ready = true;
  aco_b200_batch_tuning t = {32, 16, 1};
  return aco_b200_batch_set_tuning(b, &t);
}

int aco_b200_batch_set_tuning(aco_b200_batch *b, const aco_b200_batch_tuning *t) {
  if (!b || !b->ready || !t) return ACO_ERR_INVALID_INPUT;
  if (t->lanes_per_ant != 16 && t->lanes_per_ant != 32) return ACO_ERR_INVALID_INPUT;
  if (t->lanes_per_ant < b->k) return ACO_ERR_INVALID_INPUT;
  if (t->ants_per_block < 1 || t->ants_per_block * t->lanes_per_ant > 1024) return ACO_ERR_INVALID_INPUT;
  if ((t->ants_per_block * t->lanes_per_ant) % 32) return ACO_ERR_INVALID_INPUT;
  if (batch_v_for(t->lanes_per_ant, b->max_rows) == 0) return ACO_ERR_INVALID_INPUT;
  const int threads = t->ants_per_block * t->lanes_per_ant;
  if ((int)shape_bytes(b->max_rows, b->k, t->ants_per_block, threads, b->max_K) > construct_max_smem())
    return ACO_ERR_INVALID_INPUT;
  // Queue order: 0 = as given, 1 = largest work first.
  std::vector<int> order(b->count);
  std::iota(order.begin(), order.end(), 0);
  if (t->order == 1)
    std::stable_sort(order.begin(), order.end(),
                     [&](int x, int y) { return b->sizes[x] > b->sizes[y]; });
  cudaSetDevice(b->device);
  // Stream-ordered after any solve in flight; a pageable source is staged
  // before the call returns.
  BTRY(cudaMemcpyAsync(const_cast<int *>(b->args.order), order.data(), sizeof(int) * b->count,
                       cudaMemcpyHostToDevice, b->stream));
  b->tuning = *t;
  return ACO_OK;
}

int aco_b200_batch_get_tuning(aco_b200_batch *b, aco_b200_batch_tuning *t) {
  if (!b || !b->ready || !t) return ACO_ERR_INVALID_INPUT;
  *t = b->tuning;
  return ACO_OK;
}

int aco_b200_batch_enqueue(aco_b200_batch *b) {
  if (!b || !b->ready) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  BatchShape sh;
  int grid = 0;
  if (!choose_shape(b, &sh, &grid)) return ACO_ERR_INVALID_INPUT;
  auto record = [&](cudaStream_t s) -> cudaError_t {
    cudaError_t e = cudaMemsetAsync(b->args.queue, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    batch_kernel(sh.lpa, sh.elem)<<<grid, sh.threads, sh.total, s>>>(b->args, sh);
    return cudaGetLastError();
  };
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  BTRY(cudaStreamIsCapturing(b->stream, &cap));
  if (cap != cudaStreamCaptureStatusNone) {
    // The caller is capturing this stream into a graph of its own: record
    // the solve there.
    BTRY(record(b->stream));
    return ACO_OK;
  }
  // The key: every argument of the two graph nodes.
  std::vector<unsigned char> key(sizeof(BatchArgs) + sizeof(BatchShape) + sizeof(int));
  memcpy(key.data(), &b->args, sizeof(BatchArgs));
  memcpy(key.data() + sizeof(BatchArgs), &sh, sizeof(BatchShape));
  memcpy(key.data() + sizeof(BatchArgs) + sizeof(BatchShape), &grid, sizeof(int));
  if (!b->graph || key != b->graph_key) {
    b->drop_graph();
    cudaGraph_t g = nullptr;
    BTRY(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    const cudaError_t err = record(b->stream);
    const cudaError_t end = cudaStreamEndCapture(b->stream, &g);
    if (err != cudaSuccess || end != cudaSuccess) {
      if (g) cudaGraphDestroy(g);
      BTRY(err != cudaSuccess ? err : end);
    }
    const cudaError_t ie = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    if (ie != cudaSuccess) b->graph = nullptr;
    BTRY(ie);
    b->graph_key = key;
  }
  BTRY(cudaGraphLaunch(b->graph, b->stream));
  return ACO_OK;
}

int aco_b200_batch_solve(aco_b200_batch *b) {
  int rc = aco_b200_batch_enqueue(b);
  if (rc) return rc;
  BTRY(cudaStreamSynchronize(b->stream));
  return ACO_OK;
}

int aco_b200_batch_synchronize(aco_b200_batch *b) {
  if (!b) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  BTRY(cudaStreamSynchronize(b->stream));
  return ACO_OK;
}

int aco_b200_batch_autotune(aco_b200_batch *b, int trial_epochs, aco_b200_batch_tuning *chosen,
                            float *trial_ms, int max_trials, int *n_trials) {
  if (!b || !b->ready || trial_epochs < 1) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  const int saved_epochs = b->args.epochs;
  b->args.epochs = trial_epochs;
  const aco_b200_batch_tuning cands[] = {
      {32, 8, 1}, {32, 16, 1}, {32, 32, 1}, {16, 16, 1}, {16, 32, 1}, {16, 64, 1},
      {32, 16, 0}, {16, 32, 0}};
  // Of a shape only the queue order reaches the launch (choose_shape takes the
  // rest from the batch), so each order is timed once, behind an untimed solve,
  // and every shape that is accepted gets its order's time.
  float order_ms[2] = {-1.f, -1.f};
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const aco_b200_batch_tuning before = b->tuning;
  int nt = 0;
  for (const auto &c : cands) {
    if (aco_b200_batch_set_tuning(b, &c) != ACO_OK) continue;
    float &ms = order_ms[c.order];
    if (ms < 0.f && (nt > 0 || aco_b200_batch_enqueue(b) == ACO_OK)) {
      cudaEventRecord(e0, b->stream);
      const int rc = aco_b200_batch_enqueue(b);
      cudaEventRecord(e1, b->stream);
      if (rc != ACO_OK || cudaEventSynchronize(e1) != cudaSuccess ||
          cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess)
        ms = -1.f;
    }
    if (trial_ms && nt < max_trials) trial_ms[nt] = ms;
    ++nt;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  b->args.epochs = saved_epochs;
  if (n_trials) *n_trials = nt;
  aco_b200_batch_tuning best = before;
  const int other = before.order == 1 ? 0 : 1;
  const float kept = order_ms[1 - other], ms = order_ms[other];
  if (ms > 0.f && !(kept > 0.f && kept <= ms)) best.order = other;
  int rc = aco_b200_batch_set_tuning(b, &best);
  if (chosen) *chosen = best;
  return rc;
}

int aco_b200_batch_set_cand_k(aco_b200_batch *b, int k) {
  if (!b || !b->ready || k < 1 || k > kMaxCand) return ACO_ERR_INVALID_INPUT;
  for (const BatchInst &I : b->inst)
    if (I.n < k) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  BatchArgs &a = b->args;
  BTRY(launch_knn_levels_multi(a.coords, b->d_seg_off, b->d_seg_n, b->count, b->rows, k,
                               b->d_thr, kThresholds, const_cast<uint16_t *>(a.cand),
                               const_cast<uint16_t *>(a.lvl), const_cast<uint16_t *>(a.tier),
                               b->stream));
  b->k = k;
  a.k = k;
  // The launch shape must hold the new list: keep it when it does, else the
  // default shape (32 lanes per ant).
  aco_b200_batch_tuning t = b->tuning;
  if (aco_b200_batch_set_tuning(b, &t) != ACO_OK) {
    t = aco_b200_batch_tuning{32, 16, 1};
    const int rc = aco_b200_batch_set_tuning(b, &t);
    if (rc) return rc;
  }
  BTRY(cudaStreamSynchronize(b->stream));
  return ACO_OK;
}

int aco_b200_batch_get_cand_k(aco_b200_batch *b, int *k) {
  if (!b || !b->ready || !k) return ACO_ERR_INVALID_INPUT;
  *k = b->k;
  return ACO_OK;
}

int aco_b200_batch_autotune_k(aco_b200_batch *b, int trial_epochs, const int *ks, int nks,
                              double quality_tol, aco_b200_batch_tuning *chosen, int *chosen_k,
                              double *k_solve_ms, double *k_mean_cost, int *k_feasible,
                              float *trial_ms, int max_trials, int *n_trials) {
  if (!b || !b->ready || !ks || nks < 1 || nks > 16 || !(quality_tol >= 0.0))
    return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  const int count = b->count;
  std::vector<std::vector<double>> costs(nks);
  std::vector<double> ms(nks, -1.0);
  std::vector<int> valid(nks, 0);
  cudaEvent_t e0, e1;
  BTRY(cudaEventCreate(&e0));
  BTRY(cudaEventCreate(&e1));
  // Stage 1: one whole solve per candidate-list length, on the default
  // launch shape (the shape does not change results, the length does).
  for (int i = 0; i < nks; ++i) {
    if (aco_b200_batch_set_cand_k(b, ks[i]) != ACO_OK) continue;
    aco_b200_batch_tuning t = {32, 16, 1};
    if (aco_b200_batch_set_tuning(b, &t) != ACO_OK) continue;
    cudaEventRecord(e0, b->stream);
    const int rc = aco_b200_batch_enqueue(b);
    cudaEventRecord(e1, b->stream);
    float t_ms = -1.f;
    if (rc != ACO_OK || cudaEventSynchronize(e1) != cudaSuccess ||
        cudaEventElapsedTime(&t_ms, e0, e1) != cudaSuccess)
      continue;
    costs[i].resize(count);
    if (aco_b200_batch_get_costs(b, costs[i].data(), nullptr, nullptr) != ACO_OK) continue;
    ms[i] = t_ms;
    valid[i] = 1;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // Quality: the mean final cost over the instances every length solved;
  // a length that leaves more instances without a solution is worse.
  std::vector<int> infeasible(nks, 0);
  std::vector<char> common(count, 1);
  for (int i = 0; i < nks; ++i) {
    if (!valid[i]) continue;
    for (int j = 0; j < count; ++j) {
      if (costs[i][j] >= DBL_MAX) {
        infeasible[i] += 1;
        common[j] = 0;
      }
    }
  }
  int min_inf = count + 1;
  for (int i = 0; i < nks; ++i)
    if (valid[i] && infeasible[i] < min_inf) min_inf = infeasible[i];
  std::vector<double> mean(nks, DBL_MAX);
  double best_mean = DBL_MAX;
  for (int i = 0; i < nks; ++i) {
    if (!valid[i]) continue;
    double sum = 0.0;
    int cnt = 0;
    for (int j = 0; j < count; ++j)
      if (common[j]) {
        sum += costs[i][j];
        ++cnt;
      }
    mean[i] = cnt ? sum / cnt : DBL_MAX;
    if (infeasible[i] == min_inf && mean[i] < best_mean) best_mean = mean[i];
  }
  // The fastest length within quality_tol of the best quality.
  int pick = -1;
  for (int i = 0; i < nks; ++i) {
    if (!valid[i] || infeasible[i] != min_inf) continue;
    if (mean[i] > best_mean * (1.0 + quality_tol)) continue;
    if (pick < 0 || ms[i] < ms[pick]) pick = i;
  }
  for (int i = 0; i < nks; ++i) {
    if (k_solve_ms) k_solve_ms[i] = ms[i];
    if (k_mean_cost) k_mean_cost[i] = valid[i] ? mean[i] : -1.0;
    if (k_feasible) k_feasible[i] = valid[i] ? count - infeasible[i] : -1;
  }
  if (pick < 0) return ACO_ERR_INVALID_INPUT;
  int rc = aco_b200_batch_set_cand_k(b, ks[pick]);
  if (rc) return rc;
  if (chosen_k) *chosen_k = ks[pick];
  // Stage 2: the queue order for that length.
  return aco_b200_batch_autotune(b, trial_epochs, chosen, trial_ms, max_trials, n_trials);
}

int aco_b200_batch_get(aco_b200_batch *b, int instance, int *nodes, int *lens, double *cost,
                       int *epochs) {
  if (!b || !b->ready || instance < 0 || instance >= b->count) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  const BatchInst &I = b->inst[instance];
  cudaStream_t s = b->stream;
  BTRY(cudaMemcpyAsync(cost, b->args.out_cost + instance, sizeof(double), cudaMemcpyDeviceToHost, s));
  if (epochs)
    BTRY(cudaMemcpyAsync(epochs, b->args.out_epochs + instance, sizeof(int), cudaMemcpyDeviceToHost, s));
  if (lens)
    BTRY(cudaMemcpyAsync(lens, b->args.gbest_lens + I.gblens_off, sizeof(int) * I.K,
                         cudaMemcpyDeviceToHost, s));
  if (nodes)
    BTRY(cudaMemcpyAsync(nodes, b->args.gbest_nodes + I.gbest_off, sizeof(int) * (I.n + 2 * I.K),
                         cudaMemcpyDeviceToHost, s));
  BTRY(cudaStreamSynchronize(s));
  return *cost < DBL_MAX ? ACO_OK : ACO_ERR_NO_SOLUTION;
}

int aco_b200_batch_get_costs(aco_b200_batch *b, double *costs, int *epochs,
                             unsigned long long *steps) {
  if (!b || !b->ready) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  cudaStream_t s = b->stream;
  if (costs)
    BTRY(cudaMemcpyAsync(costs, b->args.out_cost, sizeof(double) * b->count, cudaMemcpyDeviceToHost, s));
  if (epochs)
    BTRY(cudaMemcpyAsync(epochs, b->args.out_epochs, sizeof(int) * b->count, cudaMemcpyDeviceToHost, s));
  if (steps)
    BTRY(cudaMemcpyAsync(steps, b->args.out_steps, sizeof(unsigned long long) * b->count,
                         cudaMemcpyDeviceToHost, s));
  BTRY(cudaStreamSynchronize(s));
  return ACO_OK;
}

int aco_b200_batch_get_all(aco_b200_batch *b, int *nodes, int *lens, double *costs) {
  if (!b || !b->ready) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  cudaStream_t s = b->stream;
  const BatchInst &last = b->inst[b->count - 1];
  if (nodes)
    BTRY(cudaMemcpyAsync(nodes, b->args.gbest_nodes,
                         sizeof(int) * (last.gbest_off + last.n + 2 * last.K),
                         cudaMemcpyDeviceToHost, s));
  if (lens)
    BTRY(cudaMemcpyAsync(lens, b->args.gbest_lens, sizeof(int) * (last.gblens_off + last.K),
                         cudaMemcpyDeviceToHost, s));
  if (costs)
    BTRY(cudaMemcpyAsync(costs, b->args.out_cost, sizeof(double) * b->count, cudaMemcpyDeviceToHost, s));
  BTRY(cudaStreamSynchronize(s));
  return ACO_OK;
}

}  // extern "C"

extern "C" int aco_b200_batch_apply_prior(aco_b200_batch *b, aco_b200_prior *prior, float gamma) {
  if (!b || !b->ready) return ACO_ERR_INVALID_INPUT;
  cudaSetDevice(b->device);
  cudaStream_t s = b->stream;
  const BatchArgs &a = b->args;
  uint16_t *lvl = const_cast<uint16_t *>(a.lvl);
  if (prior && gamma > 0.f) {
    const int rc = acob200::prior::learned_levels_multi(
        prior, a.coords, a.demand, &a.inst->cap, (int)(sizeof(BatchInst) / sizeof(int)),
        b->d_seg_off, b->d_seg_n, b->count, b->rows, b->k, a.cand, lvl, gamma, s);
    if (rc) return rc;
  } else {
    BTRY(launch_knn_levels_multi(a.coords, b->d_seg_off, b->d_seg_n, b->count, b->rows, b->k,
                                 b->d_thr, kThresholds, const_cast<uint16_t *>(a.cand), lvl,
                                 nullptr, s));
  }
  BTRY(cudaStreamSynchronize(s));
  return ACO_OK;
}
