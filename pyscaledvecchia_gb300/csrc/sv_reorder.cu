// Batched reorder of many independent problems: the rebuild step of the fit
// (gp.py:182-191) for every problem of a batched fit in one call.
//
// Per problem p with inputs X_e (n x d, subsample order), y_e, Z_e and
// ranges r (host values, so the division below sees numpy's exp bits):
//   Xs   = X_e / r                                (gp.py:184, IEEE division)
//   ord  = maximin order of Xs from row `first`   (ordering.py:27-73)
//   X, y, Z <- X_e[ord], y_e[ord], Z_e[ord]        (gp.py:189-191)
//   nbr  <- ordered kNN of Xs[ord], m neighbours   (ordering.py:76-116), written
//           straight into the likelihood's block columns: block blk_off + i
//           holds row i's min(i, m) neighbours, nearest first, -1 padded
//           (the _nn_groups layout, ordering.py:119-127, with row i = block i).
//
// Maximin runs one thread-block cluster per problem.  The cluster's CTAs
// split the problem's points; each keeps, in shared memory, the squared
// float64 distances, float32 skip thresholds, exact coordinates and float32
// coordinates centred on the first row.  Every decision is the reference's:
//  * screening: a rigorous bound from bf16 images on the tensor cores, then
//    one from float32 images, skip a point only when the reference would not
//    update it;
//  * update: the squared distance s_new is computed in IEEE sequential
//    float64 exactly as ordering.py:52-57 does before its square root; the
//    point is updated when s_new < s_stored (bit compare).  With a correctly
//    rounded, monotone sqrt this keeps fl(sqrt(s_stored)) equal to the
//    reference's stored distance at every step: the reference updates only
//    when fl(sqrt(s_new)) < fl(sqrt(s_stored)), which implies s_new <
//    s_stored; an update here that the reference skips has
//    fl(sqrt(s_new)) == fl(sqrt(s_stored)) and leaves the root unchanged.
//    No square root is taken on this path;
//  * argmax: many pivots per pass, each provably the reference's next choice
//    (the comment above k_maximin_cluster gives the argument); candidate
//    lists meet through distributed shared memory after one hardware cluster
//    barrier per pass (double-buffered by pass parity), so there is no
//    spin-wait at all.
// Problems are grouped by cluster size (1, 2, 4, 8 or 16 CTAs: the smallest
// whose shared memory holds the problem, or more when the SMs have room for
// all problems side by side), one launch per group, largest problems first.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "sv_maximin_ops.cuh"
#include "sv_reorder.cuh"

namespace cg = cooperative_groups;

namespace sv {

constexpr int kMcThreads = 512;
constexpr int kMcWarps = kMcThreads / 32;
constexpr int kMcSlots = 32;  // candidate slots; slot 31 holds a pivot found by a full scan
// static shared memory of k_maximin_cluster (about 3.4 KB), rounded up: the
// capacity of a cluster is computed from what is left of 227 KB
constexpr int kMcStaticSmem = 4096;
constexpr int kMcMaxCluster = 16;
// work area: the warps' candidate lists (bits + index) or the pair distances
constexpr int kMcWorkBytes = ((kMcU * kMcU * 8 > kMcWarps * 32 * 12 ? kMcU * kMcU * 8 : kMcWarps * 32 * 12) + 15) & ~15;

// candidates of a pass from a level: the room of a CTA's list and of all
// lists, and the number of keys that the next level is set for
constexpr int kMcList = 96;
constexpr int kMcGather = 256;
constexpr int kMcTarget = 48;
static_assert(kMcGather <= kMcThreads && kMcGather * 12 <= kMcWorkBytes, "the gathered keys");

struct RoProb {
  int64_t n, xe_off, ye_off, ze_off, x_off, y_off, z_off, blk_off, first;
  int64_t xs_off;   // doubles: this call's scaled rows (and their maximin-order copy)
  int64_t v_off;    // floats: centred float32 rows [n][DP]
  int64_t row_off;  // rows: order, B
  int32_t d, q, m, DP, C, flags;
};

// per-point shared memory of the pass maximin: dist f64, exact coordinates
// f64[d] (cluster form only), thr f32, B f32, float32 centred coordinates f32[d]
__host__ __device__ inline int64_t mc_point_bytes(int d, bool grid = false) {
  return 16 + (grid ? 4 : 12) * (int64_t)d;
}
// coordinates of the bf16 images, zero padded to whole steps of the screen
__host__ __device__ inline int mc_d16(int d) { return d <= 16 ? 16 : d <= 32 ? 32 : 64; }
// per-CTA shared memory before the points: candidate slots (exact, float32 and
// bf16 coordinates, squared bits, index, bound) and the work area
__host__ __device__ inline int64_t mc_fixed_bytes(int d) {
  return (int64_t)kMcSlots * (12 * d + 16 + 2 * mc_d16(d)) + kMcWorkBytes;
}

__global__ void k_ro_info_init(int32_t* info, int nprob) {
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nprob; p += gridDim.x * blockDim.x) {
    info[4 * p + 0] = 0;
    info[4 * p + 1] = -1;
    info[4 * p + 2] = 0;
    info[4 * p + 3] = 0;
  }
}

// Xs = X_e / r; grid row = problem
__global__ void k_ro_scale(const RoProb* probs, const double* ranges, int dmax, const double* Xe,
                           double* Xs) {
  const RoProb& P = probs[blockIdx.y];
  const int d = P.d;
  const int64_t tot = P.n * d;
  const double* r = ranges + (int64_t)blockIdx.y * dmax;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < tot;
       e += (int64_t)gridDim.x * blockDim.x)
    Xs[P.xs_off + e] = __ddiv_rn(Xe[P.xe_off + e], r[e % d]);
}

// shared-memory layout of one CTA of the cluster maximin (identical in every
// CTA of a cluster, so remote reads use the same offsets)
struct McSmem {
  double* Ux;      // [32][d] exact coordinates of the candidate slots
  float* Uv;       // [32][d] their centred float32 images
  long long* Ub;   // [32] squared-distance bits at the start of the selection
  int* Ui;         // [32] row index
  float* UB;       // [32] float32 rounding bound of the image
  uint32_t* Uh;    // [32][d16 / 2] the images rounded to bf16
  double* pairS;   // [31][31] exact squared distances between candidates (work area)
  long long* wlb;  // [warps][32] candidate lists (work area)
  int* wli;
  double* dist;    // [Sc] squared distance to the ordered set; -1 once ordered
  const double* xs;  // [Sc][d] exact coordinates (shared memory, or the rows in global memory)
  float* thr;      // [Sc] float32 screening threshold
  float* Bp;       // [Sc] float32 rounding bound of the image
  float* v;        // [d][Sc] centred float32 images
};

// xg: the CTA's exact rows in global memory (grid form), or null to keep
// them in shared memory (cluster form)
__device__ __forceinline__ McSmem mc_layout(unsigned char* base, int d, int Sc, const double* xg) {
  McSmem L;
  L.Ux = (double*)base;
  L.Uv = (float*)(base + (size_t)kMcSlots * 8 * d);
  L.Ub = (long long*)(base + (size_t)kMcSlots * 12 * d);
  L.Ui = (int*)(L.Ub + kMcSlots);
  L.UB = (float*)(L.Ui + kMcSlots);
  L.Uh = (uint32_t*)(base + (size_t)kMcSlots * (12 * d + 16));
  unsigned char* work = (unsigned char*)(L.Uh + kMcSlots * (mc_d16(d) / 2));
  L.pairS = (double*)work;
  L.wlb = (long long*)work;
  L.wli = (int*)(work + kMcWarps * 32 * 8);
  unsigned char* pts = work + kMcWorkBytes;
  L.dist = (double*)pts;
  L.xs = xg ? xg : L.dist + Sc;
  L.thr = (float*)(L.dist + Sc + (xg ? 0 : (size_t)Sc * d));
  L.Bp = L.thr + Sc;
  L.v = L.Bp + Sc;
  return L;
}

// queue of (point << 5 | pivot) for the exact distances, in the work area
constexpr int kMcQueue = kMcWorkBytes / 4;

// pivot e & 31 against point e >> 5: the float32 screen, then the exact
// squared distance (ordering.py:52-57), which lowers the point's distance and
// threshold.  The result of a pass is the smallest of its distances, so the
// order in which the pivots are taken is free; an ordered point's -1 is below
// any distance, and stays.
__device__ __forceinline__ void mc_update(const McSmem& M, const int* slot, unsigned e, int Sc, int d,
                                          float growth) {
  const int p = (int)(e >> 5), u = slot[e & 31];
  float s32 = 0.0f;
  for (int l = 0; l < d; ++l) {
    const float df = __fsub_rn(M.v[(size_t)l * Sc + p], M.Uv[u * d + l]);
    s32 = __fmaf_rn(df, df, s32);
  }
  if (!mc_may_update(s32, *(volatile float*)(M.thr + p), M.UB[u], growth)) return;
  const double sn = sqdist_exact(M.xs + (size_t)p * d, M.Ux + u * d, d);
  const long long b = __double_as_longlong(sn);
  if (atomicMin((long long*)(M.dist + p), b) > b)
    atomicMin((int*)(M.thr + p), __float_as_int(thr_sq(sn, M.Bp[p])));  // thresholds of live points are >= 0
}

__device__ __forceinline__ uint32_t mc_bf16x2(float a, float b, float& sq) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  const float fa = __uint_as_float(r << 16), fb = __uint_as_float(r & 0xffff0000u);
  sq = fmaf(fa, fa, fmaf(fb, fb, sq));
  return r;
}

// The (point, pivot) pairs of this pass that may update, from the tensor
// cores.  With vb the images rounded to bf16, pivot j cannot lower point p when
//   ||vb_p - vb_j||^2 >= (thr_p + e_p + e_j)^2,
// e_p = kBf ||vb_p|| the rounding to bf16, e_j that and the image's own
// (which thr_p holds for the point).  The left side is
// |vb_p|^2 + |vb_j|^2 - 2 vb_p.vb_j: the products are exact in float32, and
// all sums together err by less than 2^-16 (|vb_p|^2 + |vb_j|^2); twice that
// is added to the right side, with the largest e_j and |vb_j|^2 of the pass.
// The accumulators start at -|vb_j|^2 / 2, so a pair is settled by one
// comparison with (|vb_p|^2 - right side) / 2; a NaN anywhere keeps the pair.
// The pairs left (a few per pass, once the distances are small) meet the
// float32 screen and the exact distance in mc_update.
// KT: 16-wide steps over the coordinates.  A warp takes 32 points x 32 pivots
// at a time; the 32 pivots' operands stay in registers.
constexpr float kBf = 0x1.01p-8f;  // half a unit of bf16's 8 bits, and the roundings of |vb|
constexpr float kBp = 0x1.02p16f;  // the same in Bp_p >= 2^-24 |v_p| (|vb| <= |v| (1 + 2^-8))
template <int KT>
__device__ __forceinline__ void mc_screen(const McSmem& M, const float* Un, const float* Ue, const int* slot,
                                          int* qn, int k, int S, int Sc, int d, float growth) {
  const int lane = threadIdx.x & 31, g = lane >> 2, c2 = (lane & 3) * 2;
  uint32_t B[4][KT][2];
  float C0[4][2];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int t = nt * 8 + g;
    const uint32_t* w = M.Uh + (t < k ? slot[t] : 0) * (KT * 8) + (lane & 3);
#pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
      B[nt][kt][0] = t < k ? w[kt * 8] : 0u;
      B[nt][kt][1] = t < k ? w[kt * 8 + 4] : 0u;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)  // no pivot: below every level
      C0[nt][i] = nt * 8 + c2 + i < k ? -0.5f * Un[slot[nt * 8 + c2 + i]] : __int_as_float(0xff800000);
  }
  unsigned em = 0, nm = 0;  // as bits: a NaN is the largest
  if (lane < k) {
    em = __float_as_uint(Ue[slot[lane]]) & 0x7fffffffu;
    nm = __float_as_uint(Un[slot[lane]]) & 0x7fffffffu;
  }
  const float emax = __uint_as_float(__reduce_max_sync(0xffffffffu, em));
  const float nmax = __uint_as_float(__reduce_max_sync(0xffffffffu, nm));
  const unsigned kmask = (1u << k) - 1;  // k <= 31
  for (int r0 = (threadIdx.x >> 5) * 32; r0 < S; r0 += blockDim.x) {
    uint32_t A[2][KT][4];
    float np[4] = {}, h[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float* v0 = M.v + min(r0 + g + 8 * x, S - 1);
#pragma unroll
      for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const int l = kt * 16 + y * 8 + c2;
          A[x >> 1][kt][2 * y + (x & 1)] = mc_bf16x2(l < d ? v0[(size_t)l * Sc] : 0.0f,
                                                     l + 1 < d ? v0[(size_t)(l + 1) * Sc] : 0.0f, np[x]);
        }
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) np[x] += __shfl_xor_sync(0xffffffffu, np[x], 1);
#pragma unroll
    for (int x = 0; x < 4; ++x) np[x] += __shfl_xor_sync(0xffffffffu, np[x], 2);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int p = min(r0 + g + 8 * x, S - 1);
      const float th = *(volatile float*)(M.thr + p);
      const float t = fmaf(kBp, M.Bp[p], th + emax);
      const float rhs = fmaf(t * t, 1.0f + 0x1p-12f, fmaf(0x1p-15f, np[x] + nmax, 1e-30f));
      h[x] = 0.5f * (np[x] - rhs);
      if (th < 0.0f || r0 + g + 8 * x >= S) h[x] = __int_as_float(0x7f800000);  // ordered: nothing
    }
    float acc[4][2][4];  // rows r0 + g + 16 x (+ 8)
    bool none = true;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        float(&c)[4] = acc[nt][x];
        c[0] = c[2] = C0[nt][0];
        c[1] = c[3] = C0[nt][1];
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
          asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
              "{%0,%1,%2,%3};"
              : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
              : "r"(A[x][kt][0]), "r"(A[x][kt][1]), "r"(A[x][kt][2]), "r"(A[x][kt][3]), "r"(B[nt][kt][0]),
                "r"(B[nt][kt][1]));
#pragma unroll
        for (int i = 0; i < 4; ++i) none = none && c[i] < h[2 * x + (i >> 1)];
      }
    if (!none) {
      unsigned bits[4] = {};  // rows r0 + g + 8 x
      int cnt = 0;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int i = 0; i < 2; ++i)
            bits[x] |= (acc[nt][x >> 1][2 * (x & 1) + i] < h[x] ? 0u : 1u) << (nt * 8 + i);
        bits[x] = h[x] == __int_as_float(0x7f800000) ? 0u : bits[x] << c2 & kmask;
        cnt += __popc(bits[x]);
      }
      int at = atomicAdd(qn, cnt);
      unsigned* queue = reinterpret_cast<unsigned*>(M.pairS);
#pragma unroll
      for (int x = 0; x < 4; ++x)
        for (unsigned m = bits[x]; m; m &= m - 1, ++at) {
          if (at < kMcQueue)  // (else the pass takes all pairs)
            queue[at] = (unsigned)(r0 + g + 8 * x) << 5 | (unsigned)(__ffs(m) - 1);
        }
    }
  }
}

// This pass's pivots (slots slot[0..k)) applied to the CTA's points.  The screen takes the thresholds of the
// pass start (upper bounds of every later one, so a pair that it settles
// cannot update); the pairs left are worked off by dense warps: a float64
// warp instruction costs the same with one active lane as with 32.
// 1,316 rows of d = 10 per CTA and 31 pivots: the float32 screen of every
// pair took 24,300 cycles, this 6,600.
__device__ __forceinline__ void mc_apply(const McSmem& M, const float* Un, const float* Ue, const int* slot,
                                         int* qn, int k, int S, int Sc, int d, float growth) {
  if (d <= 16)
    mc_screen<1>(M, Un, Ue, slot, qn, k, S, Sc, d, growth);
  else if (d <= 32)
    mc_screen<2>(M, Un, Ue, slot, qn, k, S, Sc, d, growth);
  else
    mc_screen<4>(M, Un, Ue, slot, qn, k, S, Sc, d, growth);
  __syncthreads();
  const int nq = *qn;
  if (nq <= kMcQueue) {
    const unsigned* queue = reinterpret_cast<const unsigned*>(M.pairS);
    for (int e = threadIdx.x; e < nq; e += blockDim.x) mc_update(M, slot, queue[e], Sc, d, growth);
  } else {
    // images that bf16 cannot tell apart, or the first passes: every pair meets
    // the float32 screen, a thread its points (one lane's pairs at a time, where
    // the queue was full, took 4.9 ms for 5,000 rows of a cluster and 52 rows
    // 1e6 times further out, this 3.5)
    for (int p = threadIdx.x; p < S; p += blockDim.x) {
      if (__double_as_longlong(M.dist[p]) < 0) continue;  // ordered
      for (int t = 0; t < k; ++t) mc_update(M, slot, (unsigned)p << 5 | (unsigned)t, Sc, d, growth);
    }
  }
  __syncthreads();
}

// One problem of the pass maximin.
struct McRun {
  const double* X;     // the problem's rows (scaled), n x d
  int64_t n;
  int64_t first;       // the first row of the order (ordering.py:72)
  int64_t* order;
  int32_t* info;       // the problem's 4 status words
  int32_t d, flags;
  // grid form: the iteration limit of a barrier wait, and a test aid: CTA 0
  // does not arrive at the first barrier, so every wait there runs out
  unsigned spin_limit;
  int32_t skip_first_arrival;
  // grid form: candidate lists of every CTA [2][G][32], their bounds [2][G],
  // and the monotone arrival counter of the grid barrier
  long long* gl_b;
  int* gl_i;
  long long* gl_Kb;
  int* gl_Ki;
  unsigned* arrive;
  // grid form: the keys above the level [3][kMcGather] and their counts [3]
  long long* gl_gb;
  int* gl_gi;
  unsigned* gl_gn;
};

// Maximin in passes.  A pass applies a batch of pivots, in order, to every
// unordered point (the reference's update, ordering.py:49-58, once per
// pivot), then chooses the next batch:
//  * the 31 largest keys (squared bits, then index) of all CTAs form the
//    candidate set U, and R bounds the squared bits of every other point
//    (the 32nd key and every thread's third-largest key);
//  * the exact squared distances between candidates (float32-screened) give
//    each candidate's value after any pivots taken from U;
//  * repeatedly the largest surviving candidate is the reference's next
//    pivot (ordering.py:42-47: largest root, then smallest index) as long as
//    its squared bits exceed R by more than 4 ulps: distinct squares with
//    equal roots lie within 3 ulps, so every point outside U then has a
//    smaller root.  Candidates within 4 ulps of the largest are ranked by
//    their exact roots;
//  * if not even the first choice is certain (many near-equal distances, as
//    on a lattice), a tie pass takes the points whose root equals the largest
//    root, in index order.
// The CTAs' lists meet through a hardware cluster barrier and distributed
// shared memory (cluster form, kGrid false), or through global memory and a
// grid barrier with bounded waits (grid form: one CTA per SM of a
// cooperative launch, exact rows read from global memory).  flags bit 0
// ranks every choice by exact roots, bit 1 runs a tie pass every time; both
// give the same order (test aids).
template <bool kGrid>
__device__ __forceinline__ void mc_run(const McRun& Q, int C, int r) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int64_t n = Q.n;
  const int d = Q.d;
  const double* X = Q.X;
  int64_t* order = Q.order;
  const int per = (int)((n + C - 1) / C);
  const int p0 = r * per;
  const int S = (int)max((int64_t)0, min(n, (int64_t)p0 + per) - p0);
  const int Sc = per;
  const McSmem M = mc_layout(smraw, d, Sc, kGrid ? X + (size_t)p0 * d : nullptr);
  __shared__ double cen[64];
  __shared__ long long cl_b[2][kMcList], cl_Kb[2];
  __shared__ int cl_i[2][kMcList], cl_Ki[2], cl_n[2];
  __shared__ long long w_Kb[kMcWarps];
  __shared__ int w_Ki[kMcWarps];
  __shared__ int piv_slot[kMcSlots];
  __shared__ float Uthr[kMcSlots], Un[kMcSlots], Ue[kMcSlots];
  __shared__ unsigned near_m[kMcSlots], s_red;
  __shared__ int s_k, s_tie, s_err, s_Ki, s_qn, s_abort, s_cnt, s_all, s_hold;
  __shared__ unsigned s_epoch;
  __shared__ long long s_Kb, s_top, s_level;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarp = blockDim.x >> 5;
  const float growth = mc_growth(d);
  const bool roots_always = (Q.flags & 1) != 0;
  const bool scan_always = (Q.flags & 2) != 0;

  // all CTAs of the problem: the hardware cluster barrier, or the grid
  // barrier (monotone arrival counter, bounded wait); false once a wait gave up
  auto all_sync = [&]() -> bool {
    if constexpr (kGrid) {
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        if (!(Q.skip_first_arrival && r == 0 && s_epoch == 0)) atomicAdd(Q.arrive, 1u);
        const unsigned target = (unsigned)C * ++s_epoch;
        unsigned it = 0;
        while (ld_acquire_u32(Q.arrive) < target) {
          if (++it > Q.spin_limit) {
            set_error(Q.info + SV_INFO_STATUS, SV_ETIMEOUT);
            s_abort = 1;
            break;
          }
        }
        __threadfence();
      }
      __syncthreads();
      return s_abort == 0;
    } else {
      if (C > 1)
        cg::this_cluster().sync();
      else
        __syncthreads();
      return true;
    }
  };
  // element l of row idx: exact coordinate and float32 image
  auto row_elem = [&](int idx, int l, double& x, float& vv) {
    if constexpr (kGrid) {
      x = X[(size_t)idx * d + l];
      vv = __double2float_rn(x - cen[l]);
    } else {
      const int owner = idx / per, loc = idx - owner * per;
      const double* xs = M.xs;
      const float* v = M.v;
      if (C > 1 && owner != r) {
        xs = cg::this_cluster().map_shared_rank(M.xs, owner);
        v = cg::this_cluster().map_shared_rank(M.v, owner);
      }
      x = xs[(size_t)loc * d + l];
      vv = v[(size_t)l * Sc + loc];
    }
  };
  // W lanes (16 for d <= 16, so that one float64 instruction serves two
  // slots, else a warp) bring the row of slot u (below 0: none): the exact
  // row, its float32 image and rounding bound, its bf16 image, that one's
  // squared norm and bound.  The whole warp calls it.
  const int W = d <= 16 ? 16 : 32;
  auto fetch_slot = [&](int u) {
    const int l0 = lane & (W - 1), D16 = mc_d16(d);
    float e2 = 0.0f, n2 = 0.0f;
    for (int l = l0; l < D16; l += W) {
      const bool on = u >= 0 && l < d;
      double x;
      float f;
      row_elem(on ? M.Ui[u] : (int)Q.first, on ? l : 0, x, f);
      if (!on) f = 0.0f;
      float sq = 0.0f;
      const uint32_t h = mc_bf16x2(f, __shfl_down_sync(0xffffffffu, f, 1), sq);
      e2 = __fmaf_ru(f, f, e2);
      if ((lane & 1) == 0) {
        n2 += sq;
        if (u >= 0) M.Uh[(u * D16 + l) >> 1] = h;
      }
      if (on) {
        M.Ux[u * d + l] = x;
        M.Uv[u * d + l] = f;
      }
    }
    for (int o = W >> 1; o > 0; o >>= 1) {
      e2 = __fadd_ru(e2, __shfl_xor_sync(0xffffffffu, e2, o));
      n2 += __shfl_xor_sync(0xffffffffu, n2, o);
    }
    if (l0 == 0 && u >= 0) {
      const float Bu = __fmul_ru(__fsqrt_ru(e2), 1.01f * 0x1p-24f);
      M.UB[u] = Bu;
      Un[u] = n2;
      Ue[u] = fmaf(kBf, sqrtf(n2), Bu);
      if (u < kMcU) Uthr[u] = thr_sq(__longlong_as_double(M.Ub[u]), Bu);
    }
  };
  // warp 0: slots piv_slot[0..kk) are the next pivots; their rows are ordered
  // (ordering.py:58) at positions at, at + 1, ...
  auto build_pivots = [&](int kk, int64_t at) {
    __syncwarp();
    if (lane < kk) {
      const int idx = M.Ui[piv_slot[lane]];
      if (r == 0) order[at + lane] = idx;
      if (idx >= p0 && idx < p0 + S) {
        M.dist[idx - p0] = -1.0;
        M.thr[idx - p0] = __int_as_float(0xff800000);
      }
    }
    if (lane == 0) {
      s_k = kk;
      s_qn = s_cnt = s_all = 0;
    }
  };

  // centre: the first row (any shift serves the float32 screen)
  for (int l = threadIdx.x; l < d; l += blockDim.x) cen[l] = X[Q.first * d + l];
  if (threadIdx.x == 0) {
    s_abort = 0;
    s_epoch = 0;
  }
  __syncthreads();
  if constexpr (!kGrid)
    for (int e = threadIdx.x; e < S * d; e += blockDim.x) const_cast<double*>(M.xs)[e] = X[(size_t)p0 * d + e];
  for (int p = threadIdx.x; p < S; p += blockDim.x) {
    const double* xp = X + (size_t)(p0 + p) * d;
    double e2 = 0.0;
    for (int l = 0; l < d; ++l) {
      const double c = xp[l] - cen[l];
      M.v[(size_t)l * Sc + p] = __double2float_rn(c);
      e2 += c * c;
    }
    M.Bp[p] = __double2float_ru(1.01 * 0x1p-24 * sqrt(e2));
    M.dist[p] = __longlong_as_double(0x7ff0000000000000LL);  // +inf: the first pass is exact
    M.thr[p] = __int_as_float(0x7f800000);
  }
  // every CTA's rows are in place before the first remote read
  if (!all_sync()) return;
  // the first pivot: row `first` (ordering.py:38-39) in slot 31
  if (warp == 0) {
    if (lane == 0) M.Ui[kMcU] = (int)Q.first;
    __syncwarp();
    fetch_slot(lane < W ? kMcU : -1);
    if (lane == 0) {
      piv_slot[0] = kMcU;
      s_err = 0;
      s_tie = 0;
      s_level = -1;
      s_hold = 0;
    }
    build_pivots(1, 0);
  }
  __syncthreads();

  // Candidate lists: from every thread's three largest keys (b1 > b2 > b3),
  // the 32 largest keys of all CTAs land in slots 0..31 (bits Ub, index Ui)
  // and (Kb, Ki) is the largest key that may belong to a point outside slots
  // 0..30: the 32nd key or a thread's third.  The same in every CTA.
  // False once a grid wait gave up.
  int par = 0;  // parity of the list buffers, flipped per collection
  auto collect = [&](long long b1, int i1, long long b2, int i2, long long b3, int i3,
                     long long& Kb, int& Ki) -> bool {
    mc_warp_sort2(b1, i1, b2, i2);
    mc_warp_merge(b1, i1, b2, i2);
    mc_warp_max(b3, i3);
    M.wlb[warp * 32 + lane] = b1;
    M.wli[warp * 32 + lane] = i1;
    if (lane == 0) {
      w_Kb[warp] = b3;
      w_Ki[warp] = i3;
    }
    __syncthreads();
    // a tree over the lists wlb[0..nwarp): warp w < s merges list w + s
    auto tree = [&]() {
      for (int s = nwarp >> 1; s >= 1; s >>= 1) {
        if (warp < s) {
          mc_warp_merge(b1, i1, M.wlb[(warp + s) * 32 + lane], M.wli[(warp + s) * 32 + lane]);
          if (s > 1) {
            M.wlb[warp * 32 + lane] = b1;
            M.wli[warp * 32 + lane] = i1;
          }
        }
        if (s > 1) __syncthreads();
      }
    };
    tree();
    long long kb = -1LL;
    int ki = kMcNone;
    if (warp == 0) {
      if (lane < nwarp) {
        kb = w_Kb[lane];
        ki = w_Ki[lane];
      }
      mc_warp_max(kb, ki);
    }
    if (C > 1) {
      // every CTA merges all lists (the same keys, so the same result
      // everywhere).  A buffer is rewritten two collections on, after the
      // next barrier, which no CTA passes before all have read it.
      if constexpr (kGrid) {
        if (warp == 0) {
          Q.gl_b[((size_t)par * C + r) * 32 + lane] = b1;
          Q.gl_i[((size_t)par * C + r) * 32 + lane] = i1;
          if (lane == 0) {
            Q.gl_Kb[par * C + r] = kb;
            Q.gl_Ki[par * C + r] = ki;
          }
        }
        if (!all_sync()) return false;
        // warp w merges the lists of CTAs w, w + nwarp, ... (next one in flight)
        b1 = -1LL;
        i1 = kMcNone;
        long long nb = -1LL;
        int ni = kMcNone;
        if (warp < C) {
          nb = __ldcg(Q.gl_b + ((size_t)par * C + warp) * 32 + lane);
          ni = __ldcg(Q.gl_i + ((size_t)par * C + warp) * 32 + lane);
        }
        for (int c = warp; c < C; c += nwarp) {
          const long long ob = nb;
          const int oi = ni;
          if (c + nwarp < C) {
            nb = __ldcg(Q.gl_b + ((size_t)par * C + c + nwarp) * 32 + lane);
            ni = __ldcg(Q.gl_i + ((size_t)par * C + c + nwarp) * 32 + lane);
          }
          mc_warp_merge(b1, i1, ob, oi);
        }
        if (warp == 0) {
          kb = -1LL;
          ki = kMcNone;
          for (int c = lane; c < C; c += 32) {
            const long long ob = __ldcg(Q.gl_Kb + par * C + c);
            const int oi = __ldcg(Q.gl_Ki + par * C + c);
            if (mc_greater(ob, oi, kb, ki)) {
              kb = ob;
              ki = oi;
            }
          }
          mc_warp_max(kb, ki);
        }
      } else {
        cg::cluster_group cluster = cg::this_cluster();
        if (warp == 0) {
          cl_b[par][lane] = b1;
          cl_i[par][lane] = i1;
          if (lane == 0) {
            cl_Kb[par] = kb;
            cl_Ki[par] = ki;
          }
        }
        cluster.sync();
        b1 = -1LL;
        i1 = kMcNone;
        if (warp < C) {
          // warp c brings the list of CTA c (one remote round trip for all)
          b1 = cluster.map_shared_rank(&cl_b[par][0], warp)[lane];
          i1 = cluster.map_shared_rank(&cl_i[par][0], warp)[lane];
        }
        if (warp == 0) {
          kb = -1LL;
          ki = kMcNone;
          if (lane < C) {
            kb = *cluster.map_shared_rank(&cl_Kb[par], lane);
            ki = *cluster.map_shared_rank(&cl_Ki[par], lane);
          }
          mc_warp_max(kb, ki);
        }
      }
      M.wlb[warp * 32 + lane] = b1;
      M.wli[warp * 32 + lane] = i1;
      __syncthreads();
      tree();
    }
    if (warp == 0) {
      const long long b32 = __shfl_sync(0xffffffffu, b1, 31);
      const int i32 = __shfl_sync(0xffffffffu, i1, 31);
      if (mc_greater(b32, i32, kb, ki)) {
        kb = b32;
        ki = i32;
      }
      M.Ub[lane] = b1;  // slot 31 is rewritten before any use
      M.Ui[lane] = i1;
      if (lane == 0) {
        s_Kb = kb;
        s_Ki = ki;
      }
    }
    __syncthreads();
    Kb = s_Kb;
    Ki = s_Ki;
    par ^= 1;
    return true;
  };
  // The same from a level, in the common case: the keys at or above it, some
  // 48 of all CTAs, are listed and every CTA ranks them by counting.  Slots
  // 0..30 and (Kb, Ki) are as from collect (with fewer than 32 keys, the level
  // bounds the others).  The level only decides how many candidates a pass
  // sees, not which order results; it is set from the keys' density in the
  // pass before.  found: the number of keys; none, or more than the lists
  // hold, and collect has to do it.  False once a grid wait gave up.
  // Sorting every thread's keys and merging all CTAs' lists took 20,000
  // cycles of a pass over 152 CTAs (11,400 over 4), this 3,700 (4,900).
  int tri = 0;  // grid form: the buffer of three; the one after next is cleared
  auto gather = [&](long long level, int& found, long long& Kb, int& Ki) -> bool {
    long long* gb = M.wlb;
    int* gi = (int*)(gb + kMcGather);
    for (int p = threadIdx.x; p < S; p += blockDim.x) {
      const long long b = __double_as_longlong(M.dist[p]);
      if (b < level || b >= 0x7ff0000000000000LL) continue;
      const int at = atomicAdd(&s_cnt, 1);
      if (at < kMcList) {
        cl_b[par][at] = b;
        cl_i[par][at] = p0 + p;
      }
    }
    __syncthreads();
    const int cnt = s_cnt, add = cnt > kMcList ? kMcGather + 1 : cnt;
    if constexpr (kGrid) {
      long long* kb = Q.gl_gb + tri * kMcGather;
      int* ki = Q.gl_gi + tri * kMcGather;
      if (warp == 0 && cnt > 0) {
        int base = lane == 0 ? (int)atomicAdd(Q.gl_gn + tri, (unsigned)add) : 0;
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int e = lane; e < min(cnt, kMcList) && base + e < kMcGather; e += 32) {
          kb[base + e] = cl_b[par][e];
          ki[base + e] = cl_i[par][e];
        }
      }
      if (!all_sync()) return false;
      found = (int)__ldcg(Q.gl_gn + tri);
      if (threadIdx.x < kMcGather) {
        gb[threadIdx.x] = __ldcg(kb + threadIdx.x);
        gi[threadIdx.x] = __ldcg(ki + threadIdx.x);
      }
      // all read this buffer before the next barrier, and write the cleared
      // one after it
      if (r == 0 && threadIdx.x == 0) Q.gl_gn[tri == 0 ? 2 : tri - 1] = 0;
      tri = tri == 2 ? 0 : tri + 1;
      __syncthreads();
    } else {
      if (C > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        if (threadIdx.x == 0) cl_n[par] = cnt;
        cluster.sync();
        if (warp < C) {
          const long long* kb = cluster.map_shared_rank(&cl_b[par][0], warp);
          const int* ki = cluster.map_shared_rank(&cl_i[par][0], warp);
          const int nc = *cluster.map_shared_rank(&cl_n[par], warp);
          long long b = kb[lane];  // (one remote round trip for all three)
          int i = ki[lane];
          int base = lane == 0 ? atomicAdd(&s_all, nc > kMcList ? kMcGather + 1 : nc) : 0;
          base = __shfl_sync(0xffffffffu, base, 0);
          for (int e = lane; e < min(nc, kMcList) && base + e < kMcGather; e += 32) {
            if (e >= 32) {
              b = kb[e];
              i = ki[e];
            }
            gb[base + e] = b;
            gi[base + e] = i;
          }
        }
        __syncthreads();
        found = s_all;
      } else {
        if (threadIdx.x < min(cnt, kMcList)) {
          gb[threadIdx.x] = cl_b[par][threadIdx.x];
          gi[threadIdx.x] = cl_i[par][threadIdx.x];
        }
        __syncthreads();
        found = add;
      }
    }
    par ^= 1;
    if (found < 1 || found > kMcGather) return true;
    // a key's slot is the number of keys above it: eight threads a key
    for (int t0 = 0; t0 < found; t0 += kMcThreads / 8) {
      const int t = t0 + (threadIdx.x >> 3);
      const long long b = t < found ? gb[t] : -1LL;
      const int i = t < found ? gi[t] : kMcNone;
      int above = 0;
      for (int j = threadIdx.x & 7; j < found; j += 8) above += mc_greater(gb[j], gi[j], b, i) ? 1 : 0;
      above += __shfl_xor_sync(0xffffffffu, above, 1);
      above += __shfl_xor_sync(0xffffffffu, above, 2);
      above += __shfl_xor_sync(0xffffffffu, above, 4);
      if (t < found && (threadIdx.x & 7) == 0 && above < 32) {
        M.Ub[above] = b;
        M.Ui[above] = i;
        if (above == 31) {
          s_Kb = b;
          s_Ki = i;
        }
      }
    }
    if (threadIdx.x < 32 && threadIdx.x >= found) {
      M.Ub[threadIdx.x] = -1LL;
      M.Ui[threadIdx.x] = kMcNone;
      if (threadIdx.x == 31) {
        s_Kb = level - 1;
        s_Ki = kMcNone;
      }
    }
    __syncthreads();
    Kb = s_Kb;
    Ki = s_Ki;
    return true;
  };
  // the candidates' rows, then the exact squared distances of the pairs of
  // them where either can lower the other: bit b of near_m[a] for such a
  // pair, its distance in pairS; -1 where a float32 upper bound already puts
  // either below R once the other is a pivot.  s_red: the slots that a slot
  // before them lowers.
  auto fetch_pairs = [&](double Rv) {
    for (int g = warp * (32 / W); g < kMcU; g += nwarp * (32 / W)) {
      const int u = g + lane / W;
      fetch_slot(u < kMcU && M.Ub[u] >= 0 ? u : -1);
    }
    if (threadIdx.x < kMcSlots) near_m[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_red = 0;
    __syncthreads();
    // pair t: slots x and x + 1 + y (mod 31), each pair once
    for (int t = threadIdx.x; t < kMcU * (kMcU / 2); t += blockDim.x) {
      const int x = t / (kMcU / 2);
      int y = x + 1 + (t - x * (kMcU / 2));
      y -= y >= kMcU ? kMcU : 0;
      const int a = min(x, y), b = max(x, y);
      if (M.Ub[b] < 0) continue;  // (the slots are filled in order)
      float s32 = 0.0f;
      for (int l = 0; l < d; ++l) {
        const float df = __fsub_rn(M.Uv[a * d + l], M.Uv[b * d + l]);
        s32 = __fmaf_rn(df, df, s32);
      }
      if (!mc_may_update(s32, Uthr[a], M.UB[b], growth) && !mc_may_update(s32, Uthr[b], M.UB[a], growth))
        continue;  // neither can lower the other
      double sp = -1.0;  // either, once the other is a pivot, falls below R: out of this pass
      if (!(Rv >= 0.0 && (double)mc_sq_upper(s32, M.UB[a], M.UB[b], growth) < Rv))
        sp = sqdist_exact(M.Ux + a * d, M.Ux + b * d, d);  // (x_a - x_b)^2 = (x_b - x_a)^2
      M.pairS[a * kMcU + b] = sp;
      M.pairS[b * kMcU + a] = sp;
      atomicOr(&near_m[a], 1u << b);
      atomicOr(&near_m[b], 1u << a);
      if (__double_as_longlong(sp) < M.Ub[b]) atomicOr(&s_red, 1u << b);
    }
    __syncthreads();
  };

  int64_t nsel = 1;
  while (nsel < n) {
    // 1. apply the pivots to this CTA's points
    const long long level = s_level;
    mc_apply(M, Un, Ue, piv_slot, &s_qn, s_k, S, Sc, d, growth);
    // 2. candidates U = slots 0..30; R bounds every other point's bits
    long long R = -1LL, low = level;
    int Ri = kMcNone, found = 0;
    if (level >= 0 && !gather(level, found, R, Ri)) return;  // a grid wait gave up
    const bool listed = found >= 1 && found <= kMcGather;
    if (!listed) {
      // from each thread's three largest keys, its points in index order
      long long b1 = -1, b2 = -1, b3 = -1;
      int i1 = kMcNone, i2 = kMcNone, i3 = kMcNone;
      for (int p = threadIdx.x; p < S; p += blockDim.x) {
        const long long b = __double_as_longlong(M.dist[p]);
        if (b < 0 || b >= 0x7ff0000000000000LL) continue;  // ordered, or not finite
        mc_insert3(b, p0 + p, b1, i1, b2, i2, b3, i3);
      }
      if (!collect(b1, i1, b2, i2, b3, i3, R, Ri)) return;
      low = R;
      found = 32;
    }
    fetch_pairs(R >= 0 ? __longlong_as_double(R) : -1.0);
    // 3. pivots from the candidates (warp 0, one candidate per lane)
    if (warp == 0) {
      long long sb = lane < kMcU ? M.Ub[lane] : -1LL;
      const int si = lane < kMcU ? M.Ui[lane] : kMcNone;
      const unsigned nearby = lane < kMcU ? near_m[lane] : 0u;
      bool alive = sb >= 0;
      const long long top = __shfl_sync(0xffffffffu, sb, 0);  // the largest square
      int kk = 0;
      if (!scan_always && !roots_always) {
        // the leading run of slots that are certain in list order: each is
        // above R + 4 ulps, more than 4 ulps above the next slot (no equal
        // root below it) and not lowered by a slot before it
        const bool red = (s_red >> lane & 1) != 0;  // (knock-outs are < 0)
        const long long nb = __shfl_down_sync(0xffffffffu, sb, 1);
        const bool near = lane + 1 < kMcU && nb >= 0 && nb >= sb - 4;
        const bool bad = lane >= kMcU || !alive || red || near || !(R < 0 || sb > R + 4);
        const int m = (int)min((int64_t)(__ffs(__ballot_sync(0xffffffffu, bad)) - 1), n - nsel);
        if (m > 0) {
          if (lane < m) {
            piv_slot[lane] = lane;
            alive = false;
          }
          for (unsigned w = nearby & ((1u << m) - 1); alive && w; w &= w - 1) {
            const long long sn = __double_as_longlong(M.pairS[lane * kMcU + __ffs(w) - 1]);
            if (sn < 0)
              alive = false;  // below R: cannot be chosen in this pass
            else if (sn < sb)
              sb = sn;
          }
          kk = m;
        }
      }
      while (!scan_always && kk < kMcU && nsel + kk < n) {
        // the largest key among the survivors: high word, low word, index
        const unsigned hi = alive ? (unsigned)((unsigned long long)sb >> 32) + 1u : 0u;
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        if (mh == 0) break;  // none left
        const unsigned lo = alive && hi == mh ? (unsigned)sb : 0u;
        const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
        const long long mb = ((long long)(mh - 1u) << 32) | (long long)ml;
        if (!(R < 0 || mb > R + 4)) break;  // not certain
        const bool is_max = alive && hi == mh && (unsigned)sb == ml;
        int mi = (int)__reduce_min_sync(0xffffffffu, is_max ? (unsigned)si : (unsigned)kMcNone);
        const unsigned nearm = __ballot_sync(0xffffffffu, alive && sb >= mb - 4 && si < mi);
        if (nearm || roots_always) {
          // equal roots: the smaller index (ordering.py:45 keeps the first maximum)
          long long rb = -1LL;
          int ri = kMcNone;
          if (alive && sb >= mb - 4) {
            rb = __double_as_longlong(__dsqrt_rn(__longlong_as_double(sb)));
            ri = si;
          }
          mc_warp_max(rb, ri);
          mi = ri;
        }
        const int ws = __ffs(__ballot_sync(0xffffffffu, alive && si == mi)) - 1;
        if (lane == 0) piv_slot[kk] = ws;
        if (lane == ws) alive = false;
        if (alive && (nearby >> ws & 1)) {
          const long long sn = __double_as_longlong(M.pairS[lane * kMcU + ws]);
          if (sn < 0)
            alive = false;  // below R after this pivot: cannot be chosen in this pass
          else if (sn < sb)
            sb = sn;
        }
        ++kk;
      }
      build_pivots(kk, nsel);
      if (lane == 0) {
        s_tie = kk == 0;
        s_top = top;
        // The next level: as far below R as kMcTarget keys at this pass's
        // density (in bits, so near enough in logarithms).  None after many
        // equal keys, and for a few passes after a level that failed.
        s_hold = level >= 0 && !listed ? 4 : max(0, s_hold - 1);
        long long next = -1LL;
        if (R < 0)
          next = top < 0 ? -1LL : 0LL;
        else if (top > low && s_hold == 0)
          next = max(0LL, R - ((top - low) / found + 1) * kMcTarget);
        s_level = next;
      }
    }
    __syncthreads();
    if (s_tie) {
      // 4. tie pass: no choice was certain, so many squares lie within 4 ulps
      //    of the largest, top.  The largest root is fl(sqrt(top)); the points
      //    with that root, T, are the reference's next choices in index order
      //    (ordering.py:45) while they keep it.  Slots 0..30 take the 31
      //    smallest indices of T; any other member of T has an index >= the
      //    bound Ki.
      const long long top = s_top;
      if (top < 0) {
        // no finite candidate left (NaN inputs): report and stop
        if (threadIdx.x == 0) {
          s_err = 1;
          if (r == 0) {
            set_error(Q.info + SV_INFO_STATUS, SV_EINVAL);
            Q.info[SV_INFO_BLOCK] = (int)nsel;
          }
        }
      } else {
        const long long rmax = __double_as_longlong(__dsqrt_rn(__longlong_as_double(top)));
        long long b1 = -1, b2 = -1, b3 = -1;
        int i1 = kMcNone, i2 = kMcNone, i3 = kMcNone;
        for (int p = threadIdx.x; p < S; p += blockDim.x) {
          const double dp = M.dist[p];
          const long long bits = __double_as_longlong(dp);
          if (bits < 0 || bits > top || bits < top - 4) continue;
          if (__double_as_longlong(__dsqrt_rn(dp)) != rmax) continue;
          // key: the smaller index first; the low 3 bits carry top - bits
          mc_insert3(((1LL << 40) - (p0 + p)) * 8 + (top - bits), p0 + p, b1, i1, b2, i2, b3, i3);
        }
        long long Kb;
        int Ki;
        if (!collect(b1, i1, b2, i2, b3, i3, Kb, Ki)) return;
        const int bound = Kb >= 0 ? Ki : kMcNone;
        // the slots' squares from their keys
        if (threadIdx.x < kMcU && M.Ub[threadIdx.x] >= 0) M.Ub[threadIdx.x] = top - (M.Ub[threadIdx.x] & 7);
        __syncthreads();
        fetch_pairs(-1.0);
        if (warp == 0) {
          long long sb = lane < kMcU ? M.Ub[lane] : -1LL;
          const int si = lane < kMcU ? M.Ui[lane] : kMcNone;
          const unsigned nearby = lane < kMcU ? near_m[lane] : 0u;
          bool alive = sb >= 0, tied = alive;
          int kk = 0;
          while (kk < kMcU && nsel + kk < n) {
            const int mi = (int)__reduce_min_sync(0xffffffffu, alive && tied ? (unsigned)si : (unsigned)kMcNone);
            if (mi == kMcNone || mi >= bound) break;
            const int ws = __ffs(__ballot_sync(0xffffffffu, alive && si == mi)) - 1;
            if (lane == 0) piv_slot[kk] = ws;
            if (lane == ws) alive = false;
            if (alive && (nearby >> ws & 1)) {
              const double sn = M.pairS[lane * kMcU + ws];
              if (__double_as_longlong(sn) < sb) {
                sb = __double_as_longlong(sn);
                if (tied) tied = __double_as_longlong(__dsqrt_rn(sn)) == rmax;
              }
            }
            ++kk;
          }
          build_pivots(kk, nsel);
        }
      }
      __syncthreads();
    }
    if (s_err) break;  // the same value in every CTA
    nsel += s_k;
  }
  // keep this CTA's shared memory alive until every remote read is done
  if constexpr (!kGrid)
    if (C > 1) cg::this_cluster().sync();
}

__global__ void __launch_bounds__(kMcThreads, 1) k_maximin_cluster(const RoProb* probs,
                                                                   const int32_t* plist,
                                                                   const double* Xs, int64_t* ord,
                                                                   int32_t* info) {
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int pid = plist[blockIdx.x / C];
  const RoProb& P = probs[pid];
  McRun Q = {};
  Q.X = Xs + P.xs_off;
  Q.n = P.n;
  Q.first = P.first;
  Q.order = ord + P.row_off;
  Q.info = info + 4 * pid;
  Q.d = P.d;
  Q.flags = P.flags;
  mc_run<false>(Q, C, (int)cluster.block_rank());
}

// grid form: one problem over a cooperative grid (one CTA per SM)
__global__ void __launch_bounds__(kMcThreads, 1) k_maximin_grid(McRun Q) {
  mc_run<true>(Q, (int)gridDim.x, (int)blockIdx.x);
}



// X, y, Z <- rows of X_e, y_e, Z_e in maximin order; Xso <- Xs in that order;
// grid row = problem
__global__ void k_ro_permute(const RoProb* probs, const int64_t* ord, const double* Xe,
                             const double* ye, const double* Ze, const double* Xs, double* X,
                             double* y, double* Z, double* Xso, int64_t* order_out) {
  const RoProb& P = probs[blockIdx.y];
  const int d = P.d, q = P.q;
  const int64_t* o = ord + P.row_off;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t src = o[i];
    for (int l = 0; l < d; ++l) {
      X[P.x_off + i * d + l] = Xe[P.xe_off + src * d + l];
      Xso[P.xs_off + P.n * d + i * d + l] = Xs[P.xs_off + src * d + l];
    }
    y[P.y_off + i] = ye[P.ye_off + src];
    for (int c = 0; c < q; ++c) Z[P.z_off + i * q + c] = Ze[P.ze_off + src * q + c];
    if (order_out) order_out[P.row_off + i] = src;
  }
}

// centred float32 rows (zero padded to DP) and their rounding bound for the
// kNN screen, centre = row 0 of the ordered problem; grid row = problem
__global__ void k_ro_knn_prep(const RoProb* probs, const double* Xso, float* v, float* B) {
  const RoProb& P = probs[blockIdx.y];
  const int d = P.d, DP = P.DP;
  const double* X = Xso + P.xs_off + P.n * d;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < P.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    double e2 = 0.0;
    for (int l = 0; l < DP; ++l) {
      float f = 0.0f;
      if (l < d) {
        const double c = X[i * d + l] - X[l];
        f = __double2float_rn(c);
        e2 += c * c;
      }
      v[P.v_off + i * DP + l] = f;
    }
    B[P.row_off + i] = __double2float_ru(1.01 * 0x1p-24 * sqrt(e2));
  }
}

static size_t ro_align(size_t x) { return (x + 255) & ~(size_t)255; }

static int ro_max_smem() {
  int dev = 0, v = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  return v;
}

static int launch_maximin_cluster(int C, size_t smem, unsigned nclusters, const RoProb* probs,
                                  const int32_t* plist, const double* Xs, int64_t* ord,
                                  int32_t* info, cudaStream_t st);

// largest cluster the device can schedule with a full shared-memory budget
// per CTA (16 needs the non-portable cluster size; else 8)
static int g_mc_max_cluster = 0;
static int mc_max_cluster() {
  if (g_mc_max_cluster) return g_mc_max_cluster;
  int C = 8;
  if (cudaFuncSetAttribute(k_maximin_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
      cudaSuccess) {
    const int smem = ro_max_smem() - kMcStaticSmem;
    cudaFuncSetAttribute(k_maximin_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kMcMaxCluster);
    cfg.blockDim = dim3(kMcThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kMcMaxCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int nclus = 0;
    if (cudaOccupancyMaxActiveClusters(&nclus, (void*)k_maximin_cluster, &cfg) == cudaSuccess && nclus > 0)
      C = kMcMaxCluster;
  }
  cudaGetLastError();  // a refused query leaves no error behind
  g_mc_max_cluster = C;
  return C;
}

// cluster size for n rows of dimension d: 1, 2, 4, 8 (or 16), or 0 when none fits
static int mc_cluster_size(int64_t n, int d, int maxsm) {
  const int64_t budget = (int64_t)maxsm - kMcStaticSmem - mc_fixed_bytes(d);
  const int cmax = mc_max_cluster();
  for (int C = 1; C <= cmax; C *= 2) {
    const int64_t per = (n + C - 1) / C;
    if (per * mc_point_bytes(d) <= budget) return C;
  }
  return 0;
}

// the same for a problem that has the SMs to itself: up to 16 CTAs while one
// has more rows than threads.  A pass's screen and scans shrink with a CTA's
// rows, its exchange hardly grows: 5,000 rows of d = 8 take 2.65 ms on 4
// CTAs (all that their memory needs), 2.30 on 16; 60,000 of d = 1 55.9 and
// 36.6; but 300 rows 0.39 on one and 0.44 on two.
static int mc_spread(int64_t n, int C) {
  while (C > 0 && C < mc_max_cluster() && n > (int64_t)C * kMcThreads) C *= 2;
  return C;
}

struct RoPlan {
  std::vector<RoProb> probs;
  std::vector<KnnBatchProb> kprobs;
  std::vector<int32_t> plist[5];   // problems per cluster size 1, 2, 4, 8, 16
  size_t smem[5] = {0, 0, 0, 0, 0};
  std::vector<int2> tiles[8];      // kNN tiles per padded dimension
  int DPs[8] = {4, 8, 12, 16, 24, 32, 48, 64};
  int kcap[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int trows[8] = {128, 128, 128, 128, 128, 128, 128, 128};  // kNN tile heights
  int64_t nrows = 0, nxs = 0, nv = 0;
  // workspace layout
  size_t o_probs, o_kprobs, o_plist[5], o_tiles[8], o_ranges, o_xs, o_v, o_b, o_ord, total, staged;
};

static int ro_plan(const sv_reorder_desc* D, const sv_reorder_prob* hp, RoPlan& L) {
  const int maxsm = ro_max_smem();
  const int64_t np = D->nprob;
  L.probs.resize(np);
  L.kprobs.resize(np);
  int64_t spread = 0;
  for (int64_t i = 0; i < np; ++i) {
    const sv_reorder_prob& U = hp[i];
    if (U.n < 0 || U.d < 1 || U.d > D->dmax || U.d > 64 || U.q < 0 || U.m < 0 || U.m > D->ldnbr ||
        (U.n > 0 && (U.first < 0 || U.first >= U.n)) || U.n > 0x7fffffffLL)
      return SV_EINVAL;
    RoProb& R = L.probs[i];
    R.n = U.n;
    R.xe_off = U.xe_off;
    R.ye_off = U.ye_off;
    R.ze_off = U.ze_off;
    R.x_off = U.x_off;
    R.y_off = U.y_off;
    R.z_off = U.z_off;
    R.blk_off = U.blk_off;
    R.first = U.first;
    R.d = U.d;
    R.q = U.q;
    R.m = U.m;
    R.flags = U.flags & 3;  // maximin test aids: exact roots always (1), full scans (2)
    R.DP = knn_pad_dim(U.d);
    R.C = mc_cluster_size(U.n, U.d, maxsm);
    if (R.C == 0) return SV_EINVAL;
    spread += mc_spread(U.n, R.C);
    R.xs_off = L.nxs;
    L.nxs += 2 * U.n * U.d;  // scaled rows, then the same rows in maximin order
    R.v_off = L.nv;
    L.nv += U.n * R.DP;
    R.row_off = L.nrows;
    L.nrows += U.n;
    KnnBatchProb& K = L.kprobs[i];
    K.xs_off = R.xs_off + U.n * U.d;
    K.v_off = R.v_off;
    K.row_off = R.row_off;
    K.n = U.n;
    K.blk_off = U.blk_off;
    K.d = U.d;
    K.m = U.m;
  }
  if (spread <= sv_num_sms())  // room for all of them at once
    for (RoProb& R : L.probs) R.C = mc_spread(R.n, R.C);
  // largest problems first in every launch
  std::vector<int32_t> byn(np);
  for (int64_t i = 0; i < np; ++i) byn[i] = (int32_t)i;
  std::stable_sort(byn.begin(), byn.end(),
                   [&](int32_t a, int32_t b) { return L.probs[a].n > L.probs[b].n; });
  for (int32_t i : byn) {
    const RoProb& R = L.probs[i];
    if (R.n < 1) continue;
    const int g = R.C == 1 ? 0 : R.C == 2 ? 1 : R.C == 4 ? 2 : R.C == 8 ? 3 : 4;
    L.plist[g].push_back(i);
    const size_t sm = (size_t)((R.n + R.C - 1) / R.C) * (size_t)mc_point_bytes(R.d) +
                      (size_t)mc_fixed_bytes(R.d);
    L.smem[g] = std::max(L.smem[g], sm);
    if (R.m < 1 || R.n < 2) continue;
    int gi = 0;
    while (L.DPs[gi] != R.DP) ++gi;
    L.kcap[gi] = std::max(L.kcap[gi], R.m);
  }
  // kNN tiles (largest problems and, within one, the last rows first), of the
  // height the search of each padded dimension takes
  for (int g = 0; g < 8; ++g)
    L.trows[g] = L.kcap[g] > 0 ? knn_batched_tile_rows(L.DPs[g], L.kcap[g]) : 128;
  for (int32_t i : byn) {
    const RoProb& R = L.probs[i];
    if (R.n < 1 || R.m < 1 || R.n < 2) continue;
    int gi = 0;
    while (L.DPs[gi] != R.DP) ++gi;
    const int64_t nt = (R.n + L.trows[gi] - 1) / L.trows[gi];
    for (int64_t t = nt - 1; t >= 0; --t) L.tiles[gi].push_back(make_int2(i, (int)t));
  }
  // workspace: staged tables first, then the arrays
  size_t off = 0;
  L.o_probs = off;
  off = ro_align(off + sizeof(RoProb) * (size_t)np);
  L.o_kprobs = off;
  off = ro_align(off + sizeof(KnnBatchProb) * (size_t)np);
  for (int g = 0; g < 5; ++g) {
    L.o_plist[g] = off;
    off = ro_align(off + sizeof(int32_t) * L.plist[g].size());
  }
  for (int g = 0; g < 8; ++g) {
    L.o_tiles[g] = off;
    off = ro_align(off + sizeof(int2) * L.tiles[g].size());
  }
  L.o_ranges = off;
  off = ro_align(off + sizeof(double) * (size_t)np * D->dmax);
  L.staged = off;
  L.o_xs = off;
  off = ro_align(off + sizeof(double) * (size_t)L.nxs);
  L.o_v = off;
  off = ro_align(off + sizeof(float) * (size_t)L.nv);
  L.o_b = off;
  off = ro_align(off + sizeof(float) * (size_t)L.nrows);
  L.o_ord = off;
  off = ro_align(off + sizeof(int64_t) * (size_t)L.nrows);
  L.total = off;
  return SV_OK;
}

static int launch_maximin_cluster(int C, size_t smem, unsigned nclusters, const RoProb* probs,
                                  const int32_t* plist, const double* Xs, int64_t* ord,
                                  int32_t* info, cudaStream_t st) {
  SV_CUDA_TRY(cudaFuncSetAttribute(k_maximin_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nclusters * (unsigned)C);
  cfg.blockDim = dim3(kMcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SV_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_maximin_cluster, probs, plist, Xs, ord, info));
  return SV_OK;
}

// One problem through the cluster kernel (sv_maximin_order for n that fits
// one cluster).  ws: 256 bytes of device scratch.
int maximin_cluster_single(const double* X, int64_t n, int d, int64_t first, int64_t* order,
                           int32_t* info, char* ws, int flags, cudaStream_t st) {
  const int C = mc_spread(n, mc_cluster_size(n, d, ro_max_smem()));
  if (C == 0) return SV_EINVAL;
  struct {
    RoProb p;
    int32_t plist[4];
  } h;
  memset(&h, 0, sizeof(h));
  h.p.n = n;
  h.p.first = first;
  h.p.d = d;
  h.p.C = C;
  h.p.flags = flags & 3;
  SV_CUDA_TRY(cudaMemcpyAsync(ws, &h, sizeof(h), cudaMemcpyHostToDevice, st));
  const size_t smem = (size_t)((n + C - 1) / C) * (size_t)mc_point_bytes(d) + (size_t)mc_fixed_bytes(d);
  return launch_maximin_cluster(C, smem, 1, (const RoProb*)ws, (const int32_t*)(ws + sizeof(RoProb)),
                                X, order, info, st);
}

// grid form: CTAs (one per SM at most, >= 64 rows each) and rows per CTA
static int mg_plan(int64_t n, int d, int& G, int& per, size_t& smem) {
  const int nsm = sv_num_sms();
  const int64_t budget = (int64_t)ro_max_smem() - kMcStaticSmem - mc_fixed_bytes(d);
  G = (int)std::min<int64_t>(nsm, std::max<int64_t>(1, (n + 63) / 64));
  per = (int)((n + G - 1) / G);
  if ((int64_t)per * mc_point_bytes(d, true) > budget) return SV_EINVAL;
  smem = (size_t)per * (size_t)mc_point_bytes(d, true) + (size_t)mc_fixed_bytes(d);
  return SV_OK;
}

size_t maximin_grid_workspace_bytes() {
  const size_t g2 = 2 * (size_t)sv_num_sms();
  return ro_align(g2 * 32 * 8) + ro_align(g2 * 32 * 4) + ro_align(g2 * 8) + ro_align(g2 * 4) +
         ro_align(3 * kMcGather * 8) + ro_align(3 * kMcGather * 4) + 256;
}

int64_t maximin_grid_max_rows(int d) {
  if (d < 1 || d > 64) return 0;
  const int64_t budget = (int64_t)ro_max_smem() - kMcStaticSmem - mc_fixed_bytes(d);
  return (int64_t)sv_num_sms() * (budget / mc_point_bytes(d, true));
}

// One problem through the grid form (a cooperative launch, one CTA per SM).
int maximin_grid_single(const double* X, int64_t n, int d, int64_t first, int64_t* order,
                        int32_t* info, char* ws, size_t ws_bytes, int flags, cudaStream_t st) {
  int G = 0, per = 0;
  size_t smem = 0;
  if (mg_plan(n, d, G, per, smem) != SV_OK) return SV_EINVAL;
  if (ws_bytes < maximin_grid_workspace_bytes()) return SV_ENOSPC;
  SV_CUDA_TRY(cudaFuncSetAttribute(k_maximin_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int active = 0;
  SV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&active, k_maximin_grid, kMcThreads, smem));
  if (active < 1 || G > active * sv_num_sms()) return SV_EINVAL;
  const size_t g2 = 2 * (size_t)sv_num_sms();
  McRun Q = {};
  Q.X = X;
  Q.n = n;
  Q.first = first;
  Q.order = order;
  Q.info = info;
  Q.d = d;
  Q.flags = flags & 3;
  Q.skip_first_arrival = (flags & 8) ? 1 : 0;
  Q.spin_limit = (flags & 8) ? SV_SPIN_LIMIT_TEST : SV_SPIN_LIMIT;
  size_t off = 0;
  Q.gl_b = (long long*)(ws + off);
  off += ro_align(g2 * 32 * 8);
  Q.gl_i = (int*)(ws + off);
  off += ro_align(g2 * 32 * 4);
  Q.gl_Kb = (long long*)(ws + off);
  off += ro_align(g2 * 8);
  Q.gl_Ki = (int*)(ws + off);
  off += ro_align(g2 * 4);
  Q.gl_gb = (long long*)(ws + off);
  off += ro_align(3 * kMcGather * 8);
  Q.gl_gi = (int*)(ws + off);
  off += ro_align(3 * kMcGather * 4);
  Q.arrive = (unsigned*)(ws + off);
  Q.gl_gn = Q.arrive + 32;  // a line of its own
  SV_CUDA_TRY(cudaMemsetAsync(Q.arrive, 0, 256, st));
  void* args[] = {&Q};
  SV_CUDA_TRY(cudaLaunchCooperativeKernel((void*)k_maximin_grid, dim3((unsigned)G), dim3(kMcThreads), args,
                                          smem, st));
  return SV_OK;
}

// Helper streams for launches that do not depend on one another (the
// maximin launches of the cluster sizes, the neighbour-search launches of the
// dimension classes): each launch lasts as long as its largest problem, so
// running them side by side costs the longest instead of the sum.  Created
// once per device; every call forks them off its own stream with an event and
// joins them back before the work that needs their results.  Calls from
// several host threads at once may serialise on the helpers, never misorder.
constexpr int kRoHelpers = 7;
constexpr int kRoMaxDevices = 64;
static cudaStream_t g_ro_helper[kRoMaxDevices][kRoHelpers];
static bool g_ro_helper_made[kRoMaxDevices];
static std::mutex g_ro_mu;

static int ro_helper_streams(cudaStream_t* out) {
  std::lock_guard<std::mutex> lk(g_ro_mu);
  int dev = 0;
  SV_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kRoMaxDevices) return SV_EINVAL;
  if (!g_ro_helper_made[dev]) {
    for (int i = 0; i < kRoHelpers; ++i)
      SV_CUDA_TRY(cudaStreamCreateWithFlags(&g_ro_helper[dev][i], cudaStreamNonBlocking));
    g_ro_helper_made[dev] = true;
  }
  for (int i = 0; i < kRoHelpers; ++i) out[i] = g_ro_helper[dev][i];
  return SV_OK;
}

// helpers hs[0 .. n-1] wait for the work enqueued on st so far
static int ro_fork(cudaStream_t st, const cudaStream_t* hs, int n) {
  if (n <= 0) return SV_OK;
  cudaEvent_t e;
  SV_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  SV_CUDA_TRY(cudaEventRecord(e, st));
  for (int i = 0; i < n; ++i) SV_CUDA_TRY(cudaStreamWaitEvent(hs[i], e, 0));
  SV_CUDA_TRY(cudaEventDestroy(e));
  return SV_OK;
}

// st waits for the work enqueued on hs[0 .. n-1] so far
static int ro_join(cudaStream_t st, const cudaStream_t* hs, int n) {
  for (int i = 0; i < n; ++i) {
    cudaEvent_t e;
    SV_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    SV_CUDA_TRY(cudaEventRecord(e, hs[i]));
    SV_CUDA_TRY(cudaStreamWaitEvent(st, e, 0));
    SV_CUDA_TRY(cudaEventDestroy(e));
  }
  return SV_OK;
}

int64_t maximin_cluster_max_rows(int d) {
  if (d < 1 || d > 64) return 0;
  const int64_t budget = (int64_t)ro_max_smem() - kMcStaticSmem - mc_fixed_bytes(d);
  return (int64_t)mc_max_cluster() * (budget / mc_point_bytes(d));
}

}  // namespace sv

using namespace sv;

extern "C" int64_t sv_maximin_cluster_max_rows(int32_t d) { return maximin_cluster_max_rows(d); }

extern "C" size_t sv_reorder_batched_workspace_bytes(const sv_reorder_desc* D,
                                                     const sv_reorder_prob* probs) {
  if (!D || (D->nprob > 0 && !probs) || D->nprob < 0) return 0;
  RoPlan L;
  if (ro_plan(D, probs, L) != SV_OK) return 0;
  return L.total;
}

extern "C" int sv_reorder_batched(const sv_reorder_desc* D, const sv_reorder_prob* probs,
                                  const double* ranges, const double* Xe, const double* ye,
                                  const double* Ze, double* X, double* y, double* Z, int32_t* nbr,
                                  int64_t* order, int32_t* info, void* workspace,
                                  size_t workspace_bytes, sv_stream_t stream) {
  if (!D || D->nprob < 0 || D->dmax < 1 || D->dmax > 64 || D->ldnbr < 0 || !info) return SV_EINVAL;
  if (D->nprob == 0) return SV_OK;
  if (!probs || !ranges || !Xe || !ye || !X || !y) return SV_EINVAL;
  RoPlan L;
  int rc = ro_plan(D, probs, L);
  if (rc != SV_OK) return rc;
  bool anyq = false, anym = false;
  for (const RoProb& R : L.probs) {
    anyq = anyq || R.q > 0;
    anym = anym || (R.m > 0 && R.n > 1);
  }
  if ((anyq && (!Ze || !Z)) || (anym && (!nbr || D->ldnbr < 1))) return SV_EINVAL;
  if (!workspace || workspace_bytes < L.total) return SV_ENOSPC;
  cudaStream_t st = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  const int np = (int)D->nprob;

  // one staged copy of every table
  std::vector<char> host(L.staged, 0);
  memcpy(host.data() + L.o_probs, L.probs.data(), sizeof(RoProb) * np);
  memcpy(host.data() + L.o_kprobs, L.kprobs.data(), sizeof(KnnBatchProb) * np);
  for (int g = 0; g < 5; ++g)
    if (!L.plist[g].empty())
      memcpy(host.data() + L.o_plist[g], L.plist[g].data(), sizeof(int32_t) * L.plist[g].size());
  for (int g = 0; g < 8; ++g)
    if (!L.tiles[g].empty())
      memcpy(host.data() + L.o_tiles[g], L.tiles[g].data(), sizeof(int2) * L.tiles[g].size());
  memcpy(host.data() + L.o_ranges, ranges, sizeof(double) * (size_t)np * D->dmax);
  SV_CUDA_TRY(cudaMemcpyAsync(ws, host.data(), L.staged, cudaMemcpyHostToDevice, st));
  const RoProb* dprobs = (const RoProb*)(ws + L.o_probs);
  double* Xs = (double*)(ws + L.o_xs);
  float* v = (float*)(ws + L.o_v);
  float* B = (float*)(ws + L.o_b);
  int64_t* ord = (int64_t*)(ws + L.o_ord);

  k_ro_info_init<<<(np + 255) / 256, 256, 0, st>>>(info, np);
  SV_CUDA_TRY(cudaGetLastError());
  int64_t maxn = 0;
  for (const RoProb& R : L.probs) maxn = std::max(maxn, R.n);
  int64_t gx = (maxn * D->dmax + 255) / 256;
  gx = std::max<int64_t>(1, std::min<int64_t>(gx, 64));
  k_ro_scale<<<dim3((unsigned)gx, np), 256, 0, st>>>(dprobs, (const double*)(ws + L.o_ranges),
                                                      D->dmax, Xe, Xs);
  SV_CUDA_TRY(cudaGetLastError());

  cudaStream_t hs[kRoHelpers];
  if ((rc = ro_helper_streams(hs)) != SV_OK) return rc;
  // maximin: one launch per cluster size, side by side (the first on st)
  {
    int used = 0;
    for (int g = 0; g < 5; ++g) used += L.plist[g].empty() ? 0 : 1;
    const int nh = used > 1 ? used - 1 : 0;
    if ((rc = ro_fork(st, hs, nh)) != SV_OK) return rc;
    int slot = 0;
    for (int g = 0; g < 5; ++g) {
      if (L.plist[g].empty()) continue;
      cudaStream_t sg = slot == 0 ? st : hs[slot - 1];
      ++slot;
      rc = launch_maximin_cluster(1 << g, L.smem[g], (unsigned)L.plist[g].size(), dprobs,
                                  (const int32_t*)(ws + L.o_plist[g]), (const double*)Xs, ord, info, sg);
      if (rc != SV_OK) return rc;
    }
    if ((rc = ro_join(st, hs, nh)) != SV_OK) return rc;
  }

  gx = (maxn + 255) / 256;
  gx = std::max<int64_t>(1, std::min<int64_t>(gx, 64));
  k_ro_permute<<<dim3((unsigned)gx, np), 256, 0, st>>>(dprobs, ord, Xe, ye, Ze, Xs, X, y, Z, Xs, order);
  SV_CUDA_TRY(cudaGetLastError());
  k_ro_knn_prep<<<dim3((unsigned)gx, np), 256, 0, st>>>(dprobs, Xs, v, B);
  SV_CUDA_TRY(cudaGetLastError());
  // neighbour search: one launch per dimension class, side by side
  {
    int used = 0;
    for (int g = 0; g < 8; ++g) used += L.tiles[g].empty() ? 0 : 1;
    const int nh = used > 1 ? used - 1 : 0;
    if ((rc = ro_fork(st, hs, nh)) != SV_OK) return rc;
    int slot = 0;
    for (int g = 0; g < 8; ++g) {
      if (L.tiles[g].empty()) continue;
      cudaStream_t sg = slot == 0 ? st : hs[slot - 1];
      ++slot;
      rc = launch_knn_batched(L.DPs[g], (const KnnBatchProb*)(ws + L.o_kprobs),
                              (const int2*)(ws + L.o_tiles[g]), (int64_t)L.tiles[g].size(), Xs, v, B,
                              nbr, D->ldnbr, L.kcap[g], sg);
      if (rc != SV_OK) return rc;
    }
    if ((rc = ro_join(st, hs, nh)) != SV_OK) return rc;
  }
  return SV_OK;
}
