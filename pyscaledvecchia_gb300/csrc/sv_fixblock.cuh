// Team-level factorisation of the fixed-point block kernel (sv_loglik_fix.cu).
//
// A team of G lanes owns one block of at most G points, lane i its row i: a
// whole warp (G = 32), or half of one (G = 16), whose warp runs two blocks in
// step: every loop is warp-uniform up to the larger block's size, so the
// shuffles and barriers are reached by all lanes (work beyond a block's own
// size is never stored).
#pragma once
#include "sv_fix.cuh"
#include "sv_loglik.cuh"

namespace sv {

constexpr int kFixPanel = 4;         // columns per panel
constexpr int kFixPivotShift = 34;   // pivots below 2^-34 of the unit diagonal: the float64 kernels
constexpr int kFixHead = 2;          // bits of growth left in a row of the inverse at first,
constexpr int kFixStep = 4;          // and added where an element does not fit
constexpr unsigned kFull = 0xffffffffu;

template <int G>
struct FixDim {
  static constexpr int kSt = G + 2;  // even: a panel's rows of a column are 16-byte aligned
  static constexpr int kCs = G + 1;  // column stride of the solutions (odd: conflict-free)
};

template <int G>
__device__ __forceinline__ int team_max(int v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(kFull, v, o, G));
  return v;
}
// four consecutive split numbers, 16-byte aligned
__device__ __forceinline__ void load4(const Fx2* p, Fx2 (&v)[4]) {
  const int4 a = *(const int4*)p, b = *(const int4*)(p + 2);
  v[0].h = a.x; v[0].l = a.y; v[1].h = a.z; v[1].l = a.w;
  v[2].h = b.x; v[2].l = b.y; v[3].h = b.z; v[3].l = b.w;
}

// The products of low limbs that fx_mac leaves out average to nothing in a sum
// of products of different numbers, but in a row's sum of squares (its pivot)
// they are all positive, a third of a unit each. fx_sq adds one up (in units
// of 2^-50 of Q58's), fx_sq_val is their sum in Q58.
__device__ __forceinline__ void fx_sq(int64_t& s, Fx2 x) {
  const int t = x.l >> 4;
  s += (int64_t)t * t;
}
__device__ __forceinline__ int64_t fx_sq_val(int64_t s) { return (s + (1ll << 49)) >> 50; }

// x where keep is -1, 0 where it is 0: by a mask the compiler cannot see
// through (it would otherwise select between whole products)
__device__ __forceinline__ Fx2 fx_keep(Fx2 x, int keep) {
  asm("" : "+r"(keep));
  x.h &= keep;
  x.l &= keep;
  return x;
}

// The inverse of the Cholesky factor of a unit-scaled covariance S = C C^T.
//
// Left-looking by panels of columns: row i of C takes
// C_ik = (S_ik - sum_{j<k} C_ij C_kj) / C_kk for k <= i, and row i of the
// identity the same recurrence, T_ki = (0 - sum_{i<=j<k} T_ji C_kj) / C_kk for
// k > i, T_ii = 1 / C_ii, where T = C^-1. Lane i is at work on its row of C
// while k <= i and on its column of T after that: one set of accumulators, one
// broadcast of C's rows k, all lanes busy throughout; the factor and its
// inverse cost what the factor alone does with a lane per row.
//
// M (column stride kSt): S_ij as a plain Q58 integer at M[j kSt + i], i >= j,
// on entry. On return (split Q58) C_ij there for i > j, and T_ji 2^-E_i at
// M[j kSt + i] for j >= i; the exponent E_i is lane i's result E, its C_ii the
// result cd. An element of T that would leave its row's scale rescales the
// row. The return value is the smallest pivot (Q58; when that lies
// below 2^-34 the rest is meaningless: the caller leaves the block to the
// float64 kernels), 0 when rescaling does not help.
template <int G>
__device__ __forceinline__ int64_t fix_factor(int K, int Kw, int tl, Fx2* M, int64_t& cd, int& E) {
  constexpr int St = FixDim<G>::kSt;
  int64_t dmin = 1ll << 58, sq = 0;
  E = 0;
  cd = 0;
  for (int k0 = 0; k0 < Kw; k0 += kFixPanel) {
    FxAcc acc[kFixPanel];
#pragma unroll
    for (int w = 0; w < kFixPanel; ++w) acc[w] = {0, 0};
    const Fx2* col = M;
    const int j0 = tl < k0 ? tl : 0;  // a row of T starts at its own column
#pragma unroll 4
    for (int j = 0; j < k0; ++j, col += St) {
      Fx2 b[4];
      load4(col + k0, b);
      const Fx2 x = fx_keep(col[tl], (j0 - 1 - j) >> 31);
#pragma unroll
      for (int w = 0; w < kFixPanel; ++w) fx_mac(acc[w], x, b[w]);
    }
#pragma unroll
    for (int w = 0; w < kFixPanel; ++w) {
      const int k = k0 + w;
      if (k >= Kw) break;
      Fx2* ck = M + k * St + tl;
      int64_t v = 0;
      if (tl >= k && tl < K) v = *(const int64_t*)ck;
      v -= fx_val(acc[w]);
      if (tl == k) v -= fx_sq_val(sq);
      int64_t d = __shfl_sync(kFull, (long long)v, k, G);
      if (k < K && d < dmin) dmin = d;
      if (d < (1ll << (58 - kFixPivotShift)) || d > (1ll << 58)) d = 1ll << 58;
      int e;
      const int64_t Yq = fx_rsqrt_pivot(d, e);
      const Fx2 Y = fx_split(Yq);
      if (tl < k && k < K) {
        int tries = 0;
        int hi = (int)(v >> 32);
        while (((hi ^ (hi >> 31)) >> (26 - e)) != 0) {  // |v| 2^e >= 2^58
          if (++tries > 20) {
            dmin = 0;
            v = 0;
            break;
          }
          E += kFixStep;
          for (int j = tl; j < k; ++j) M[j * St + tl] = fx_split(fx_join(M[j * St + tl]) >> kFixStep);
#pragma unroll
          for (int w2 = 0; w2 < kFixPanel; ++w2) {
            acc[w2].h >>= kFixStep;
            acc[w2].m >>= kFixStep;
          }
          v >>= kFixStep;
          hi = (int)(v >> 32);
        }
      }
      int64_t x = fx_mul(fx_split((int64_t)((uint64_t)v << e)), Y);
      if (tl == k) {
        cd = x;
        E = e + kFixHead;
        x = Yq >> kFixHead;
#pragma unroll
        for (int w2 = w + 1; w2 < kFixPanel; ++w2) acc[w2] = {0, 0};
      }
      const Fx2 c = fx_split(x);
      if (tl > k) fx_sq(sq, c);
      if (tl < K && k < K) *ck = c;
#pragma unroll
      for (int w2 = w + 1; w2 < kFixPanel; ++w2) {
        Fx2 b;
        b.h = __shfl_sync(kFull, c.h, k0 + w2, G);
        b.l = __shfl_sync(kFull, c.l, k0 + w2, G);
        fx_mac(acc[w2], c, b);
      }
    }
    // nothing left but blocks that are not kept
    if (__all_sync(kFull, dmin < (1ll << (58 - kFixPivotShift)) || k0 + kFixPanel >= K)) break;
    __syncwarp();
  }
  __syncwarp();
  return dmin;
}

// a = C^-T e_K as us 2^su, |us| < 1/2: row K of T, then one step of refinement,
// a + T^T (e_K - C^T a). The row's own errors are those of separate solves;
// the residual's are those of a back substitution, which smooth combinations
// of a (a.Z for a trend column Z, a.y) do not feel. On return the rows of C are
// zeroed: M holds T alone. Returns false when the residual is not small.
template <int G>
__device__ __forceinline__ bool fix_last_row(int K, int Kw, int tl, Fx2* M, int64_t cd, int E, Fx2* us, int& su, Fx2& usi) {
  constexpr int St = FixDim<G>::kSt;
  const bool own = tl < K;
  int64_t x = own ? fx_join(M[(K - 1) * St + tl]) : 0;
  su = team_max<G>(own ? fx_bits(x) + E : -100000) - 57;
  x = own ? fx_scale2(x, E - su) : 0;
  usi = fx_split(x);
  us[tl] = usi;
  __syncwarp();
  FxAcc acc = {0, 0};
  fx_mac(acc, fx_split(cd), usi);
  Fx2* col = M + (own ? tl : 0) * St;
#pragma unroll 4
  for (int i = 1; i < K; ++i) {
    fx_mac(acc, fx_keep(col[i], (tl - i) >> 31), us[i]);
  }
  const int64_t r = (own && tl == K - 1 ? fx_scale2(1ll << 58, -su) : 0) - fx_val(acc);
  const bool ok = !own || (r < (1ll << 30) && r > -(1ll << 30));
  const int r32 = own && ok ? (int)r : 0;
  int64_t dl = 0;
  const Fx2* tc = M + tl;
#pragma unroll 4
  for (int k = 0; k < Kw; ++k, tc += St) {
    const int rk = __shfl_sync(kFull, r32, k, G);
    if (k >= tl && k < K) dl += (int64_t)tc->h * rk;
  }
  x += fx_scale2(dl, E - 28);
  usi = fx_split(own ? x : 0);
  us[tl] = usi;
  if (own)
    for (int i = tl + 1; i < K; ++i) col[i] = {0, 0};
  __syncwarp();
  return ok;
}

}  // namespace sv
