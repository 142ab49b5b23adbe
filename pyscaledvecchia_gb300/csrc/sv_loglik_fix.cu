// The fixed-point block kernel of the Vecchia likelihood / score / Fisher
// evaluation: the float64 form's kernel for blocks of at most 32 points with
// Matern smoothness 3/2 or 5/2 (d <= 12, at most 32 right-hand sides).
//
// Same per-block record as k_block_warp (likelihood.py:111-144 of the
// reference), from arithmetic at least as fine as float64's: every quantity
// with a known bound is a 64-bit integer in units of 2^-58 or so of that bound
// (sv_fix.cuh). k_block_warp is bound by the float64 pipe (64 cycles per warp
// instruction and scheduler, 2,310 of them per block of 31); here the pipe is
// left with the coordinate differences and the conversion of the results, and
// the work is on the integer multiply-adds (4 cycles each).
//
//   * coordinates centred on the block's own point, in units of 2^-61 of 4 to
//     8 times the block's largest coordinate; r^2 as the exact sum of the
//     squared differences, with an exponent of its own;
//   * the covariance is scaled by its own variance and a power of two,
//     Sigma = s2 2^ek (M 2^-ek + tau 2^-ek I), so that its diagonal lies in
//     (1/2, 1] and its Cholesky factor's entries are below 1 whatever the
//     conditioning: the backward error of the factorisation is about 2^-57 of
//     the diagonal, where float64's is about K 2^-53;
//   * the factor's inverse T comes with it (fix_factor): its last row is
//     a = C^-T e_K, and the solves W = C^-1 V are products with T;
//   * dSigma_l a = sum_j g_ij (U_i - U_j)^2 a_j from the differences as well,
//     every pair's in units of the pair's own distance 2^E (their square
//     joins g, which is bounded however far the points): errors of 2^-58 of
//     the variance at any extent. (As three matrix products, U_i^2 (G a)_i -
//     2 U_i (G aU)_i + (G aU^2)_i, they were 2^-58 of the extent's square, and
//     it takes as many multiply-adds);
//   * rows of T, right-hand sides and solutions carry power-of-two scales.
//
// Measured at n = 200,000, d = 10, m = 30: 11.2 ms (d = 8: 9.6, d = 12: 11.8), where
// k_block_warp takes 27.3 ms; the integer multiply pipe is 61 to 65 % busy, the
// float64 pipe 6 % (3 warps per scheduler, one block of 17 KB of shared memory
// each; at 200,000 blocks a tenth of the warps' waits are for instructions).
//
// Errors against binary128 (float64 kernels in brackets), n = 240, m = 30, rows
// evenly spread, in clusters of six 0.02 ranges across, or three times each,
// reaching 0.5 to 30 ranges, tau = 1e-8 to 0.1, d = 3 and 8: log-likelihood, score
// and Fisher as close as the float64 kernels' or closer, but for single results
// of 1e-16 to 1e-15; clusters, d = 3, 10 ranges, tau = 1e-8: log-likelihood 1e-13
// (3e-12), score 2e-12 (3e-11), Fisher 3e-12 (7e-11). n = 200,000, d = 10, tau =
// 3e-3: log-likelihood 4e-17 (4e-15).
//
// What has no such bound goes to the float64 kernels: a block with a pivot
// below 2^-34 of the diagonal (its jitter ladder is theirs), coordinates
// beyond 32 ranges of the block's own point, non-finite or huge data, another
// smoothness. The choice depends on the block and its problem alone, so a
// block has the same bits in every launch that holds it.
#include "sv_fixblock.cuh"

namespace sv {

constexpr int kFixThreads = 384;
constexpr int kFixV = 6;  // inputs per pass over the pairs' g at most
constexpr int kFixEsMin = -27;  // smallest unit of the coordinates (pairs' exponents are bytes)

__device__ __forceinline__ double pow2(int n) {
  return n < -1022 ? 0.0 : __longlong_as_double((long long)(min(n, 1023) + 1023) << 52);
}

// shared memory of one team, in 8-byte words.  rs: words per point of the
// coordinates (padded to a multiple of 4 inputs) and of the right-hand sides
// that replace them; 2 more than a multiple of 4, so that eight lanes' 16-byte
// loads of the same entries of consecutive points meet all banks once
__host__ __device__ inline int fix_g_words(int G, int kcap, int ncol) {
  const int g = kcap * (kcap - 1) / 2, w = (G + 1) * ncol;  // pairs' g, then the solutions
  return ((g > w ? g : w) + 1) & ~1;
}
// exponents of the pairs' distances (at most 496 bytes), then the columns'
// scales and last rows
constexpr int kFixPWords = 2 * kFixCols;
__host__ __device__ inline int fix_slot_words(int G, int kcap, int ncol, int rs) {
  int s = kcap * (G + 2);            // M
  s += fix_g_words(G, kcap, ncol);
  s += rs * kcap;                    // coordinates, then right-hand sides
  s += kFixPWords;
  s += G;                            // a
  return (s + 1) & ~1;
}

template <int G>
struct FixSlot {
  Fx2* M;
  Fx2* Gp;   // g 2^(2 E) of the pairs i > j at i(i-1)/2 + j; then the solutions (column stride kCs)
  signed char* Ep;  // their E
  Fx2* cv;   // [point][rs]
  Fx2* us;
  int rs;
};

// Sigma / (s2 2^ek) below the diagonal of M and g: in round r lane i takes
// the pair (i, i + r mod K), so each unordered pair is met once; two rounds at
// a time, whose chains of dependent products overlap
template <int G, int CODE>
__device__ __forceinline__ void fix_assemble(int K, int d, int tl, int es, int ek, const FixSlot<G>& S,
                                             const uint64_t* T) {
  constexpr int St = FixDim<G>::kSt;
  Fx2 ui[kFixMaxD];
#pragma unroll
  for (int g = 0; g < kFixMaxD; g += 4)
    if (g < d) {
#pragma unroll
      for (int l = g; l < g + 4; ++l) ui[l] = S.cv[tl * S.rs + l];
    }
  for (int r = 1; 2 * r <= K; r += 2) {
    int jj[2], E[2];
    uint64_t s[2], m[2], g[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      int j = tl + r + t;
      if (j >= K) j -= K;
      if (2 * (r + t) > K || (2 * (r + t) == K && tl >= r + t)) j = tl;  // no such pair
      jj[t] = j;
      const Fx2* uj = S.cv + j * S.rs;
      FxSq q = {0, 0, 0};
#pragma unroll
      for (int g4 = 0; g4 < kFixMaxD; g4 += 4)
        if (g4 < d) {
          Fx2 v[4];
          load4(uj + g4, v);
          if (g4 == 8) fx_sqcarry(q);
#pragma unroll
          for (int l = 0; l < 4; ++l) fx_sqdiff(q, ui[g4 + l], v[l]);
        }
      s[t] = fx_sqnorm(q, es, E[t]);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) fx_matern_norm<CODE, true>(s[t], E[t], T, m[t], g[t]);
#pragma unroll
    for (int t = 0; t < 2; ++t)
      if (jj[t] != tl) {
        const int lo = min(tl, jj[t]), hi = max(tl, jj[t]);
        *(int64_t*)(S.M + lo * St + hi) = (int64_t)((m[t] + (4ull << ek)) >> (3 + ek));
        S.Gp[hi * (hi - 1) / 2 + lo] = fx_split((int64_t)((g[t] + 4) >> 3));
        S.Ep[hi * (hi - 1) / 2 + lo] = (signed char)E[t];
      }
  }
}

// a right-hand side (this lane's element x, in units 2^-58, its row of T at
// scale 2^E): stored as split x 2^(E - f), below 1/2, f being the result
template <int G>
__device__ __forceinline__ int fix_put_rhs(int64_t x, int E, bool own, Fx2* p) {
  const int f = team_max<G>(own ? fx_bits(x) + E : -100000) - 57;
  if (own) *p = fx_split(fx_scale2(x, E - f));
  return f;
}

// dSigma_l a for NV inputs l0 .. l0 + NV - 1, in place of their coordinates
// (plain Q61 integers here); fc[l] their scales. Each unordered pair is met
// once, as in fix_assemble: lane i squares the difference to i + r, and lane
// i + r has the square from it by a shuffle. The square in units of the pair's
// 2^(2 E) is at most 1 (Q62; 2: the mean of what is dropped below it, 0 for equal
// rows), its weight g 2^(2 E) a_j below 0.75 (Q58)
template <int G, int NV>
__device__ __forceinline__ void fix_dsig(int K, int Kw, int d, int l0, int tl, int es, int E, const FixSlot<G>& S,
                                         int& fc) {
  const bool own = tl < K;
  const int i = own ? tl : 0;
  Fx2* cv = S.cv + i * S.rs;
  int64_t U[NV];
#pragma unroll
  for (int t = 0; t < NV; ++t) U[t] = *(const int64_t*)(cv + l0 + t);
  int64_t ah[NV], am[NV];  // Q58, Q88
#pragma unroll
  for (int t = 0; t < NV; ++t) ah[t] = am[t] = 0;
#pragma unroll 1
  for (int r = 1; 2 * r <= Kw; ++r) {
    const bool fwd = own && 2 * r <= K, rev = own && 2 * r < K;
    int j = i + r, jr = i - r;
    if (j >= K) j -= K;
    if (jr < 0) jr += K;
    if (!fwd) j = i;
    if (!rev) jr = i;
    const int hi = max(i, j), at = fwd ? hi * (hi - 1) / 2 + min(i, j) : 0;
    const int hr = max(i, jr), ar = rev ? hr * (hr - 1) / 2 + min(i, jr) : 0;
    const Fx2 w = fx_keep(fx_split(fx_mul(S.Gp[at], S.us[j])), fwd ? -1 : 0);
    const Fx2 wr = fx_keep(fx_split(fx_mul(S.Gp[ar], S.us[jr])), rev ? -1 : 0);
    const int k = es + 2 - S.Ep[at];
    const Fx2* uj = S.cv + j * S.rs + l0;
#pragma unroll
    for (int t = 0; t < NV; t += 2) {
      const longlong2 v = *(const longlong2*)(uj + t);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int64_t D = (int64_t)((uint64_t)(U[t + u] - (u ? v.y : v.x)) << (k & 63));  // Q63
        const int h = (int)(D >> 32), l = (int)((uint32_t)D >> 1);
        const int64_t q = (int64_t)h * h + 2 + (((int64_t)h * l) >> 30);
        const int qh = (int)(q >> 32), ql = (int)((uint32_t)q >> 2);
        const int rh = __shfl_sync(kFull, qh, jr, G), rl = __shfl_sync(kFull, ql, jr, G);
        ah[t + u] += (int64_t)w.h * qh;
        ah[t + u] += (int64_t)wr.h * rh;
        am[t + u] += (int64_t)w.h * ql;
        am[t + u] += (int64_t)w.l * qh;
        am[t + u] += (int64_t)wr.h * rl;
        am[t + u] += (int64_t)wr.l * rh;
      }
    }
    if ((r & 3) == 3) {  // the middle sums hold 9 pairs' at least
#pragma unroll
      for (int t = 0; t < NV; ++t) {
        ah[t] += am[t] >> 30;
        am[t] &= (1ll << 30) - 1;
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int t = 0; t < NV; ++t)
    if (l0 + t < kFixMaxD) {
      const bool put = own && l0 + t < d;
      const int f = fix_put_rhs<G>(ah[t] + ((am[t] + (1ll << 29)) >> 30), E, put, cv + l0 + t);
      if (tl == l0 + t) fc = f;
    }
  __syncwarp();
}

template <int G>
__global__ void __launch_bounds__(kFixThreads, 1) k_block_fix(LikArgs A, int wpc, int ncap, int rs, int kmin) {
  extern __shared__ double smem[];
  constexpr int St = FixDim<G>::kSt, Cs = FixDim<G>::kCs, NB = 32 / G;
  uint64_t* T = (uint64_t*)smem;
  for (int i = threadIdx.x; i < 256; i += blockDim.x) T[i] = kFxExp2[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tm = lane / G, tl = lane % G;
  const int kcap = A.kcap < G ? A.kcap : G;
  FixSlot<G> S;
  S.M = (Fx2*)(smem + 256 + (int64_t)(warp * NB + tm) * fix_slot_words(G, kcap, ncap, rs));
  S.Gp = S.M + kcap * St;
  S.cv = S.Gp + fix_g_words(G, kcap, ncap);
  double* scg = (double*)(S.cv + rs * kcap);  // column scales and last rows, after dSigma a
  S.Ep = (signed char*)scg;
  S.us = (Fx2*)scg + kFixPWords;
  S.rs = rs;
  double* wkd = scg + kFixCols;  // w_K of the parameters, then z_K of y and Z

  const int64_t nb = A.b1 - A.b0;
  const int64_t stride = (int64_t)gridDim.x * wpc * NB;
  for (int64_t base = ((int64_t)blockIdx.x * wpc + warp) * NB; base < nb; base += stride) {
    const int64_t tix = base + tm;
    bool active = tix < nb;
    const int64_t b = active ? launch_block(A, A.b0 + tix) : 0;
    const int pid = active ? block_problem(A, b) : 0;
    const ProbInfo& PI = A.probs[pid];
    if (active && PI.skip) active = false;
    int K = active ? A.kb[b] + 1 : 0;
    if (K <= kmin) active = false;  // another launch's
    if (active && K > 32) {
      if (tl == 0) set_error(A.info + 4 * pid + SV_INFO_STATUS, SV_EINVAL);
      active = false;
    }
    // fix_ek < 0: a problem this kernel does not take
    if (active && (PI.fix_ek < 0 || K > kcap)) {
      if (K <= 16 || G == 32 || A.kcap <= 16) {  // else the 32-lane launch's
        if (tl == 0) {
          A.level[b] = 0;
          A.redo[b] = 1;
          A.flags[1] = 1;
        }
      }
      active = false;
    }
    if (!active) K = 0;
    const int Kw = __reduce_max_sync(kFull, K);
    if (Kw == 0) continue;
    const int d = PI.d, q = PI.q, P = PI.P;
    bool bad = false;  // to the float64 kernels
    auto leave = [&](bool redo) {
      if (active && tl == 0) {
        A.level[b] = 0;
        A.redo[b] = redo ? 1 : 0;
        if (redo) A.flags[1] = 1;
      }
      __syncwarp();
    };
    const int ek = PI.fix_ek;
    const bool own = tl < K;

    // ---- gather: neighbours first, self last; coordinates centred on self,
    //      a lane takes its own row, all its loads in flight at once
    int row = 0, exm = 0;
    if (own) row = (tl < K - 1) ? A.nbr[b * A.ldnbr + tl] : A.rowb[b];
    {
      const int self = __shfl_sync(kFull, row, K > 0 ? K - 1 : 0, G);
      const double* xi = A.X + PI.x_off + (int64_t)row * d;
      const double* xs = A.X + PI.x_off + (int64_t)self * d;
      double v[kFixMaxD];
#pragma unroll
      for (int l = 0; l < kFixMaxD; ++l) v[l] = (own && l < d) ? xi[l] - xs[l] : 0.0;
#pragma unroll
      for (int l = 0; l < kFixMaxD; ++l)
        if (l < d) {
          v[l] *= PI.invlam[l];
          exm = max(exm, (int)((dbits(v[l]) >> 52) & 0x7ff));
        }
      exm = team_max<G>(exm);
      if (exm > 1023 + 4) {  // |u| >= 32, infinities, NaN
        bad = true;
        exm = 2046;
      }
      exm = max(exm, kFixEsMin + 1023 - 3);
      // Q61 with |U| < 1/4
#pragma unroll
      for (int g = 0; g < kFixMaxD; g += 4)
        if (g < d) {
#pragma unroll
          for (int l = g; l < g + 4; ++l) {
            const Fx2 u = fx_split(fx_from_bits<6>(dbits(v[l]), exm));
            if (own) S.cv[tl * rs + l] = u;
          }
        }
    }
    // no work on blocks that are not kept: 100,000 of them beyond 32 ranges,
    // each computed twice in full, took 13.2 ms where the float64 kernels alone
    // take 9.2, now 9.5; with pivots below the limit 13.1, now 10.3
    if (__all_sync(kFull, bad || !active)) {
      leave(bad);
      continue;
    }
    const int es = bad ? 0 : exm - 1023 + 3;  // |u| 2^-es < 1/4
    if (own) *(int64_t*)(S.M + tl * St + tl) = PI.fix_diag;
    __syncwarp();

    if (own) {
      if (PI.closed == 1)
        fix_assemble<G, 1>(K, d, tl, es, ek, S, T);
      else
        fix_assemble<G, 2>(K, d, tl, es, ek, S, T);
    }
    __syncwarp();

    // ---- C C^T = Sigma / (s2 2^ek), T = C^-1
    int E, su;
    int64_t cd;
    const int64_t dmin = fix_factor<G>(K, Kw, tl, S.M, cd, E);
    bad |= dmin < (1ll << (58 - kFixPivotShift));
    if (__all_sync(kFull, bad || !active)) {
      leave(bad);
      continue;
    }
    Fx2 usi;
    bad |= !fix_last_row<G>(K, Kw, tl, S.M, cd, E, S.us, su, usi);

    // ---- right-hand sides: d inputs, nugget, y, q trend columns; fc: scale
    //      of the column tl (fc2: tl + G)
    int fc = 0, fc2 = 0;
    Fx2* cv = S.cv + tl * rs;
    if (A.need_grad) {
      const int dw = __reduce_max_sync(kFull, active ? d : 0);
      if (own) {
#pragma unroll
        for (int l = 0; l < kFixMaxD; ++l)
          if (l < ((d + 3) & ~3)) *(int64_t*)(cv + l) = fx_join(cv[l]);
      }
      __syncwarp();
      int l0 = 0;
#pragma unroll 1
      for (; l0 + 4 < dw; l0 += kFixV) fix_dsig<G, kFixV>(K, Kw, d, l0, tl, es, E, S, fc);
      if (l0 + 2 < dw)
        fix_dsig<G, 4>(K, Kw, d, l0, tl, es, E, S, fc);
      else if (l0 < dw)
        fix_dsig<G, 2>(K, Kw, d, l0, tl, es, E, S, fc);
      const int f = fix_put_rhs<G>(fx_join(usi), E, own, cv + d);  // nugget: s2 tau a
      if (tl == d) fc = f;
    }
    double* rec = A.cache + b * (int64_t)A.CS;
    const double rsig = PI.fix_rsig;
    const int np = d + 1;  // columns before y: parameters 1 .. d + 1
    double* zk = wkd + np;
    const int qw = __reduce_max_sync(kFull, active ? q : 0);
    for (int c = 0; c <= qw; ++c) {
      const bool in = own && c <= q;
      int64_t x = 0;
      if (in) x = dbits(c == 0 ? A.y[PI.y_off + row] : A.Z[PI.z_off + (int64_t)row * q + (c - 1)]);
      const int em = team_max<G>((int)((x >> 52) & 0x7ff));
      if (em > 1023 + 600) bad = true;
      x = fx_from_bits<5>(x, em);  // units 2^(em - 1022 - 58)
      // a.y, a.Z = (L^-1 y)_K, (L^-1 Z)_K (likelihood.py:129-134)
      FxAcc p = {0, 0};
      if (in) fx_mac(p, usi, fx_split(x));
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {
        p.h += __shfl_xor_sync(kFull, (long long)p.h, o, G);
        p.m += __shfl_xor_sync(kFull, (long long)p.m, o, G);
      }
      if (active && c <= q && tl == 0) {
        const double az = (double)fx_val(p) * (rsig * pow2(em - 1022)) * pow2(su - 58);
        rec[1 + c] = az;
        rec[2 + q + c] = az;
        zk[c] = az;
      }
      if (A.need_grad) {
        const int f = fix_put_rhs<G>(x, E, in, cv + np + c) + em - 1022;
        if (np + c == tl) fc = f;
        if (np + c == tl + G) fc2 = f;
      }
    }
    if (own && tl == K - 1) rec[0] = PI.fix_sig * ((double)cd * pow2(-58));  // L_KK
    __syncwarp();
    if (A.need_grad) {
      // ---- W = C^-1 V = T V (likelihood.py:139, 154): lane k its row of T
      //      and of every column, four columns at a time; kept at the scale
      //      of the column's largest element
      const int NR = d + 2 + q;
      const int NRw = __reduce_max_sync(kFull, active ? NR : 0);
      const double pu = pow2(su - ek);
      Fx2* W = S.Gp;
      const Fx2* tr = S.M + (own ? tl : 0) * St;
      for (int c0 = 0; c0 < NRw; c0 += 4) {
        FxAcc acc[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) acc[w] = {0, 0};
        const Fx2* vj = S.cv + c0;
#pragma unroll 4
        for (int j = 0; j < K; ++j, vj += rs) {
          Fx2 v[4];
          load4(vj, v);
          const Fx2 t = tr[j];
#pragma unroll
          for (int w = 0; w < 4; ++w) fx_mac(acc[w], t, v[w]);
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const int c = c0 + w;
          const int64_t x = own && c < NR ? fx_val(acc[w]) : 0;
          const int s = team_max<G>(fx_bits(x)) - 57;
          if (own && c < NR) W[c * Cs + tl] = fx_split(fx_scale2(x, -s));
          if (c == tl) fc += s;
          if (c == tl + G) fc2 += s;
        }
      }
      __syncwarp();
      for (int c = tl; active && c < NR; c += G) {
        // true value = W 2^-58 sc
        double sc = pow2(c < G ? fc : fc2);
        if (c > d)
          sc *= rsig;
        else if (c == d)
          sc *= PI.tau * pu;
        else
          sc *= (PI.closed == 1 ? 3.0 : 5.0 / 3.0) * pu;
        sc *= pow2(-29);
        scg[c] = sc;
        const double wk = c < np ? (double)fx_join(W[c * Cs + K - 1]) * sc * pow2(-29) : zk[c - np];
        if (c < np) wkd[c] = wk;
        // ---- record: z_K, w_K and what involves W_0 = e_K (parameter 0 is
        //      Sigma itself); columns c < np are parameters c + 1
        double* wK = rec + 3 + 2 * q;
        double* wzy = wK + P;
        double* wzZ = wzy + P;
        double* F = wzZ + P * q;
        if (c < np) {
          wK[c + 1] = wk;
          F[tri_off(c + 1, 0)] = 0.5 * wk;
        } else {
          if (c == np)
            wzy[0] = wk;
          else
            wzZ[c - np - 1] = wk;
        }
        if (c == 0) {
          wK[0] = 1.0;
          F[0] = 0.5;
        }
      }
      __syncwarp();
      if (active) {
        // ---- record: W z, F = W W^T - w_K w_K^T / 2 (likelihood.py:140-142)
        //      by 2 x 2 tiles: columns (c2, c2 + 1) of the parameters, rows
        //      (c1, c1 + 1) from c1 = c2 on
        double* wzy = rec + 3 + 2 * q + P;
        double* wzZ = wzy + P;
        double* F = wzZ + P * q;
        auto tiles_of = [&](int t) { return (NR - 2 * t + 1) / 2; };
        int ntile = 0;
        for (int t = 0; 2 * t < np; ++t) ntile += tiles_of(t);
        auto put = [&](int c1, int c2, const FxAcc& a) {
          if (c1 >= NR || c2 >= np || c1 < c2) return;
          const double v = (double)fx_val(a) * (scg[c1] * scg[c2]);
          if (c1 < np)
            F[tri_off(c1 + 1, c2 + 1)] = fma(-0.5 * wkd[c1], wkd[c2], v);
          else if (c1 == np)
            wzy[c2 + 1] = v;
          else
            wzZ[(c2 + 1) * q + (c1 - np - 1)] = v;
        };
        for (int t = tl; t < ntile; t += G) {
          int pu2 = 0, rem = t;
          while (rem >= tiles_of(pu2)) {
            rem -= tiles_of(pu2);
            ++pu2;
          }
          const int c2 = 2 * pu2, c1 = c2 + 2 * rem;
          const Fx2* xa = W + c1 * Cs;
          const Fx2* xb = W + min(c1 + 1, NR - 1) * Cs;
          const Fx2* ya = W + c2 * Cs;
          const Fx2* yb = W + min(c2 + 1, NR - 1) * Cs;
          FxAcc g00 = {0, 0}, g01 = {0, 0}, g10 = {0, 0}, g11 = {0, 0};
#pragma unroll 2
          for (int i = 0; i < K; ++i) {
            const Fx2 a0 = xa[i], a1 = xb[i], b0 = ya[i], b1 = yb[i];
            fx_mac(g00, a0, b0);
            fx_mac(g01, a0, b1);
            fx_mac(g10, a1, b0);
            fx_mac(g11, a1, b1);
          }
          put(c1, c2, g00);
          put(c1, c2 + 1, g01);
          put(c1 + 1, c2, g10);
          put(c1 + 1, c2 + 1, g11);
        }
      }
    }
    const unsigned badm = __ballot_sync(kFull, bad) & (G == 32 ? kFull : 0xffffu << (16 * tm));
    leave(badm != 0);
  }
}

namespace {

template <int G>
int launch_fix_g(const LikArgs& A, int kmin, int maxsm, cudaStream_t st) {
  // columns of the largest problem taken
  const int dm = A.dmax < kFixMaxD ? A.dmax : kFixMaxD;
  int ncap = dm + 2 + A.qmax;
  if (ncap > kFixCols) ncap = kFixCols;
  const int pad = (dm + 3) & ~3, col4 = (ncap + 3) & ~3;
  const int rs = (pad > col4 ? pad : col4) + 2;
  const int kcap = A.kcap < G ? A.kcap : G;
  const size_t per_warp = (32 / G) * sizeof(double) * (size_t)fix_slot_words(G, kcap, ncap, rs),
               fixed = 256 * sizeof(double);
  int wpc = kFixThreads / 32;
  while (wpc > 1 && fixed + wpc * per_warp > (size_t)maxsm) --wpc;
  // no more warps per CTA than the fewest rounds over the SMs need: a block is
  // a long chain, and 500 of them on 42 SMs take 107 us, on all SMs less
  const int64_t share = (A.b1 - A.b0 + (int64_t)(32 / G) * sv_num_sms() - 1) / ((int64_t)(32 / G) * sv_num_sms());
  const int64_t rounds = (share + wpc - 1) / wpc;
  if (rounds > 0) wpc = (int)((share + rounds - 1) / rounds);
  const size_t smem = fixed + wpc * per_warp;
  if (smem > (size_t)maxsm) return SV_EINVAL;
  SV_CUDA_TRY(cudaFuncSetAttribute(k_block_fix<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_block_fix<G>, 32 * wpc, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  const int64_t per_cta = (int64_t)wpc * (32 / G);
  int64_t grid = (A.b1 - A.b0 + per_cta - 1) / per_cta;
  if (grid > (int64_t)per_sm * sv_num_sms()) grid = (int64_t)per_sm * sv_num_sms();
  if (grid < 1) grid = 1;
  k_block_fix<G><<<(unsigned)grid, 32 * wpc, smem, st>>>(A, wpc, ncap, rs, kmin);
  SV_CUDA_TRY(cudaGetLastError());
  return SV_OK;
}

}  // namespace

int launch_block_fix(const LikArgs& A, int maxsm, cudaStream_t st) {
  if (A.kcap <= 16) return launch_fix_g<16>(A, 0, maxsm, st);
  // a batch may hold many blocks of at most 16 points: they go two to a warp.
  // One problem has at most 16 of them, not worth a launch
  int kmin = 0;
  if (A.nprob > 1) {
    const int rc = launch_fix_g<16>(A, 0, maxsm, st);
    if (rc != SV_OK) return rc;
    kmin = 16;
  }
  return launch_fix_g<32>(A, kmin, maxsm, st);
}

}  // namespace sv
