// Prediction blocks in fixed point: the same results as k_pred_cta
// (sv_predict.cu) from the Q58 arithmetic of sv_fix.cuh.
//
// k_pred_cta is bound by the float64 pipe (64 cycles per warp instruction and
// scheduler): K^3/6 multiply-adds of the LDL^T and, in the float64 form, a
// distance, a square root and an exponential per entry. Here the block's
// covariance is scaled to a diagonal in (1/2, 1] (its Cholesky factor is then
// bounded by 1) and factored in integers, three 4-cycle multiply-adds for one
// of float64's; the entries come from fx_matern_norm (float64 form, nu = 3/2 and
// 5/2) or, as before, from the float32 deficits (split form).
//
// One CTA per block, 16 rows per warp, two lanes per row: lanes t and t + 16
// of a warp take every other term of their row's sums. Left-looking by panels
// of 8 columns, stored column by column from the panel's first row on, so that
// a warp reads consecutive rows of a column and all lanes the same 8 rows of
// the panel (four 16-byte loads for 24 multiply-adds a lane). The chain of
// pivots bounds a block, so a warp of its own factors the panels' diagonal
// blocks (and inverts them, which makes the back substitution a product per
// panel) while the rows' warps take the next panel's sums over the columns
// before. Two CTAs of a 141-point block (106 KB) fill an SM.
//
// Weights beyond 2^11, pivots below 2^-34 of the diagonal (split form: below
// rho_min), coordinates beyond 32 ranges of the target and non-finite data: the
// split form's block is redone as the float64 form's, that one by pred_block
// in the same CTA.
#include "sv_fixblock.cuh"
#include "sv_predict.cuh"

namespace sv {

constexpr int kPfW = 8;     // columns per panel
// weights |a_j| < 2^(shift - 1) / C_KK, shift = 3 first; where one does not fit,
// two bits more than it needs, up to 12: the column's unit stays below float64's
// for its largest weight
constexpr int kPfShift = 3, kPfShiftMax = 12;

// column j's rows start at row 8 (j / 8); two words of padding keep the
// columns' 16-byte loads apart
__device__ __forceinline__ int pf_col(int j, int K8) {
  const int p = j >> 3;
  return 8 * p * (K8 + 2) - 32 * p * (p - 1) + (j & 7) * (K8 - 8 * p + 2) - 8 * p;
}
__host__ __device__ inline int64_t pf_matrix_words(int K8) {
  const int64_t p = K8 / 8;
  return 8 * p * (K8 + 2) - 32 * p * (p - 1) + 16;
}
// words per point of the coordinates (at least 8: the panels' inverse blocks
// take their place)
__host__ __device__ inline int pf_rs(int d) { return d <= 4 ? 10 : ((d + 3) & ~3) + 2; }
__host__ __device__ inline int64_t pf_words(int kt, int d) {
  const int64_t K8 = (kt + 7) & ~7;
  // matrix, coordinates, pivot thresholds, reciprocal roots and exponents, weights, exponents
  const int64_t fix = pf_matrix_words((int)K8) + K8 * pf_rs(d) + K8 + K8 + K8 / 2 + K8 + K8 / 2 + 4;
  const int64_t old = pred_team_doubles(kt, d);
  return (fix > old ? fix : old) + 2;
}

__device__ __forceinline__ int64_t pf_from_float(float x) {  // x >= 0, in Q58
  const unsigned b = __float_as_uint(x);
  const int e = (int)(b >> 23) - 127;
  if (e < -90) return 0;
  const int64_t m = (b & 0x7fffffu) | 0x800000u;
  return fx_scale2(m, e + 35);
}

__device__ __noinline__ void pf_fallback(const PredArgs& A0, const PredPrm* prm, int64_t b, double* sm) {
  PredArgs A = A0;
  A.split = 0;
  if (blockDim.x <= 128)
    pred_block<128>(A, prm, b, sm);
  else if (blockDim.x <= 192)
    pred_block<192>(A, prm, b, sm);
  else if (blockDim.x <= 256)
    pred_block<256>(A, prm, b, sm);
  else if (blockDim.x <= 320)
    pred_block<320>(A, prm, b, sm);
  else
    pred_block<448>(A, prm, b, sm);
}

// One panel's diagonal block (8 lanes, the others in step with them): C_ij in
// place of its entries, and the inverse T of the block as fix_factor takes it
// (lane r its row of C, then its column of T), T_jr 2^-E_r at Tp[8 j + r].
__device__ __forceinline__ void pf_diag(int K, int k0, int r, bool writer, Fx2* pc, int Lp, const int64_t* thr,
                                        Fx2* ivy, int* ive, Fx2* Tp, int* Te, int64_t* last, int* bad) {
  FxAcc acc[kPfW];
#pragma unroll
  for (int w = 0; w < kPfW; ++w) acc[w] = {0, 0};
  int E = 0;
  int64_t sq = 0;
#pragma unroll
  for (int w = 0; w < kPfW; ++w) {
    const int c = k0 + w;
    int64_t v = (r >= w ? *(const int64_t*)(pc + w * Lp + k0 + r) : 0) - fx_val(acc[w]);
    if (r == w) v -= fx_sq_val(sq);
    const int64_t dv = __shfl_sync(kFull, (long long)v, w, 8);
    if (c < K && writer && r == w && (dv < thr[c] || dv > (1ll << 58))) *bad = 1;
    const int64_t dc = (dv < (1ll << (58 - kFixPivotShift)) || dv > (1ll << 58)) ? 1ll << 58 : dv;
    int e;
    const int64_t Yq = fx_rsqrt_pivot(dc, e);
    const Fx2 Y = fx_split(Yq);
    if (r < w) {
      int tries = 0;
      int hi = (int)(v >> 32);
      while (((hi ^ (hi >> 31)) >> (26 - e)) != 0) {  // |v| 2^e >= 2^58
        if (++tries > 12) {
          *bad = 1;
          v = 0;
          break;
        }
        E += kFixStep;
        if (writer)
          for (int j = r; j < w; ++j) Tp[8 * j + r] = fx_split(fx_join(Tp[8 * j + r]) >> kFixStep);
#pragma unroll
        for (int w2 = 0; w2 < kPfW; ++w2) {
          acc[w2].h >>= kFixStep;
          acc[w2].m >>= kFixStep;
        }
        v >>= kFixStep;
        hi = (int)(v >> 32);
      }
    }
    int64_t x = fx_mul(fx_split((int64_t)((uint64_t)v << e)), Y);
    if (r == w) {
      if (writer) {
        ivy[c] = Y;
        ive[c] = e;
        if (c == K - 1) *last = dv;
      }
      E = e + kFixHead;
      x = Yq >> kFixHead;
#pragma unroll
      for (int w2 = w + 1; w2 < kPfW; ++w2) acc[w2] = {0, 0};
    }
    const Fx2 cs = fx_split(x);
    if (r > w) fx_sq(sq, cs);
    if (writer) {
      if (r > w)
        pc[w * Lp + k0 + r] = cs;
      else
        Tp[8 * w + r] = cs;
    }
#pragma unroll
    for (int w2 = w + 1; w2 < kPfW; ++w2) {
      Fx2 o;
      o.h = __shfl_sync(kFull, cs.h, w2, 8);
      o.l = __shfl_sync(kFull, cs.l, w2, 8);
      fx_mac(acc[w2], cs, o);
    }
  }
  if (writer) Te[k0 + r] = E;
}

// after a failed attempt: the float64 form's, when that was the split form's
// (counted) and the float64 form has one here
__device__ __forceinline__ bool pf_next(const PredArgs& A, bool& split, int& s_bad, int& s_max) {
  __syncthreads();
  const bool again = split && (A.closed == 1 || A.closed == 2);
  if (threadIdx.x == 0) {
    if (split) atomicAdd(A.info + SV_INFO_AUX, 1);
    s_bad = 0;
    s_max = 0;
  }
  split = false;
  __syncthreads();
  return again;
}

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_pred_fix(PredArgs A) {
  extern __shared__ double smem[];
  PredPrm* prm = (PredPrm*)smem;
  pred_params(A, prm);
  uint64_t* T = (uint64_t*)(smem + (sizeof(PredPrm) + 15) / 16 * 2);
  for (int i = threadIdx.x; i < 256; i += blockDim.x) T[i] = kFxExp2[i];
  double* region = (double*)(T + 256);
  __shared__ int s_k, s_max, s_bad;
  __shared__ double s_red[NT / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, half = lane >> 4;
  const bool boss = warp == (int)(blockDim.x >> 5) - 1;  // the warp of the panels' diagonal blocks
  const int i = 16 * warp + (lane & 15);                 // this thread's row
  const int d = A.d, rs = pf_rs(d);
  const double s2 = prm->s2, tau = prm->tau;
  // Sigma = s2 2^ek times a matrix of diagonal (1 + tau mask) 2^-ek <= 1
  int ek = 0;
  while (ek < 20 && (double)(1 << ek) < 1.0 + tau) ++ek;
  const bool prm_ok = tau >= 0.0 && tau <= 1e6 && s2 > 1e-200 && s2 < 1e200;
  const int64_t one = 1ll << (58 - ek);
  const int64_t tauq = prm_ok ? llrint(ldexp(tau, 58 - ek)) : 0;
  __syncthreads();

  for (int64_t b = blockIdx.x; b < A.nblk; b += gridDim.x) {
    // neighbours are packed at the front of the row; -1 marks absent entries
    if (threadIdx.x == 0) {
      s_k = A.k;
      s_max = 0;
      s_bad = prm_ok ? 0 : 1;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < A.k; t += blockDim.x)
      if (A.nbr[b * A.ldnbr + t] < 0) atomicMin(&s_k, t);
    __syncthreads();
    const int k = s_k, K = k + 1, K8 = (K + 7) & ~7;
    Fx2* M = (Fx2*)region;
    Fx2* cv = M + pf_matrix_words(K8);
    int64_t* thr = (int64_t*)(cv + K8 * rs);  // pivot thresholds
    Fx2* ivy = (Fx2*)(thr + K8);
    int* ive = (int*)(ivy + K8);
    Fx2* us = (Fx2*)(ive + K8);
    int* Te = (int*)(us + K8);
    int64_t* last = (int64_t*)(Te + K8);   // pivot of the last row
    Fx2* Tp = cv;                          // panels' inverse blocks, once the entries are there
    const bool own = !boss && i < K;
    const int row = own ? (i < k ? A.nbr[b * A.ldnbr + i] : A.tgt[b]) : 0;
    // gp.py:263-265, 336-339: nugget on observations only (a prior draw keeps
    // it on every row, target included)
    const bool nug = (i < k && row < A.nobs) || (i == k && A.target_nugget);
    const int64_t diag = one + (nug ? tauq : 0);

    // the split form's attempt, then (or first) the float64 form's
    for (bool split = A.split && prm_ok;;) {
    // ---- coordinates centred on the target, a lane every other input
    {
      const double* xt = A.Xall + (int64_t)A.tgt[b] * d;
      const double* xi = A.Xall + (int64_t)row * d;
      double v[kFixMaxD / 2];
      int exm = 0;
#pragma unroll
      for (int t = 0; t < kFixMaxD / 2; ++t) {
        const int l = 2 * t + half;
        v[t] = (own && l < d) ? (xi[l] - xt[l]) * prm->invlam[l] : 0.0;
        exm = max(exm, (int)((dbits(v[t]) >> 52) & 0x7ff));
      }
      if (split) {
        if (exm >= 0x43B) s_bad = 1;  // 2^60
#pragma unroll
        for (int t = 0; t < kFixMaxD / 2; ++t) {
          const int l = 2 * t + half;
          if (own && l < d) {
            const float hi = d2f_int(v[t]);
            ((float2*)cv)[i * rs + l] = make_float2(hi, d2f_int(v[t] - f2d_int(hi)));
          }
        }
      } else {
        exm = team_max<32>(exm);
        if (lane == 0) atomicMax(&s_max, exm);
        __syncthreads();
        exm = s_max;
        if (exm > 1023 + 4) {
          if (threadIdx.x == 0) s_bad = 1;
          exm = 2046;
        }
#pragma unroll
        for (int t = 0; t < kFixMaxD / 2; ++t) {
          const int l = 2 * t + half;
          if (l < ((d + 3) & ~3) && own) cv[i * rs + l] = fx_split(fx_from_bits<6>(dbits(v[t]), exm));
        }
      }
    }
    if (own && half == 0) *(int64_t*)(M + pf_col(i, K8) + i) = diag;
    if (!boss && half == 0 && i >= K && i < K8)  // rows of padding
      for (int j = 0; j <= i; ++j) *(int64_t*)(M + pf_col(j, K8) + i) = 0;
    __syncthreads();

    // ---- entries: in round r row i takes the pair (i, i + r mod K), the two
    //      lanes of a row every other round
    if (own && !s_bad) {
      if (split) {
        const MaternF32 mf = prm->mf;
        const float2* ci = (const float2*)cv + i * rs;
        for (int r = 1 + half; 2 * r <= K; r += 2) {
          if (2 * r == K && i >= r) break;
          int j = i + r;
          if (j >= K) j -= K;
          const float2* cj = (const float2*)cv + j * rs;
          float r2 = 0.0f;
          for (int l = 0; l < d; ++l) {
            const float2 a = ci[l], c = cj[l];
            const float df = (a.x - c.x) + (a.y - c.y);
            r2 = fmaf(df, df, r2);
          }
          const int64_t x = (1ll << 58) - pf_from_float(matern_deficit_f32(mf, sqrtf(r2)));
          const int lo = min(i, j), hi = max(i, j);
          *(int64_t*)(M + pf_col(lo, K8) + hi) = fx_scale2(x, -ek);
        }
      } else {
        const int es = s_max - 1023 + 3;
        Fx2 ui[kFixMaxD];
#pragma unroll
        for (int g = 0; g < kFixMaxD; g += 4)
          if (g < d) {
#pragma unroll
            for (int l = g; l < g + 4; ++l) ui[l] = cv[i * rs + l];
          }
        for (int r = 1 + half; 2 * r <= K; r += 2) {
          if (2 * r == K && i >= r) break;
          int j = i + r;
          if (j >= K) j -= K;
          const Fx2* uj = cv + j * rs;
          FxSq q = {0, 0, 0};
#pragma unroll
          for (int g4 = 0; g4 < kFixMaxD; g4 += 4)
            if (g4 < d) {
              Fx2 w[4];
              load4(uj + g4, w);
              if (g4 == 8) fx_sqcarry(q);
#pragma unroll
              for (int l = 0; l < 4; ++l) fx_sqdiff(q, ui[g4 + l], w[l]);
            }
          int E;
          uint64_t m, g;
          const uint64_t s = fx_sqnorm(q, es, E);
          if (A.closed == 1)
            fx_matern_norm<1, false>(s, E, T, m, g);
          else
            fx_matern_norm<2, false>(s, E, T, m, g);
          const int lo = min(i, j), hi = max(i, j);
          *(int64_t*)(M + pf_col(lo, K8) + hi) = (int64_t)((m + (4ull << ek)) >> (3 + ek));
        }
      }
    }
    __syncthreads();
    if (own && half == 0) thr[i] = split ? (int64_t)(A.rho_min * (double)diag) : 1ll << (58 - kFixPivotShift);
    __syncthreads();

    // ---- Cholesky factor, panels of 8 columns.  At the start of a panel its
    //      columns hold S less the earlier columns' products
    int64_t sq = 0;
    for (int k0 = 0; k0 < K8; k0 += kPfW) {
      Fx2* pc = M + pf_col(k0, K8);
      const int Lp = K8 - k0 + 2, k1 = k0 + kPfW;
      const bool busy = !boss && k1 < K8 && 16 * warp + 15 >= k1 && 16 * warp < K8;
      FxAcc acc[kPfW];
#pragma unroll
      for (int w = 0; w < kPfW; ++w) acc[w] = {0, 0};
      if (boss) {
        pf_diag(K, k0, lane & 7, lane < 8, pc, Lp, thr, ivy, ive, Tp + 8 * k0, Te, last, &s_bad);
      } else if (busy) {
        // the next panel's sums over the columns before this one
        for (int j0 = 0; j0 < k0; j0 += 8) {
          const int L = K8 - j0 + 2;
          const Fx2* col = M + pf_col(j0, K8) + half * L;
#pragma unroll 2
          for (int t = 0; t < 4; ++t, col += 2 * L) {
            const Fx2 x = col[i];
            Fx2 v[4];
            load4(col + k1, v);
#pragma unroll
            for (int w = 0; w < 4; ++w) fx_mac(acc[w], x, v[w]);
            load4(col + k1 + 4, v);
#pragma unroll
            for (int w = 0; w < 4; ++w) fx_mac(acc[4 + w], x, v[w]);
          }
        }
      }
      __syncthreads();
      if (s_bad) break;
      Fx2 c[kPfW];
      const bool below = busy && i >= k1 && i < K8;
      if (busy) {
#pragma unroll
        for (int w = 0; w < kPfW; ++w) {
          FxAcc t = {0, 0};
#pragma unroll
          for (int u = 0; u < w; ++u) fx_mac(t, c[u], pc[u * Lp + k0 + w]);
          const int64_t v = below ? *(const int64_t*)(pc + w * Lp + i) - fx_val(t) : 0;
          c[w] = fx_split(fx_mul(fx_split((int64_t)((uint64_t)v << ive[k0 + w])), ivy[k0 + w]));
          fx_sq(sq, c[w]);
          if (below && half == 0) pc[w * Lp + i] = c[w];
        }
      }
      __syncthreads();
      if (busy) {
        // this panel's share of the next one's sums, four columns a lane
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const Fx2 x = half ? c[4 + t] : c[t];
          const Fx2* col = pc + (4 * half + t) * Lp;
          Fx2 v[4];
          load4(col + k1, v);
#pragma unroll
          for (int w = 0; w < 4; ++w) fx_mac(acc[w], x, v[w]);
          load4(col + k1 + 4, v);
#pragma unroll
          for (int w = 0; w < 4; ++w) fx_mac(acc[4 + w], x, v[w]);
        }
        Fx2* pn = M + pf_col(k1, K8) + i;
        const int Ln = Lp - kPfW;
#pragma unroll
        for (int w = 0; w < kPfW; ++w) {
          acc[w].h += __shfl_xor_sync(kFull, (long long)acc[w].h, 16);
          acc[w].m += __shfl_xor_sync(kFull, (long long)acc[w].m, 16);
          if (half == (w & 1) && i >= k1 + w && i < K8)
            *(int64_t*)(pn + w * Ln) -= fx_val(acc[w]) + (i == k1 + w ? fx_sq_val(sq) : 0);
        }
      }
      __syncthreads();
    }
    if (s_bad) {
      if (pf_next(A, split, s_bad, s_max)) continue;
      pf_fallback(A, prm, b, region);
      break;
    }

    // ---- a = C^-T e_K, panels from the last to the first: the panel's 8 rows
    //      by the inverse of its diagonal block, then every earlier row its
    //      terms (the two lanes of a row four each).  a = us 2^sa.  The sums
    //      keep 2^-86 of the scale, since the inverse's entries magnify what
    //      they lose: with one rounding to 2^-58 (and the products of low limbs
    //      left out) a row's error was 8 2^-57 / C_jj, more than float64's
    int shift = kPfShift;
    Fx2 ui = {0, 0};
    for (;;) {
      const int sa = ive[K - 1] + shift;
      FxAcc acc = {0, 0};
      for (int k0 = K8 - kPfW; k0 >= 0; k0 -= kPfW) {
        if (!boss && warp == (k0 >> 4)) {
          const bool mine = i >= k0 && i < k0 + kPfW;
          FxAcc tot = acc;
          tot.h += __shfl_xor_sync(kFull, (long long)acc.h, 16);
          tot.m += __shfl_xor_sync(kFull, (long long)acc.m, 16);
          const bool first = s_bad == 0;  // (behind a column that does not fit come meaningless ones)
          // r 2^28 + lo in Q86
          int64_t r = 0, lo = 0;
          if (mine && own) {
            lo = -tot.m & ((1ll << 28) - 1);
            r = (-tot.m >> 28) - (int64_t)((uint64_t)tot.h << 2);
            if (i == K - 1) r += 1ll << (58 - sa);
          }
          const int g = 57 - team_max<32>(fx_bits(r));  // the panel's largest below 2^57
          const Fx2 rs2 = fx_split(fx_scale2(r, g) + (g >= 28 ? lo << (g - 28) : g > 0 ? lo >> (28 - g) : 0));
          const Fx2* t = Tp + 8 * k0 + (i & 7);
          FxAcc u = {0, 0};
#pragma unroll
          for (int w = 0; w < kPfW; ++w) {
            Fx2 o;
            o.h = __shfl_sync(kFull, rs2.h, (k0 & 15) + w);
            o.l = __shfl_sync(kFull, rs2.l, (k0 & 15) + w);
            if (w >= (i & 7)) fx_mac(u, t[8 * w], o);
          }
          if (mine) {
            const int64_t x = fx_val(u);
            int sh = Te[i] - g;
            if (own && fx_bits(x) + sh > 57 && x != 0) {
              if (first) atomicMax(&s_bad, fx_bits(x) + sh - 57);
              sh = 0;
            }
            ui = fx_split(own ? fx_scale2(x, sh) : 0);
            if (half == 0) us[i] = ui;
          }
        }
        __syncthreads();
        if (!boss && i < k0) {
          Fx2 c4[4], u4[4];
          load4(M + pf_col(i, K8) + k0 + 4 * half, c4);
          load4(us + k0 + 4 * half, u4);
          int64_t low = 1ll << 29;
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            fx_mac(acc, c4[w], u4[w]);
            low += (int64_t)c4[w].l * u4[w].l;
          }
          acc.m += low >> 30;
        }
      }
      __syncthreads();
      if (!s_bad || shift >= kPfShiftMax) break;
      shift = min(shift + s_bad + 2, kPfShiftMax);
      __syncthreads();
      if (threadIdx.x == 0) s_bad = 0;
      __syncthreads();
    }
    if (s_bad) {
      if (pf_next(A, split, s_bad, s_max)) continue;
      pf_fallback(A, prm, b, region);
      break;
    }

    // ---- Sigma = sig^2 C C^T: mean = -(a.r) / a_K, a_K = 1 / C_KK = Y 2^e,
    //      var = sig^2 d_K, the column of U a / sig
    const double uq = (double)fx_join(ui) * 0x1p-58;
    double sm = 0.0;
    if (!boss && half == 0 && i < k && row < A.nobs && A.resid) sm = uq * A.resid[row];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sm += __shfl_xor_sync(kFull, sm, o);
    if (lane == 0) s_red[warp] = sm;
    __syncthreads();
    sm = 0.0;
    for (int w = 0; 16 * w < K; ++w) sm += s_red[w];
    const double sc = ldexp(s2, ek), p2 = (double)(1 << (ive[K - 1] + shift));
    if (threadIdx.x == 0) {
      if (A.mean) A.mean[b] = -sm * (double)(1 << shift) / ((double)fx_join(ivy[K - 1]) * 0x1p-58);
      if (A.var) A.var[b] = sc * ((double)*last * 0x1p-58);
    }
    if (A.rhs || A.acol) {
      const double rs1 = p2 / sqrt(sc);
      if (A.rhs && threadIdx.x == 0) A.rhs[b] = -sm * rs1;
      if (A.acol) {
        // [neighbour slots 0..k-1, target]; absent neighbour slots hold 0
        double* ac = A.acol + b * (int64_t)(A.k + 1);
        if (!boss && half == 0 && i < K) ac[i < k ? i : A.k] = uq * rs1;
        for (int t = k + threadIdx.x; t < A.k; t += blockDim.x) ac[t] = 0.0;
      }
    }
    break;
    }
    __syncthreads();
  }
}

namespace {
size_t pf_smem(const PredArgs& A) {
  return (sizeof(PredPrm) + 15) / 16 * 16 + 256 * 8 + 8 * (size_t)pf_words(A.kt, A.d);
}
}  // namespace

bool pred_fix_takes(const PredArgs& A, int maxsm) {
  // blocks of at most 32 points: a warp each (sv_predict.cu)
  if (A.d > kFixMaxD || A.kt <= 32 || A.kt > 208 || pf_smem(A) > (size_t)maxsm) return false;
  // the split form's pivot guard has to be the tighter one
  return A.split ? A.rho_min >= 1e-9 : (A.closed == 1 || A.closed == 2);
}

int launch_pred_fix(const PredArgs& A, int maxsm, cudaStream_t st) {
  const size_t smem = pf_smem(A);
  const int nt = 32 * ((A.kt + 15) / 16 + 1);  // the rows' warps and the diagonal blocks'
  auto run = [&](auto kern, int threads) -> int {
    SV_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    int64_t grid = A.nblk;
    if (grid > (int64_t)per_sm * sv_num_sms()) grid = (int64_t)per_sm * sv_num_sms();
    kern<<<(unsigned)grid, threads, smem, st>>>(A);
    SV_CUDA_TRY(cudaGetLastError());
    return SV_OK;
  };
  if (nt <= 128) return run(k_pred_fix<128, 5>, 128);
  if (nt <= 192) return run(k_pred_fix<192, 3>, 192);
  if (nt <= 256) return run(k_pred_fix<256, 2>, 256);
  if (nt <= 320) return run(k_pred_fix<320, 2>, 320);
  return run(k_pred_fix<448, 1>, 448);
}

}  // namespace sv
