// Shared definitions of the prediction block kernels (sv_predict.cu: float64
// factorisation; sv_predict_fix.cu: fixed point).
#pragma once
#include "sv_block.cuh"

namespace sv {

struct PredArgs {
  const double* theta;  // [log s2, log lam_1..d, log tau]
  const double* Xall;
  const int32_t* tgt;
  const int32_t* nbr;
  const double* resid;
  double* mean;
  double* var;
  double* acol;
  double* rhs;
  int32_t* info;
  int64_t nobs, nblk;
  int d, k, ldnbr, kt;
  int closed;
  int target_nugget;
  int split;       // 1: float32 assembly (closed-form nu only)
  double rho_min;  // split: smallest pivot ratio d_k / Sigma_kk kept
  double nu;
  const double* tab;    // general nu: its Matern table (or null: K_nu per entry)
  const float4* ftab;   // general nu, split: the table's float32 part (or null)
};

struct PredPrm {
  double s2, tau;
  MaternMode mm;
  MaternF32 mf;  // the split form's float32 Matern: a closed form or the table
  double invlam[64];
};

__device__ inline void pred_params(const PredArgs& A, PredPrm* prm) {
  if (threadIdx.x == 0) {
    prm->s2 = exp(A.theta[0]);
    prm->tau = exp(A.theta[1 + A.d]);
    MaternMode mm;
    mm.closed = A.closed;
    mm.estimate_nu = 0;
    mm.nu = A.nu;
    mm.log_coef = A.closed < 0 ? matern_log_coef(A.nu) : 0.0;
    mm.nu_p = mm.nu_m = mm.lc_p = mm.lc_m = 0.0;
    mm.inv2h = 0.0;
    mm.tab = A.closed < 0 ? A.tab : nullptr;
    mm.tab_fixed = 0;
    mm.tab_elo = mm.tab ? mtab_elo(A.nu) : 0;
    mm.s2n = sqrt(2.0 * A.nu);
    mm.tab_p = mm.tab_m = nullptr;
    mm.elo_p = mm.elo_m = 0;
    mm.s2n_p = mm.s2n_m = 0.0;
    prm->mm = mm;
    MaternF32 mf;
    mf.code = A.closed >= 0 ? A.closed : (A.ftab ? 3 : -1);
    mf.elo = A.ftab ? mtab_elo(A.nu) : 0;
    mf.esw = ftab_switch(A.nu);
    mf.s2n = (float)sqrt(2.0 * A.nu);
    mf.tab = A.closed >= 0 ? nullptr : A.ftab;
    mf.dtab = nullptr;
    mf.nuf = (float)A.nu;
    prm->mf = mf;
  }
  for (int l = threadIdx.x; l < A.d; l += blockDim.x) prm->invlam[l] = exp(-A.theta[1 + l]);
  __syncthreads();
}

// columns per panel of the blocked LDL^T
constexpr int kPredW = 8;

__host__ __device__ inline int64_t pred_team_doubles(int kt, int d) {
  return (int64_t)kt * d + (int64_t)kt * (kt + 1) / 2 + (4 + kPredW) * (int64_t)kt + (kt + 1) / 2 +
         1 + 40;
}

// |x| below 2^60: d <= 64 squared float32 differences of such coordinates
// stay finite
constexpr long long kBitsCoordMax = 0x43B0000000000000LL;

// The split form's attempt at a block: coordinates centred on the target
// (scaled differences formed in float64, kept as float32 (hi, lo) pairs), the entries
// below the diagonal s2 (1 - D(r_ij)) with D the float32 correlation deficit
// (accurate for close pairs), the diagonal s2 (1 + tau mask_i) in float64,
// then the LDL^T with the pivot-ratio guard (thresholds rho_min Sigma_kk in
// rb).  Returns false when the block must be redone in float64: a coordinate
// out of range, a pivot that is not > 0 or below its threshold.
template <int T>
__device__ bool pred_split_factor(const PredArgs& A, const PredPrm* prm, int K, double* u,
                                  double* Lp, double* invd, double* acc, const double* mask,
                                  long long* rb, const int* idx, volatile int* flag) {
  const int lane = Team<T>::lane();
  const int d = A.d;
  float2* u2 = (float2*)u;
  const double* xt = A.Xall + (int64_t)idx[K - 1] * d;
  if (lane == 0) flag[1] = 0;
  Team<T>::sync();
  bool in_range = true;
  for (int t = lane; t < K * d; t += T) {
    const int i = t / d, l = t - (t / d) * d;
    const double v = (A.Xall[(int64_t)idx[i] * d + l] - xt[l]) * prm->invlam[l];
    in_range = in_range && (dbits(v) & 0x7FFFFFFFFFFFFFFFLL) < kBitsCoordMax;
    const float hi = d2f_int(v);
    u2[t] = make_float2(hi, d2f_int(v - f2d_int(hi)));
  }
  if (!in_range) flag[1] = 1;
  const double s2 = prm->s2, tau = prm->tau;
  for (int i = lane; i < K; i += T) rb[i] = dbits(A.rho_min * (s2 * (1.0 + tau * mask[i])));
  Team<T>::sync();
  if (flag[1]) return false;
  const MaternF32 mf = prm->mf;
  const int npair = K * (K + 1) / 2;
  for (int t = lane; t < npair; t += T) {
    int i, j;
    tri_index(t, i, j);
    double v;
    if (i == j) {
      v = s2 * (1.0 + tau * mask[i]);
    } else {
      const float2* ui = u2 + i * d;
      const float2* uj = u2 + j * d;
      float r2 = 0.0f;
      for (int l = 0; l < d; ++l) {
        // (hi_i - hi_j) + (lo_i - lo_j): the difference to about one float32
        // rounding of itself, however far the pair lies from the target
        const float2 a = ui[l], c = uj[l];
        const float df = (a.x - c.x) + (a.y - c.y);
        r2 = fmaf(df, df, r2);
      }
      v = fma(-s2, f2d_int(matern_deficit_f32(mf, sqrtf(r2))), s2);
    }
    Lp[t] = v;
  }
  if (lane == 0) *flag = 0;
  Team<T>::sync();
  const bool ok = ldlt_blocked<T, kPredW>(K, Lp, invd, acc, A.kt, flag, rb);
  Team<T>::sync();
  return ok;
}

template <int T>
__device__ void pred_block(const PredArgs& A, const PredPrm* prm, int64_t b, double* sm) {
  const int lane = Team<T>::lane();
  const int d = A.d, kcap = A.k, kt = A.kt;
  double* u = sm;
  double* Lp = u + (int64_t)kt * d;
  double* a = Lp + (int64_t)kt * (kt + 1) / 2;
  double* invd = a + kt;
  double* acc = invd + kt;                 // kPredW columns of kt
  double* mask = acc + kPredW * kt;
  double* rv = mask + kt;
  int* idx = (int*)(rv + kt);
  volatile int* flag = idx + kt;
  double* red = (double*)(rv + kt + (kt + 1) / 2 + 1);

  // neighbours are packed at the front of the row; -1 marks absent entries
  // (rows with fewer than k predecessors)
  if (lane == 0) {
    int kb = 0;
    while (kb < kcap && A.nbr[b * A.ldnbr + kb] >= 0) ++kb;
    *flag = kb;
  }
  Team<T>::sync();
  const int k = *flag;
  const int K = k + 1;
  Team<T>::sync();
  for (int i = lane; i < K; i += T) {
    const int ix = (i < k) ? A.nbr[b * A.ldnbr + i] : A.tgt[b];
    idx[i] = ix;
    // gp.py:263-265, 336-339: nugget on observations only, target noise-free
    // (a prior draw keeps the nugget on every row, target included)
    mask[i] = ((i < k && ix < A.nobs) || (i == k && A.target_nugget)) ? 1.0 : 0.0;
    rv[i] = (A.resid && i < k && ix < A.nobs) ? A.resid[ix] : 0.0;
  }
  Team<T>::sync();
  const double s2 = prm->s2, tau = prm->tau;
  bool ok = false;
  if (A.split) ok = pred_split_factor<T>(A, prm, K, u, Lp, invd, acc, mask, (long long*)a, idx, flag);
  if (!ok) {
    if (A.split && lane == 0) atomicAdd(A.info + SV_INFO_AUX, 1);
    for (int t = lane; t < K * d; t += T) {
      const int i = t / d, l = t - (t / d) * d;
      u[i * d + l] = A.Xall[(int64_t)idx[i] * d + l] * prm->invlam[l];
    }
    Team<T>::sync();
  }
  for (int lv = 0; lv <= 9 && !ok; ++lv) {
    double jit = 0.0;
    if (lv > 0) {
      // 10^p * mean(diag Sigma)   (_covariance.py:245-249)
      double sc = 0.0;
      for (int i = 0; i < K; ++i) sc += s2 * (1.0 + tau * mask[i]);
      const double p10[10] = {0.0, 1e-12, 1e-11, 1e-10, 1e-9, 1e-8, 1e-7, 1e-6, 1e-5, 1e-4};
      jit = p10[lv] * (sc / (double)K);
    }
    if (lane == 0) *flag = 0;
    assemble_sigma<T>(K, d, u, mask, s2, tau, jit, prm->mm, Lp, nullptr, nullptr);
    Team<T>::sync();
    ok = ldlt_blocked<T, kPredW>(K, Lp, invd, acc, kt, flag);
    Team<T>::sync();
    if (ok) {
      if (lv > 0 && lane == 0) atomicMax(A.info + SV_INFO_JITTER, lv);
      break;
    }
  }
  if (!ok) {
    if (lane == 0) {
      set_error(A.info + SV_INFO_STATUS, SV_ECHOL);
      atomicCAS(A.info + SV_INFO_BLOCK, -1, (int)b);
    }
    return;
  }
  // Sigma = L D L^T = C C^T with C = L D^(1/2): a = C^-T e_K = u / sqrt(d_K),
  // u = L^-T e_K (u_K = 1), so mean = -a[:k].r / a_K = -u[:k].r and
  // var = 1 / a_K^2 = d_K; only the U column needs the square root
  backsolve_unit_eK<T>(K, Lp, a, acc);
  Team<T>::sync();
  double s = 0.0;
  for (int i = lane; i < k; i += T) s += a[i] * rv[i];
  s = team_sum<T>(s, red);
  const double dK = Lp[tri_off(K - 1, K - 1)];
  const double sK = 1.0 / sqrt(dK);
  if (lane == 0) {
    if (A.mean) A.mean[b] = -s;
    if (A.var) A.var[b] = dK;
    if (A.rhs) A.rhs[b] = -s * sK;
  }
  if (A.acol) {
    // column of U laid out as [neighbour slots 0..kcap-1, target]; absent
    // neighbour slots hold 0
    const int Kc = kcap + 1;
    for (int i = lane; i < Kc; i += T)
      A.acol[b * (int64_t)Kc + i] = (i < k) ? a[i] * sK : (i == kcap ? sK : 0.0);
  }
}


// the fixed-point kernel (sv_predict_fix.cu), for blocks of at most A.kt
// points: whether it takes this call, and its launch
bool pred_fix_takes(const PredArgs& A, int maxsm);
int launch_pred_fix(const PredArgs& A, int maxsm, cudaStream_t st);

}  // namespace sv
