// Prediction blocks and the sparse triangular solve of the joint predictive
// distribution.
//
//   k_pred_*      : gp.py:257-276 (_predict_scaled) and gp.py:329-348
//                   (_joint_factor): per target, the block [neighbours, target]
//                   with a noise-free target (nugget only on observation rows),
//                   Cholesky with jitter retry, a = L^-T e_K; marginal mean
//                   -a[:k].r / a_K and variance 1 / a_K^2, or the column a of
//                   the sparse inverse Cholesky factor U.
//                   Split form (closed-form nu): the entries below the
//                   diagonal from coordinates centred on the target, held as
//                   float32 (hi, lo) pairs, and the float32 correlation
//                   deficit, one float64 FMA each; the diagonal,
//                   the LDL^T and every solve in float64.  A block with a
//                   pivot ratio d_k / Sigma_kk below rho_min, or that does not
//                   factor, is redone in float64 from the start.
//   k_joint_solve : U_pp^T x = rhs (gp.py:380-401, scipy spsolve_triangular),
//                   one CTA per row (its threads split the right-hand sides),
//                   rows claimed in order, bounded waits on the rows it
//                   depends on.
#include "sv_predict.cuh"

namespace sv {

__global__ void k_pred_warp(PredArgs A) {
  extern __shared__ double smem[];
  PredPrm* prm = (PredPrm*)smem;
  pred_params(A, prm);
  const int64_t per = pred_team_doubles(32, A.d);
  const int w = threadIdx.x >> 5;
  double* sm = smem + (sizeof(PredPrm) + 7) / 8 + w * per;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + w; b < A.nblk; b += nw) {
    pred_block<32>(A, prm, b, sm);
    __syncwarp();
  }
}

// threads of the CTA that owns one large prediction block: two CTAs of a
// 141-point block fill an SM's shared memory, so 12 warps each keep 24 warps
// resident to cover the float64 and shared-memory latency (measured at 50,000
// blocks of 141: 256 threads 58.9 ms, 384 57.8 ms, 512 86 ms, where the
// registers allow one CTA per SM)
constexpr int kPredCta = 384;

__global__ void __launch_bounds__(kPredCta) k_pred_cta(PredArgs A) {
  extern __shared__ double smem[];
  PredPrm* prm = (PredPrm*)smem;
  pred_params(A, prm);
  double* sm = smem + (sizeof(PredPrm) + 7) / 8;
  for (int64_t b = blockIdx.x; b < A.nblk; b += gridDim.x) {
    pred_block<kPredCta>(A, prm, b, sm);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// sparse triangular solve  U_pp^T X = R
// ---------------------------------------------------------------------------
struct JsArgs {
  int64_t npred, nobs;
  int k, ldnbr, nrhs;
  const int32_t* nbr;
  const double* acol;
  const double* R;
  double* X;
  int* ready;
  unsigned* counter;
  unsigned* progress;    // rows published so far
  int32_t* info;
  unsigned spin_limit;   // polls without progress anywhere before a wait gives up
  int skip_ready_row0;   // test aid: row 0 never publishes, its dependants' waits run out
};

// One CTA per row at a time, rows claimed in order by an atomic counter (a
// row depends only on rows claimed before it, so every awaited row is held
// by a running CTA).  The row's earlier-prediction neighbours and their
// coefficients go to shared memory, one thread waits per dependency, then
// the threads split the right-hand sides; each right-hand side is the same
// sum in the same order as a one-thread solve.  A wait gives up when neither
// its row nor any other row has been published for spin_limit polls (a
// stall, not a long dependency chain: a row's time grows with nrhs).
__global__ void k_joint_solve(JsArgs A) {
  extern __shared__ double js_sm[];
  double* s_a = js_sm;                              // [k] coefficients
  int* s_p = (int*)(js_sm + (A.k > 0 ? A.k : 1));   // [k] earlier rows
  __shared__ long long s_c;
  __shared__ int s_np;
  const int K = A.k + 1;
  while (true) {
    if (threadIdx.x == 0) s_c = (long long)atomicAdd(A.counter, 1u);
    __syncthreads();
    const int64_t c = s_c;
    if (c >= A.npred) break;
    const double* ac = A.acol + c * (int64_t)K;
    if (threadIdx.x == 0) {
      int np = 0;
      for (int i = 0; i < A.k; ++i) {
        const int64_t ix = A.nbr[c * (int64_t)A.ldnbr + i];
        if (ix < 0 || ix < A.nobs) continue;  // absent slot or observation
        s_p[np] = (int)(ix - A.nobs);         // an earlier prediction row
        s_a[np] = ac[i];
        ++np;
      }
      s_np = np;
    }
    __syncthreads();
    const int np = s_np;
    for (int j = threadIdx.x; j < np; j += blockDim.x) {
      const int p = s_p[j];
      unsigned it = 0, seen = ld_acquire_u32(A.progress);
      while (ld_acquire_s32(A.ready + p) == 0) {
        if (++it > A.spin_limit) {
          const unsigned now = ld_acquire_u32(A.progress);
          if (now != seen) {
            seen = now;
            it = 0;
            continue;
          }
          set_error(A.info + SV_INFO_STATUS, SV_ETIMEOUT);
          atomicCAS(A.info + SV_INFO_BLOCK, -1, (int)c);
          break;
        }
      }
    }
    __syncthreads();
    const double aK = ac[K - 1];
    for (int r = threadIdx.x; r < A.nrhs; r += blockDim.x) {
      double v = A.R[c * (int64_t)A.nrhs + r];
#pragma unroll 4
      for (int j = 0; j < np; ++j) v -= s_a[j] * __ldcg(A.X + (int64_t)s_p[j] * A.nrhs + r);
      A.X[c * (int64_t)A.nrhs + r] = v / aK;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && !(A.skip_ready_row0 && c == 0)) {
      st_release_s32(A.ready + c, 1);
      atomicAdd(A.progress, 1u);
    }
  }
}

// ---------------------------------------------------------------------------
// diag((U_pp U_pp^T)^-1): rows of S = U_pp^-T against identity columns
// ---------------------------------------------------------------------------
struct JvArgs {
  int64_t npred, nobs, row0;  // panel: identity columns row0 .. row0 + w - 1
  int k, ldnbr, w;
  const int32_t* nbr;
  const double* acol;
  double* S;        // rows row0 .. npred-1 of the panel, row stride w
  double* var;      // += the panel's sum of squares of each row
  int* ready;
  unsigned* counter;
  unsigned* progress;
  int32_t* info;
  unsigned spin_limit;
};

// Row c of S = U_pp^-T restricted to the panel's columns: the recurrence of
// k_joint_solve with the identity as right-hand side, S_cr = (delta(c, row0
// + r) - sum_j a_j S_{p_j r}) / a_K.  S is lower triangular, so rows before
// row0 are zero in the panel (never formed, their dependencies skipped) and
// row c is zero beyond column c - row0 (never formed; a dependency p is read
// only where r <= p - row0).  The row's sum of squares is added to var[c].
__global__ void k_joint_inv_rows(JvArgs A) {
  extern __shared__ double jv_sm[];
  double* s_a = jv_sm;
  int* s_p = (int*)(jv_sm + (A.k > 0 ? A.k : 1));
  __shared__ long long s_c;
  __shared__ int s_np;
  __shared__ double s_red[32];
  const int K = A.k + 1;
  while (true) {
    if (threadIdx.x == 0) s_c = A.row0 + (long long)atomicAdd(A.counter, 1u);
    __syncthreads();
    const int64_t c = s_c;
    if (c >= A.npred) break;
    const double* ac = A.acol + c * (int64_t)K;
    if (threadIdx.x == 0) {
      int np = 0;
      for (int i = 0; i < A.k; ++i) {
        const int64_t ix = A.nbr[c * (int64_t)A.ldnbr + i];
        if (ix < 0 || ix < A.nobs || ix - A.nobs < A.row0) continue;  // zero in this panel
        s_p[np] = (int)(ix - A.nobs);
        s_a[np] = ac[i];
        ++np;
      }
      s_np = np;
    }
    __syncthreads();
    const int np = s_np;
    for (int j = threadIdx.x; j < np; j += blockDim.x) {
      const int p = s_p[j];
      unsigned it = 0, seen = ld_acquire_u32(A.progress);
      while (ld_acquire_s32(A.ready + p) == 0) {
        if (++it > A.spin_limit) {
          const unsigned now = ld_acquire_u32(A.progress);
          if (now != seen) {
            seen = now;
            it = 0;
            continue;
          }
          set_error(A.info + SV_INFO_STATUS, SV_ETIMEOUT);
          atomicCAS(A.info + SV_INFO_BLOCK, -1, (int)c);
          break;
        }
      }
    }
    __syncthreads();
    const double aK = ac[K - 1];
    const int64_t own = c - A.row0;
    const int64_t lim = own < A.w - 1 ? own : A.w - 1;
    double sq = 0.0;
    for (int64_t r = threadIdx.x; r <= lim; r += blockDim.x) {
      double v = (r == own) ? 1.0 : 0.0;
      for (int j = 0; j < np; ++j) {
        const int64_t pr = s_p[j] - A.row0;
        if (r <= pr) v -= s_a[j] * __ldcg(A.S + pr * A.w + r);
      }
      v = v / aK;
      A.S[own * A.w + r] = v;
      sq = fma(v, v, sq);
    }
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = sq;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_red[w];
      A.var[c] += t;
      st_release_s32(A.ready + c, 1);
      atomicAdd(A.progress, 1u);
    }
  }
}

}  // namespace sv

using namespace sv;

extern "C" int sv_predict_blocks(const sv_pred_desc* D, const double* theta, const double* Xall,
                                 const int32_t* tgt, const int32_t* nbr, const double* resid,
                                 double* mean, double* var, double* acol, double* rhs, int32_t* info,
                                 sv_stream_t stream) {
  if (!D || !theta || !Xall || !tgt || !info) return SV_EINVAL;
  if (D->d < 1 || D->d > 64 || D->k < 0 || D->nblk < 0 || (D->k > 0 && (!nbr || D->ldnbr < D->k)))
    return SV_EINVAL;
  if (!(D->nu > 0.0)) return SV_EINVAL;
  const int closed = matern_closed_code(D->nu);
  if (!D->general && closed < 0) return SV_EINVAL;
  if (D->matern_table && (!D->general || !mtab_ok(D->nu))) return SV_EINVAL;
  if (D->nobs > 0 && !resid && (mean || rhs)) return SV_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  int32_t init_info[4] = {0, -1, 0, 0};
  SV_CUDA_TRY(cudaMemcpyAsync(info, init_info, sizeof(init_info), cudaMemcpyHostToDevice, st));
  if (D->nblk == 0) return SV_OK;
  PredArgs A;
  A.theta = theta;
  A.Xall = Xall;
  A.tgt = tgt;
  A.nbr = nbr;
  A.resid = resid;
  A.mean = mean;
  A.var = var;
  A.acol = acol;
  A.rhs = rhs;
  A.info = info;
  A.nobs = D->nobs;
  A.nblk = D->nblk;
  A.d = D->d;
  A.k = D->k;
  A.ldnbr = D->ldnbr;
  A.closed = D->general ? -1 : closed;
  A.target_nugget = D->target_nugget;
  A.nu = D->nu;
  A.tab = D->matern_table;
  // the float32 part of the table (built where the nu has one)
  A.ftab = (D->matern_table && ftab_ok(D->nu)) ? (const float4*)(D->matern_table + kMtabMaxDoubles) : nullptr;
  if (D->precision < 0 || D->precision > 1) return SV_EINVAL;
  A.split = (D->precision == 1 && (A.closed >= 0 || A.ftab)) ? 1 : 0;
  A.rho_min = D->split_rho_min > 0.0 ? D->split_rho_min : 1e-4;
  int dev = 0, maxsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t prm = (sizeof(PredPrm) + 7) / 8 * 8;
  const int nsm = sv_num_sms();
  // the fixed-point kernel takes nu = 3/2 and 5/2, and split calls whose pivot
  // guard is at least 1e-9, of 33 to 208 points a block, d <= 12 and what shared
  // memory holds (20,000 blocks of 141, d = 6: 18.6 ms against k_pred_cta's 37.0;
  // 9,001 split blocks of 141, d = 7: 7.2 against 10.6; 3,000 of 36, d = 6: 0.37
  // against 0.58, split 0.30 against 0.47). Up to two blocks per SM of fewer than
  // 60 points take 5 to 20 us longer than there, so that a block's bits do not
  // depend on how many there are. 20,000 calls of 21 points take 5.3 ms
  // with a warp each and 5.6 with a CTA each
  A.kt = D->k + 1;
  if (pred_fix_takes(A, maxsm)) return launch_pred_fix(A, maxsm, st);
  if (D->k + 1 <= 32) {
    A.kt = 32;
    const size_t team = sizeof(double) * pred_team_doubles(32, D->d);
    int wpc = 8;
    while (wpc > 1 && prm + wpc * team > (size_t)maxsm) --wpc;
    const size_t smem = prm + wpc * team;
    if (smem > (size_t)maxsm) return SV_EINVAL;
    SV_CUDA_TRY(cudaFuncSetAttribute(k_pred_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int64_t grid = (D->nblk + wpc - 1) / wpc;
    if (grid > 64LL * nsm) grid = 64LL * nsm;
    k_pred_warp<<<(unsigned)grid, 32 * wpc, smem, st>>>(A);
  } else {
    A.kt = D->k + 1;
    const size_t smem = prm + sizeof(double) * pred_team_doubles(A.kt, D->d);
    if (smem > (size_t)maxsm) return SV_EINVAL;
    SV_CUDA_TRY(cudaFuncSetAttribute(k_pred_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int64_t grid = D->nblk;
    if (grid > 16LL * nsm) grid = 16LL * nsm;
    k_pred_cta<<<(unsigned)grid, kPredCta, smem, st>>>(A);
  }
  SV_CUDA_TRY(cudaGetLastError());
  return SV_OK;
}

extern "C" size_t sv_joint_solve_workspace_bytes(int64_t npred) {
  return 256 + ((sizeof(int) * (size_t)(npred > 0 ? npred : 1) + 255) & ~(size_t)255);
}

static int joint_solve(int64_t npred, int64_t nobs, int32_t k, int32_t ldnbr, const int32_t* nbr,
                       const double* acol, const double* R, int32_t nrhs, double* X, int32_t* info,
                       void* workspace, size_t workspace_bytes, int32_t flags, sv_stream_t stream) {
  if (npred < 0 || nobs < 0 || k < 0 || k > 4096 || nrhs < 1 || !info || flags < 0 || flags > 1)
    return SV_EINVAL;
  if (npred > 0 && (!acol || !R || !X || (k > 0 && (!nbr || ldnbr < k)))) return SV_EINVAL;
  if (npred > 0x7fffffffLL) return SV_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  int32_t init_info[4] = {0, -1, 0, 0};
  SV_CUDA_TRY(cudaMemcpyAsync(info, init_info, sizeof(init_info), cudaMemcpyHostToDevice, st));
  if (npred == 0) return SV_OK;
  if (!workspace || workspace_bytes < sv_joint_solve_workspace_bytes(npred)) return SV_ENOSPC;
  unsigned* counter = (unsigned*)workspace;
  unsigned* progress = counter + 1;
  int* ready = (int*)((char*)workspace + 256);
  SV_CUDA_TRY(cudaMemsetAsync(workspace, 0, sv_joint_solve_workspace_bytes(npred), st));
  JsArgs A;
  A.npred = npred;
  A.nobs = nobs;
  A.k = k;
  A.ldnbr = ldnbr;
  A.nrhs = nrhs;
  A.nbr = nbr;
  A.acol = acol;
  A.R = R;
  A.X = X;
  A.ready = ready;
  A.counter = counter;
  A.progress = progress;
  A.info = info;
  A.skip_ready_row0 = flags & 1;
  A.spin_limit = (flags & 1) ? SV_SPIN_LIMIT_TEST : SV_SPIN_LIMIT;
  const int nsm = sv_num_sms();
  // threads per row: the right-hand sides, rounded to whole warps, at most 256
  int tpb = ((nrhs + 31) / 32) * 32;
  if (tpb > 256) tpb = 256;
  const size_t smem = (size_t)(k > 0 ? k : 1) * (sizeof(double) + sizeof(int)) + 8;
  int per_sm = 0;
  SV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_joint_solve, tpb, smem));
  if (per_sm < 1) return SV_EINVAL;
  int64_t grid = (int64_t)per_sm * nsm;
  if (grid > npred) grid = npred;
  k_joint_solve<<<(unsigned)grid, tpb, smem, st>>>(A);
  SV_CUDA_TRY(cudaGetLastError());
  return SV_OK;
}

extern "C" int sv_joint_solve(int64_t npred, int64_t nobs, int32_t k, int32_t ldnbr,
                              const int32_t* nbr, const double* acol, const double* R, int32_t nrhs,
                              double* X, int32_t* info, void* workspace, size_t workspace_bytes,
                              sv_stream_t stream) {
  return joint_solve(npred, nobs, k, ldnbr, nbr, acol, R, nrhs, X, info, workspace, workspace_bytes,
                     0, stream);
}

extern "C" int sv_joint_solve_flags(int64_t npred, int64_t nobs, int32_t k, int32_t ldnbr,
                                    const int32_t* nbr, const double* acol, const double* R,
                                    int32_t nrhs, double* X, int32_t* info, void* workspace,
                                    size_t workspace_bytes, int32_t flags, sv_stream_t stream) {
  return joint_solve(npred, nobs, k, ldnbr, nbr, acol, R, nrhs, X, info, workspace, workspace_bytes,
                     flags, stream);
}

extern "C" int sv_joint_var_diag(int64_t npred, int64_t nobs, int32_t k, int32_t ldnbr,
                                 const int32_t* nbr, const double* acol, double* var, int32_t* info,
                                 void* workspace, size_t workspace_bytes, double* panel,
                                 size_t panel_bytes, sv_stream_t stream) {
  if (npred < 0 || nobs < 0 || k < 0 || k > 4096 || !info) return SV_EINVAL;
  if (npred > 0 && (!acol || !var || !panel || (k > 0 && (!nbr || ldnbr < k)))) return SV_EINVAL;
  if (npred > 0x7fffffffLL) return SV_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  int32_t init_info[4] = {0, -1, 0, 0};
  SV_CUDA_TRY(cudaMemcpyAsync(info, init_info, sizeof(init_info), cudaMemcpyHostToDevice, st));
  if (npred == 0) return SV_OK;
  if (!workspace || workspace_bytes < sv_joint_solve_workspace_bytes(npred)) return SV_ENOSPC;
  const int64_t pd = (int64_t)(panel_bytes / sizeof(double));
  if (pd < npred) return SV_ENOSPC;  // one column of all rows at least
  SV_CUDA_TRY(cudaMemsetAsync(var, 0, sizeof(double) * (size_t)npred, st));
  JvArgs A;
  A.npred = npred;
  A.nobs = nobs;
  A.k = k;
  A.ldnbr = ldnbr;
  A.nbr = nbr;
  A.acol = acol;
  A.S = panel;
  A.var = var;
  A.counter = (unsigned*)workspace;
  A.progress = A.counter + 1;
  A.ready = (int*)((char*)workspace + 256);
  A.info = info;
  A.spin_limit = SV_SPIN_LIMIT;
  const int nsm = sv_num_sms();
  const size_t smem = (size_t)(k > 0 ? k : 1) * (sizeof(double) + sizeof(int)) + 8;
  for (int64_t c0 = 0; c0 < npred;) {
    // the widest panel whose rows c0 .. npred-1 fit
    const int64_t rows = npred - c0;
    int64_t w = pd / rows;
    if (w > rows) w = rows;
    if (w > 0x7fffffffLL) w = 0x7fffffffLL;
    A.row0 = c0;
    A.w = (int)w;
    SV_CUDA_TRY(cudaMemsetAsync(workspace, 0, sv_joint_solve_workspace_bytes(npred), st));
    int tpb = (int)(((w + 31) / 32) * 32);
    if (tpb > 256) tpb = 256;
    int per_sm = 0;
    SV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_joint_inv_rows, tpb, smem));
    if (per_sm < 1) return SV_EINVAL;
    int64_t grid = (int64_t)per_sm * nsm;
    if (grid > rows) grid = rows;
    k_joint_inv_rows<<<(unsigned)grid, tpb, smem, st>>>(A);
    SV_CUDA_TRY(cudaGetLastError());
    c0 += w;
  }
  return SV_OK;
}
