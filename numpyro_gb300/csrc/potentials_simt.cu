// potentials_simt.cu -- FP32 CUDA-core potentials and hand-written adjoints.
//
// Every kernel evaluates numpyro's potential_energy (numpyro/infer/util.py:333-358)
// for a batch of latent points (one per chain) and its gradient, written by
// hand (no autodiff).  Log-densities follow numpyro/distributions:
//   Normal continuous.py:2975-2989, Cauchy :390-406, HalfCauchy :1149-1150,
//   HalfNormal :1190-1191, Exponential :715-726, StudentT :3229-3238,
//   GaussianRandomWalk :1104-1112, BernoulliLogits discrete.py:263 with
//   binary_cross_entropy_with_logits distributions/util.py:317-320;
// positive sites use biject_to(positive) = ExpTransform with log|det J| = x
// (transforms.py:641-644, :2115-2118).  Per-term arithmetic is FP32, sums
// are accumulated in FP64 so potential differences stay exact to ~1e-9
// relative even for 581k-row likelihoods.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>
#include <cmath>

#include "common.cuh"
#include "hier_potential.cuh"
#include "internal.h"
#include "hs_finish.cuh"
#include "lr_finish.cuh"
#include "logreg_fp32.cuh"
#include "sv_potential.cuh"

namespace gbn {

constexpr double LOG_2PI = 1.8378770664093453;
constexpr double LOG_PI = 1.1447298858494002;
constexpr double LOG_2 = 0.6931471805599453;

// ============================================================ hierarchical (non-centred)
// z = [mu, log tau, theta_base(J)];  warp per point; model m = point / cpm
__global__ void __launch_bounds__(512) hier_nc_kernel(const float* __restrict__ Q, int npts, int ld,
                                                      const float* __restrict__ y, const float* __restrict__ sinv,
                                                      const double* __restrict__ cmodel,
                                                      const int32_t* __restrict__ off, int cpm, int num_models,
                                                      float inv_ms2, float inv_ts, double* __restrict__ PE,
                                                      float* __restrict__ G, const int32_t* pending) {
  if (pending && *pending == 0) return;
  int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // a warp per point
  int lane = threadIdx.x & 31;
  if (c >= npts) return;
  int m = c / cpm;
  if (m >= num_models) m = num_models - 1;  // points beyond the configured chains reuse the last model
  int j0 = off[m], J = off[m + 1] - j0;
  hier_nc_potential_warp(Q + (size_t)c * ld, G + (size_t)c * ld, PE + c, J, y + j0, sinv + j0, cmodel[m], inv_ms2,
                         inv_ts, lane);
}

// ============================================================ logistic regression
// sum the tensor-core kernel's partials, or the FP32 one's of many points, add the N(0, scale) prior; warp per point
// lin (FP64 [p]): a linear term lin . b of the log-likelihood computed outside the kernel
__global__ void logreg_finish_kernel(const float* __restrict__ Q, int npts, int ld, int p, int row_groups,
                                     const float* __restrict__ part_g, const double* __restrict__ part_ll,
                                     const double* __restrict__ lin, float inv_var_f, double pe_const,
                                     double* __restrict__ PE, float* __restrict__ G, const int32_t* pending,
                                     const int32_t* __restrict__ split3 = nullptr, bool e_tanh = false) {
  tick_wait();
  tick_trigger();
  if (pending && *pending == 0) return;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c >= npts) return;
  logreg_finish_warp(Q, c, npts, ld, p, row_groups, part_g, part_ll, lin, inv_var_f, pe_const, PE, G,
                     threadIdx.x & 31, split3, e_tanh);
}

// 1 / s^2 (FP32, as the gradient uses it) and p (log(2 pi) / 2 + log s) of the Normal(0, s) prior
void logreg_prior_consts(double prior_scale, int p, float* inv_var_f, double* pe_const) {
  *inv_var_f = (float)(1.0 / (prior_scale * prior_scale));
  *pe_const = (double)p * (0.5 * LOG_2PI + std::log(prior_scale));
}

// ============================================================ horseshoe: FP32 GEMMs + prior terms
// Both contractions of the Gaussian GLM run as one "NN" SGEMM, C[m][n] = sum_k A[k][m] B[k][n],
// with A and B row-major and m/n contiguous (rows padded to a multiple of 4 floats, so every
// tile row is float4-aligned):
//   residuals  R[row][c]  = y[row] - sum_p Xt[p][row] Bt[p][c]       (Xt = X^T, Bt = beta^T)
//   adjoint    GB[c][p]   = sum_row R[row][c] X[row][p]              (split over row ranges)
// X^T and a padded X are built once per model; beta^T is packed from the chains' positions each
// tick.  Residual sums of squares per (row tile, chain) leave the GEMM in FP64 (BM / 16 rows each in FP32).
//
// Tiles of BM x 64 outputs, 4 x 8 a thread.  At 2000 x 1000 x 256 chains a GEMM has 512,000 outputs, under one
// warp of 32 outputs a thread for each scheduler.  Bound: shared-memory reads (a 16-byte read of a warp takes
// four cycles, broadcast or not, so 4 x 4 outputs a thread read 8 cycles for 4 of multiply-adds, 4 x 8 12
// for 8).  cp.async runs STAGES - 1 K steps of BK ahead: 3 stages of 32 where the multiply-adds bound it (80 us a
// potential at that size; 2 stages of 32 88, 4 of 16 85), 4 of 16 where a CTA has a few steps and their latency does
// (542 x 130 x 3 chains: a run of 0.89 ms; 3 of 32 0.93, 2 of 32 0.95).
constexpr int HS_BN = 64;
constexpr int HS_SPLIT_ROWS = 16;  // a row range of the adjoint GEMM is a multiple of this
constexpr int HS_MIN_BM = 32;     // smallest tile height; the partials are sized for it
constexpr int HS_MAX_SPLITS = 8;  // most row ranges of the adjoint GEMM

template <int BM, int BK, int STAGES>
__global__ void __launch_bounds__(BM * HS_BN / 32)
    hs_sgemm_nn_kernel(const float* __restrict__ A, int lda, const float* __restrict__ B, int ldb, int M, int N, int K,
                       int k_per_split, float* __restrict__ Out, int ldo, int64_t split_stride,
                       const float* __restrict__ yv, double* __restrict__ part_rr, int ld_rr, const int32_t* pending) {
  if (pending && *pending == 0) return;
  constexpr int NTH = BM * HS_BN / 32, TX = HS_BN / 8, TY = BM / 4;
  __shared__ __align__(16) float As[STAGES][BK][BM];
  __shared__ __align__(16) float Bs[STAGES][BK][HS_BN];
  constexpr int SQ_ROWS = BM / 16;  // rows a sum of squares takes in FP32
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * HS_BN;
  const int kb = blockIdx.z * k_per_split, ke = min(K, kb + k_per_split);
  const int steps = ke > kb ? (ke - kb + BK - 1) / BK : 0;
  auto stage = [&](int step) {  // one K step of both operands; past the end an empty group
    if (step < steps) {
      const int k0 = kb + step * BK, s = step % STAGES;
#pragma unroll
      for (int q = tid; q < BK * BM / 4; q += NTH) {
        const int k = q / (BM / 4), m = 4 * (q % (BM / 4));
        const bool in = k0 + k < ke && m0 + m < M;
        cp_async16(&As[s][k][m], in ? A + (size_t)(k0 + k) * lda + m0 + m : A, in);
      }
#pragma unroll
      for (int q = tid; q < BK * HS_BN / 4; q += NTH) {
        const int k = q / (HS_BN / 4), n = 4 * (q % (HS_BN / 4));
        const bool in = k0 + k < ke && n0 + n < N;
        cp_async16(&Bs[s][k][n], in ? B + (size_t)(k0 + k) * ldb + n0 + n : B, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) stage(i);
  float acc[4][8] = {};
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // this step has landed, and every thread is done with the stage filled next
    stage(step + STAGES - 1);
    const int s = step % STAGES;
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[s][kk][4 * ty]);
      const float4 b4 = *reinterpret_cast<const float4*>(&Bs[s][kk][4 * tx]);
      const float4 c4 = *reinterpret_cast<const float4*>(&Bs[s][kk][HS_BN / 2 + 4 * tx]);
      const float aa[4] = {a4.x, a4.y, a4.z, a4.w}, bb[8] = {b4.x, b4.y, b4.z, b4.w, c4.x, c4.y, c4.z, c4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(aa[i], bb[j], acc[i][j]);
    }
  }
  float* out = Out + (size_t)blockIdx.z * split_stride;
  if (yv == nullptr) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = m0 + ty * 4 + i;
      if (m >= M) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int nn = n0 + h * (HS_BN / 2) + 4 * tx;
        if (nn < N)
          *reinterpret_cast<float4*>(out + (size_t)m * ldo + nn) =
              make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]);
      }
    }
    return;
  }
  // residual epilogue: R = y - acc, and per-chain sums of R^2 over this row tile
  float(*const rr)[HS_BN] = reinterpret_cast<float(*)[HS_BN]>(&As[0][0][0]);  // [TY * 4 / SQ_ROWS], over the operands
  __syncthreads();
  float sq[8] = {};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    const bool in = m < M;
    const float y = in ? yv[m] : 0.0f;
    float r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      r[j] = in ? y - acc[i][j] : 0.0f;
      sq[j] = fmaf(r[j], r[j], sq[j]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int nn = n0 + h * (HS_BN / 2) + 4 * tx;
      if (in && nn < N)
        *reinterpret_cast<float4*>(out + (size_t)m * ldo + nn) = make_float4(r[4 * h], r[4 * h + 1], r[4 * h + 2], r[4 * h + 3]);
    }
    if ((i + 1) % SQ_ROWS == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        rr[(4 * ty + i) / SQ_ROWS][(j >> 2) * (HS_BN / 2) + 4 * tx + (j & 3)] = sq[j];
        sq[j] = 0.0f;
      }
    }
  }
  __syncthreads();
  for (int n = tid; n < HS_BN && n0 + n < N; n += NTH) {
    double t = 0.0;
    for (int k = 0; k < TY * 4 / SQ_ROWS; ++k) t += (double)rr[k][n];
    part_rr[(size_t)blockIdx.y * ld_rr + n0 + n] = t;
  }
}

// Bt[p][c] = beta_c[p] (p < P, c < npts), zero in the padding; 32 x 32 tiles through shared memory.
// Centred: beta is z[0:P].  Non-centred: beta = exp(log tau + log lambda) * unscaled_beta.
__global__ void __launch_bounds__(256) hs_pack_kernel(const float* __restrict__ Q, int ld, int npts, int P,
                                                      int noncentred, float* __restrict__ Bt, int ldb, int prows,
                                                      const int32_t* pending) {
  if (pending && *pending == 0) return;
  __shared__ float t[32][33];
  const int c0 = blockIdx.x * 32, p0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int k = ty; k < 32; k += 8) {
    const int c = c0 + k, p = p0 + tx;
    float v = 0.0f;
    if (c < npts && p < P) {
      const float* z = Q + (size_t)c * ld;
      v = noncentred ? expf(z[P + 1] + z[p]) * z[P + 2 + p] : z[p];
    }
    t[k][tx] = v;
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    const int p = p0 + k, c = c0 + tx;
    if (p < prows && c < ldb) Bt[(size_t)p * ldb + c] = t[tx][k];
  }
}

// Prior terms and the gradient of the horseshoe GLM, one CTA per chain, FP32 per coordinate with
// float-float sums.  Centred: z = [beta(P), log lambda(P), log sigma, log tau] (sorted sites).
// Non-centred (unscaled_betas ~ Normal(0, 1), beta = tau lambda unscaled_beta, as
// examples/horseshoe_regression.py:33-49): z = [log lambda(P), log sigma, log tau, unscaled_beta(P)];
// with g = X^T R / sigma^2: dU/d unscaled_d = eta_d - tau lambda_d g_d, dU/d log lambda_d =
// -beta_d g_d + 2 lambda^2/(1+lambda^2) - 1, dU/d log tau = -sum_d beta_d g_d + 2 tau^2/(1+tau^2) - 1.
//   beta_d ~ Normal(0, tau lambda_d): 0.5 b^2/s^2 + log s, s = tau lambda  (the log lambda cancels
//   against the Exp log-det);  lambda_d, tau ~ HalfCauchy(1);  sigma ~ HalfNormal(1).
// log(1 + lambda^2) = 2 max(l, 0) + log1p(e^{-2|l|}) and 2 lambda^2/(1 + lambda^2) = 2 / (1 + e^{-2l})
// stay finite for any l.
__global__ void __launch_bounds__(256) horseshoe_finish_kernel(const float* __restrict__ Q, int npts, int ld, int P,
                                                               int64_t N, const float* __restrict__ part_gb,
                                                               int splits, int ldg, const double* __restrict__ part_rr,
                                                               int ld_rr, int mtiles, int noncentred,
                                                               double* __restrict__ PE, float* __restrict__ G,
                                                               const int32_t* pending) {
  if (pending && *pending == 0) return;
  __shared__ double red[16];
  horseshoe_finish_block(Q, blockIdx.x, ld, P, N, part_gb, splits, ldg, npts, part_rr, ld_rr, mtiles, noncentred, PE,
                         G, threadIdx.x, red);
}

// ============================================================ stochastic volatility
// z = [h(T) or h_base(T), log nu, log s]; CTA per point (sv_potential.cuh): non-centred walks of more than
// SV_REG_CHUNK steps a thread.
__global__ void __launch_bounds__(256) sv_nc_long_kernel(const float* __restrict__ Q, int ld, int T,
                                                         const float* __restrict__ ret, double s_rate, double nu_rate,
                                                         double* __restrict__ PE, float* __restrict__ G,
                                                         const int32_t* pending) {
  if (pending && *pending == 0) return;
  __shared__ SvSmem<256> sm;
  const size_t c = blockIdx.x;
  sv_nc_potential_block<256, 8>(Q + c * ld, G + c * ld, PE + c, T, ret, s_rate, nu_rate, threadIdx.x, sm);
}

// CTA per point: eight element warps, and two scalar warps for what is FP64 or long (on GB300 a log-gamma takes
// 1,700 to 3,100 cycles, a dependent FP64 operation 64): warp 8 the digammas, warp 9 the log-gammas, beside
// the elements; then U in warp 9, dU/d log nu in warp 8 and dU/d log s in warp 0 beside one another.  With one
// thread for all of it after the elements, and the log-gammas in front of two element warps, a point took
// 20,000 cycles.  NC: the walk's rows pass through shared memory, as a thread's steps are consecutive.
// Arithmetic and order of the sums are the block functions', so all engines give the same bits.
// 4,096 steps x 1,024 points, non-centred: 53 -> 37 us (41 with two blocks an SM; 48 registers for four are no faster).  What is left
// is issue: 218 instructions a step, most of them the seven compensated sums, at 2.7 a cycle and SM.
template <int K, bool NC>
__global__ void __launch_bounds__(320, 3) sv_potential_kernel(const float* __restrict__ Q, int ld, int T,
                                                           const float* __restrict__ ret, double s_rate,
                                                           double nu_rate, double* __restrict__ PE,
                                                           float* __restrict__ G, const int32_t* pending) {
  if (pending && *pending == 0) return;
  __shared__ float2 r1[5][8], wt[2][8];
  extern __shared__ float rows[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* const z = Q + (size_t)blockIdx.x * ld;
  float* const g = G + (size_t)blockIdx.x * ld;
  const float lnuf = z[T], lsf = z[T + 1];
  float* const zs = rows;
  float* const rets = rows + sv_pos(T) + 1;
  if (NC && warp < 8) {
    float a[K], b[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const bool in = tid + 256 * k < T;
      a[k] = in ? z[tid + 256 * k] : 0.0f;
      b[k] = in ? ret[tid + 256 * k] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (tid + 256 * k < T) {
        zs[sv_pos(tid + 256 * k)] = a[k];
        rets[sv_pos(tid + 256 * k)] = b[k];
      }
    asm volatile("bar.sync 2, 256;" ::: "memory");
  }
  const float nuf = expf(lnuf), sf = expf(lsf), inv_nuf = 1.0f / nuf;
  float dg = 0.0f;
  double lg = 0.0;
  if (warp == 9) {
    const double nu = (double)nuf;
    lg = lgamma(0.5 * (lane == 1 ? nu + 1.0 : nu));
  } else if (warp == 8) {
    dg = digamma_f(0.5f * (lane == 1 ? nuf + 1.0f : nuf));
  } else if (NC) {
    sv_nc_elements<K>(zs, rets, rets, T, tid, sf, nuf, inv_nuf, r1, wt);
  } else {
    const float inv_s2 = 1.0f / (sf * sf);
    Comp32 sdd{0.0f, 0.0f}, sl1p{0.0f, 0.0f}, sfrac{0.0f, 0.0f}, sh{0.0f, 0.0f};
    for (int t0 = tid; t0 < T; t0 += K * 256) {  // loads of K steps are issued before their gradient stores
      float hv[K], hp[K], hn[K], rv[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int t = t0 + k * 256;
        hv[k] = t < T ? z[t] : 0.0f;
        hp[k] = (t < T && t > 0) ? z[t - 1] : 0.0f;
        hn[k] = (t + 1 < T) ? z[t + 1] : 0.0f;
        rv[k] = t < T ? ret[t] : 0.0f;
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int t = t0 + k * 256;
        if (t < T) g[t] = sv_centred_step(t, T, hv[k], hp[k], hn[k], rv[k], nuf, inv_nuf, inv_s2, sdd, sl1p, sfrac, sh);
      }
    }
    const FF v = warp_sum4ff(comp_ff(sdd), comp_ff(sl1p), comp_ff(sfrac), comp_ff(sh), lane);
    if ((lane & 7) == 0) r1[lane >> 3][warp] = make_float2(v.hi, v.lo);
  }
  __syncthreads();
  if (NC && warp < 8)
    for (int t = tid; t < T; t += 256) g[t] = rets[sv_pos(t)];
  if (warp >= 8 || warp == 0) {
    const double sums = ff_value(sv_fold(r1, lane < (NC ? 5 : 4) ? lane : 0));
    const double nu = (double)nuf, s = (double)sf, inv_s = (double)(1.0f / sf);
    const uint32_t FULL = 0xffffffffu;
    const double S0 = __shfl_sync(FULL, sums, 0), S1 = __shfl_sync(FULL, sums, 1), S2 = __shfl_sync(FULL, sums, 2),
                 S3 = __shfl_sync(FULL, sums, 3), S4 = __shfl_sync(FULL, sums, 4);
    const double S_l1p = NC ? S0 : S1, S_frac = NC ? S1 : S2, S_h = NC ? S2 : S3;
    if (warp == 8) {
      const double special[6] = {0.0, 0.0, (double)__shfl_sync(FULL, dg, 0), (double)__shfl_sync(FULL, dg, 1), nu,
                                 (double)inv_nuf};
      const float gl = sv_grad_lnu(S_l1p, S_frac, (double)T, nu_rate, special);
      if (lane == 0) g[T] = gl;
    } else if (warp == 9) {
      const double lg0 = __shfl_sync(FULL, lg, 0), lg1 = __shfl_sync(FULL, lg, 1);
      const double log_rates = (double)(logf((float)s_rate) + logf((float)nu_rate));
      const double pe = -sv_log_joint(NC, NC ? S4 : S0, S_l1p, S_h, (double)T, lnuf, lsf, nu, s, inv_s, log_rates, s_rate,
                                      nu_rate, lg0, lg1);
      if (lane == 0) PE[blockIdx.x] = pe;
    } else {
      const float gl = sv_grad_ls(NC, NC ? S3 : S0, (double)T, s, inv_s, s_rate);
      if (lane == 0) g[T + 1] = gl;
    }
  }
}

__global__ void scale_rows_kernel(const double* __restrict__ cot, float* __restrict__ G, int npts, int D) {
  size_t total = (size_t)npts * D;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x)
    G[k] = (float)((double)G[k] * cot[k / D]);
}

// ============================================================ host side
cudaError_t ensure_potential_scratch(ModelDev& m, int points) {
  if (points <= m.scratch_points) return cudaSuccess;
  free_potential_scratch(m);
  cudaError_t e = cudaSuccess;
  if (m.family == 2) {
    // Partials: the FP32 kernel's row groups follow its rule, the tensor-core one takes at most 4 x 152 over blocks
    // of 64 chains (it has blocks of 128 and 152 CTAs, more only for fewer points than these); GBN_TUNE may ask
    // for twice as many.
    const int64_t ntiles = (m.n + 63) / 64, blocks = (points + 63) / 64;
    m.row_groups = m.tc ? (int)std::min<int64_t>((4 * 152 + blocks - 1) / blocks, ntiles)
                        : logreg_fp32_row_groups(m.n, m.p, points, 0);
    m.row_groups_cap = (int)std::min<int64_t>(2 * (int64_t)m.row_groups, ntiles);
    if (m.tune.lr_rg > m.row_groups_cap) m.tune.lr_rg = 0;
    e = cudaMalloc(&m.part_g, sizeof(float) * (size_t)m.row_groups_cap * points * 64);
    if (e == cudaSuccess) e = cudaMalloc(&m.part_ll, sizeof(double) * (size_t)m.row_groups_cap * points);
  } else if (m.family == 3) {
    const int cp = pad4(points), pp = pad4(m.p);
    const int mt = (int)((m.n + HS_MIN_BM - 1) / HS_MIN_BM);
    e = cudaMalloc(&m.resid, sizeof(float) * (size_t)m.n * cp);
    if (e == cudaSuccess) e = cudaMalloc(&m.part_rr, sizeof(double) * (size_t)mt * cp);
    if (e == cudaSuccess) e = cudaMalloc(&m.part_gb, sizeof(float) * (size_t)HS_MAX_SPLITS * points * pp);
    if (e == cudaSuccess) e = cudaMalloc(&m.hs_bt, sizeof(float) * (size_t)pp * cp);
  }
  if (e == cudaSuccess) {
    m.scratch_points = points;
    if (m.tc) e = logreg_tc_prepare(m, points);
  }
  return e;
}

void free_potential_scratch(ModelDev& m) {
  cudaFree(m.part_g);
  cudaFree(m.part_ll);
  cudaFree(m.resid);
  cudaFree(m.part_rr);
  cudaFree(m.part_gb);
  cudaFree(m.hs_bt);
  m.hs_bt = nullptr;
  m.part_g = nullptr;
  m.part_ll = nullptr;
  m.resid = nullptr;
  m.part_rr = nullptr;
  m.part_gb = nullptr;
  m.scratch_points = 0;
}

namespace {
std::mutex g_simt_attr_mu;
std::vector<char> g_simt_attr_done;  // per device ordinal: the shared-memory limit is raised
}  // namespace

// The FP32 logistic kernels need up to 104 KB of dynamic shared memory, above the 48 KB default.  The
// limit is a per-device attribute of a kernel, so it is raised once for every device they run on (with
// that device current), under a mutex.
cudaError_t logreg_simt_smem_attr() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_simt_attr_mu);
  if ((int)g_simt_attr_done.size() <= dev) g_simt_attr_done.resize((size_t)dev + 1, 0);
  if (g_simt_attr_done[(size_t)dev]) return cudaSuccess;
  LogregArgs probe{};
  probe.p = 1;
  probe.npts = 1;
  e = logreg_fp32_launch(-1, probe, 1, 0, false);
  if (e == cudaSuccess) g_simt_attr_done[(size_t)dev] = 1;
  return e;
}

static cudaError_t launch_logreg_fp32(int variant, const float* x, const float* y, int64_t n, int p, double prior_scale,
                                      const float* Q, int npts, int ld, int row_groups, float* part_g, double* part_ll,
                                      double* PE, float* G, const int32_t* pending, cudaStream_t st,
                                      bool dependent) {
  cudaError_t e = logreg_simt_smem_attr();
  if (e != cudaSuccess) return e;
  const LogregArgs A{x, y, n, p, Q, npts, ld, part_g, part_ll, pending};
  e = logreg_fp32_launch(variant, A, row_groups, st, dependent);
  if (e != cudaSuccess) return e;  // checked per launch, so the first failing launch is the one reported
  float ivf;
  double pec;
  logreg_prior_consts(prior_scale, p, &ivf, &pec);
  if (logreg_fp32_finish_by_warp(npts, row_groups))
    return launch_tick(logreg_finish_kernel, (npts + 7) / 8, 256, 0, st, dependent, Q, npts, ld, p, row_groups, part_g,
                       part_ll, nullptr, ivf, pec, PE, G, pending, nullptr, false);
  return launch_tick(logreg_fp32_finish_kernel, npts, 256, 0, st, dependent, A, row_groups, ivf, pec, PE, G);
}

// Steps a thread: those of the walk, rounded up to the next instance.
static void launch_sv(const float* Q, int npts, int ld, int T, const float* ret, double s_rate, double nu_rate,
                      bool noncentred, double* PE, float* G, const int32_t* pending, cudaStream_t st) {
  const int chunk = (T + 255) / 256;
  const size_t smem = noncentred ? sizeof(float) * 2 * (size_t)(T + T / 16 + 1) : 0;
#define SV_POTENTIAL(K, NC) \
  sv_potential_kernel<K, NC><<<npts, 320, smem, st>>>(Q, ld, T, ret, s_rate, nu_rate, PE, G, pending)
  if (noncentred && chunk > SV_REG_CHUNK)
    sv_nc_long_kernel<<<npts, 256, 0, st>>>(Q, ld, T, ret, s_rate, nu_rate, PE, G, pending);
  else if (noncentred) {
    if (chunk <= 1) SV_POTENTIAL(1, true);
    else if (chunk <= 2) SV_POTENTIAL(2, true);
    else if (chunk <= 4) SV_POTENTIAL(4, true);
    else if (chunk <= 6) SV_POTENTIAL(6, true);
    else if (chunk <= 9) SV_POTENTIAL(9, true);
    else if (chunk <= 12) SV_POTENTIAL(12, true);
    else SV_POTENTIAL(16, true);
  } else {
    if (chunk <= 1) SV_POTENTIAL(1, false);
    else if (chunk <= 2) SV_POTENTIAL(2, false);
    else SV_POTENTIAL(4, false);
  }
#undef SV_POTENTIAL
}

cudaError_t launch_potential(ModelDev& m, const float* Q, int npts, double* PE, float* G, const int32_t* pending,
                             cudaStream_t st, bool fused_tick, bool dependent) {
  if (npts <= 0) return cudaSuccess;
  cudaError_t e = ensure_potential_scratch(m, npts);
  if (e != cudaSuccess) return e;
  const int ld = m.D;
  switch (m.family) {
    case 1:
    {
      const int cpb = m.tune.hier_cpb;
      hier_nc_kernel<<<(npts + cpb - 1) / cpb, 32 * cpb, 0, st>>>(
          Q, npts, ld, m.y, m.hier_sinv, m.hier_cmodel, m.offsets, m.chains_per_model, m.num_models,
          (float)(1.0 / (m.hyper[0] * m.hyper[0])), (float)(1.0 / m.hyper[1]), PE, G, pending);
    }
      break;
    case 2: {
      if (m.precision == 1 && m.tc) return logreg_tc_launch(m, Q, npts, PE, G, pending, st, fused_tick);
      // forced row groups belong to the handle's own number of points; the partials bound any other
      const int want = npts == m.scratch_points ? m.tune.lr_rg : 0;
      const int rg = (int)std::min<int64_t>(logreg_fp32_row_groups(m.n, m.p, npts, want),
                                            (int64_t)m.row_groups_cap * m.scratch_points / npts);
      e = launch_logreg_fp32(logreg_fp32_shape(m.n, npts, INT_MAX).variant, m.x, m.y, m.n, m.p, m.hyper[0], Q, npts, ld,
                             rg, m.part_g, m.part_ll, PE, G, pending, st, dependent);
      if (e != cudaSuccess) return e;
      break;
    }
    case 3: {
      if (m.precision == 1 && m.hs_tc) return horseshoe_tc_launch(m, Q, npts, PE, G, pending, st, fused_tick, dependent && fused_tick);
      const int P = m.p, M = (int)m.n, cp = pad4(npts), pp = pad4(P);
      const int tm = m.tune.hs_tm, splits = m.tune.hs_splits, bm = 16 * tm;
      const int mt = (M + bm - 1) / bm;
      // beta^T for the chains' query points
      dim3 gp((cp + 31) / 32, (pp + 31) / 32);
      const int nc = m.hyper[0] != 0.0;
      hs_pack_kernel<<<gp, 256, 0, st>>>(Q, ld, npts, P, nc, m.hs_bt, cp, pp, pending);
      // R[row][c] = y[row] - sum_p X[row][p] beta_c[p]
      dim3 g1((npts + HS_BN - 1) / HS_BN, mt, 1);
      auto gemm1 = [&](auto kernel, int threads) {
        kernel<<<g1, threads, 0, st>>>(m.hs_xt, pad4(M), m.hs_bt, cp, M, npts, P, P, m.resid, cp, 0, m.y, m.part_rr, cp,
                                       pending);
      };
      // as the tile height's rule (rule_shapes); three stages of 32 gain 4 us at the line (1000 x 1000 x 128: 59.5
      // against 63.6) and as much below it where features are many (256 x 1000 x 128: 55.4 against 59.4), and lose 2
      // where they are few (542 x 130 x 32: 28.7 against 26.7)
      const bool large = npts >= 128 && m.n * P >= 1000000;
      if (tm == 2)
        large ? gemm1(hs_sgemm_nn_kernel<32, 32, 3>, 64) : gemm1(hs_sgemm_nn_kernel<32, 16, 4>, 64);
      else
        large ? gemm1(hs_sgemm_nn_kernel<64, 32, 3>, 128) : gemm1(hs_sgemm_nn_kernel<64, 16, 4>, 128);
      // GB[s][c][p] = sum_{row in split s} R[row][c] X[row][p]
      const int kps = (((M + splits - 1) / splits) + HS_SPLIT_ROWS - 1) / HS_SPLIT_ROWS * HS_SPLIT_ROWS;
      dim3 g2((P + HS_BN - 1) / HS_BN, (npts + 63) / 64, splits);
      auto gemm2 = [&](auto kernel) {
        kernel<<<g2, 128, 0, st>>>(m.resid, cp, m.hs_xp, pp, npts, P, M, kps, m.part_gb, pp, (int64_t)npts * pp, nullptr,
                                   nullptr, 0, pending);
      };
      large ? gemm2(hs_sgemm_nn_kernel<64, 32, 3>) : gemm2(hs_sgemm_nn_kernel<64, 16, 4>);
      horseshoe_finish_kernel<<<npts, 256, 0, st>>>(Q, npts, ld, P, m.n, m.part_gb, splits, pp, m.part_rr, cp, mt,
                                                    nc, PE, G, pending);
      break;
    }
    case 4:
      launch_sv(Q, npts, ld, (int)m.n, m.y, m.hyper[0], m.hyper[1], m.hyper[2] != 0.0, PE, G, pending, st);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// ============================================================ autotuner
namespace {
std::mutex g_tune_mu;
std::map<std::string, TuneParams> g_tune_cache;

// mean CUDA-event time of one potential launch (after one untimed launch)
cudaError_t time_potential(ModelDev& m, const float* Q, int npts, double* PE, float* G, cudaStream_t st, int reps,
                           float* ms) {
  cudaEvent_t a = nullptr, b = nullptr;
  cudaError_t e = cudaEventCreate(&a);
  if (e == cudaSuccess) e = cudaEventCreate(&b);
  if (e == cudaSuccess) e = launch_potential(m, Q, npts, PE, G, nullptr, st);
  if (e == cudaSuccess) e = cudaEventRecord(a, st);
  for (int r = 0; r < reps && e == cudaSuccess; ++r) e = launch_potential(m, Q, npts, PE, G, nullptr, st);
  if (e == cudaSuccess) e = cudaEventRecord(b, st);
  if (e == cudaSuccess) e = cudaEventSynchronize(b);
  float t = 0.0f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&t, a, b);
  *ms = t / (float)reps;
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  return e;
}

std::string tune_report(const ModelDev& m) {
  char buf[160];
  switch (m.family) {
    case 1: snprintf(buf, sizeof(buf), "hier_chains_per_cta=%d", m.tune.hier_cpb); break;
    case 2:
      snprintf(buf, sizeof(buf), "logreg_row_groups=%d", m.tune.lr_rg > 0 ? m.tune.lr_rg : m.row_groups);
      break;
    case 3:
      snprintf(buf, sizeof(buf), "horseshoe_tile_rows=%d horseshoe_splits=%d", 16 * m.tune.hs_tm,
               m.tune.hs_splits);
      break;
    default: buf[0] = 0; break;
  }
  return std::string(buf);
}
}  // namespace

bool tick_dependent(const ModelDev& m, int points) {
  return m.family != 2 || m.tc || logreg_fp32_dependent(m.n, points);
}

// The horseshoe's tile height and row ranges: by rule, not by timing, as both set the order of FP32 sums and a choice
// made by a few launches' times made a model's results differ between processes.  Measured (us a potential, 300
// shapes of 50 to 2,000 rows, 20 to 1,000 features, 1 to 256 points): 64 rows for large problems take 80.0 against 82.0
// at 2000 x 1000 x 256 and 49.2 against 51.2 at 2000 x 500 x 256, at most 2 us either way below; the rule is 3.5 % from
// the best of all on average, at most 2 us on small problems: 8 ranges are better than 4 from 129 rows on for few points (200 x 50: 22.6
// against 24.6) and worse for 256 (25.6 against 24.6).
void rule_shapes(ModelDev& m, int points) {
  if (m.family != 3) return;
  m.tune.hs_tm = points >= 128 && m.n * m.p >= 1000000 ? 4 : 2;
  m.tune.hs_splits = m.n <= 64 ? 2 : (m.n <= 200 ? 4 : 8);
}

cudaError_t autotune_potential(ModelDev& m, const float* Q, int npts, double* PE, float* G, cudaStream_t st,
                               std::string* report) {
  int dev = 0;
  cudaGetDevice(&dev);
  char key[192];
  snprintf(key, sizeof(key), "%d|%d|%lld|%d|%d|%d|%d|%d|%g", dev, m.family, (long long)m.n, m.p, m.D, m.num_models,
           npts, m.precision, m.hyper[0]);
  std::lock_guard<std::mutex> lock(g_tune_mu);
  cudaError_t e = ensure_potential_scratch(m, npts);
  if (e != cudaSuccess) return e;
  const char* forced = getenv("GBN_TUNE");  // "hier_cpb=16 hs_tm=2 hs_splits=8 lr_rg=32": fixed shapes
  if (forced && forced[0]) {
    int v = 0;
    const char* p;
    if ((p = strstr(forced, "hier_cpb=")) && sscanf(p + 9, "%d", &v) == 1 && (v == 4 || v == 8 || v == 16))
      m.tune.hier_cpb = v;
    if ((p = strstr(forced, "hs_tm=")) && sscanf(p + 6, "%d", &v) == 1 && (v == 2 || v == 4)) m.tune.hs_tm = v;
    if ((p = strstr(forced, "hs_splits=")) && sscanf(p + 10, "%d", &v) == 1 && v >= 1 && v <= HS_MAX_SPLITS)
      m.tune.hs_splits = v;
    if ((p = strstr(forced, "lr_rg=")) && sscanf(p + 6, "%d", &v) == 1 && v >= 1 && v <= m.row_groups_cap)
      m.tune.lr_rg = v;
  } else if (m.family == 1) {
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      m.tune = it->second;
    } else {
      float best = 1e30f;
      TuneParams pick = m.tune;
      for (int cpb : {4, 8, 16}) {
        m.tune.hier_cpb = cpb;
        float ms = 0.0f;
        e = time_potential(m, Q, npts, PE, G, st, 3, &ms);
        if (e != cudaSuccess) return e;
        if (ms < best) {
          best = ms;
          pick = m.tune;
        }
      }
      m.tune = pick;
      g_tune_cache[key] = pick;
    }
  }
  if (report) *report = tune_report(m);
  return cudaSuccess;
}

// ============================================================ special-function throughput
// Peak rate of the special-function unit for the operations of the tensor-core logistic epilogue
// (ex2.approx, tanh.approx, rcp.approx, lg2.approx), measured with independent dependency chains
// (8 per thread) so the unit, not latency, sets the rate.  MIX issues them in the epilogue's
// proportion: per 16 logits 16 ex2, 8 tanh, 1 rcp and 2 lg2 (1.6875 per logit).
template <int MODE>
__global__ void __launch_bounds__(256) sfu_rate_kernel(int iters, float* __restrict__ out) {
  float v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = 0.25f + 0.01f * (float)(k + (threadIdx.x & 7));
  for (int i = 0; i < iters; ++i) {
    if (MODE == 2) {
#pragma unroll
      for (int k = 0; k < 16; ++k) asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(v[k & 7]) : "f"(-v[k & 7]));
#pragma unroll
      for (int k = 0; k < 8; ++k) asm volatile("tanh.approx.f32 %0, %1;" : "=f"(v[k]) : "f"(v[k]));
      asm volatile("rcp.approx.ftz.f32 %0, %1;" : "=f"(v[0]) : "f"(1.0f + v[0]));
      asm volatile("lg2.approx.ftz.f32 %0, %1;" : "=f"(v[1]) : "f"(1.5f + v[1]));
      asm volatile("lg2.approx.ftz.f32 %0, %1;" : "=f"(v[2]) : "f"(1.5f + v[2]));
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (MODE == 0)
          asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(v[k]) : "f"(-v[k]));
        else
          asm volatile("tanh.approx.f32 %0, %1;" : "=f"(v[k]) : "f"(v[k]));
      }
    }
  }
  float acc = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) acc += v[k];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = acc;  // every chain's result is stored
}

cudaError_t measure_sfu_rate(int mode, cudaStream_t st, double* ops_per_s) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t a = nullptr, b = nullptr;
  float* out = nullptr;  // one float per thread: the chains' results, so none is dead code
  e = cudaMalloc(&out, sizeof(float) * (size_t)blocks * threads);
  if (e == cudaSuccess) e = cudaEventCreate(&a);
  if (e == cudaSuccess) e = cudaEventCreate(&b);
  auto launch = [&]() {
    if (mode == 0) sfu_rate_kernel<0><<<blocks, threads, 0, st>>>(iters, out);
    else if (mode == 1) sfu_rate_kernel<1><<<blocks, threads, 0, st>>>(iters, out);
    else sfu_rate_kernel<2><<<blocks, threads, 0, st>>>(iters, out);
  };
  if (e == cudaSuccess) {
    launch();  // warm-up
    e = cudaEventRecord(a, st);
  }
  const int reps = 5;
  for (int r = 0; r < reps && e == cudaSuccess; ++r) launch();
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaEventRecord(b, st);
  if (e == cudaSuccess) e = cudaEventSynchronize(b);
  float ms = 0.0f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
  // operations per launch: per thread and iteration 8 (one per chain), or the mix's 27
  const double per_thread = (mode == 2 ? 27.0 : 8.0) * iters;
  if (e == cudaSuccess) *ops_per_s = per_thread * blocks * threads * reps / (ms * 1e-3);
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  if (out) cudaFree(out);
  return e;
}

cudaError_t launch_scale_rows(const double* cot, float* G, int npts, int D, cudaStream_t st) {
  size_t total = (size_t)npts * D;
  int blocks = (int)((total + 255) / 256);
  if (blocks > 4096) blocks = 4096;
  if (blocks < 1) blocks = 1;
  scale_rows_kernel<<<blocks, 256, 0, st>>>(cot, G, npts, D);
  return cudaGetLastError();
}

}  // namespace gbn

namespace gbn {
// FP32 logistic potential with scratch supplied by the caller (no allocation):
// part_g needs row_groups * npts * 64 floats, part_ll row_groups * npts doubles.
cudaError_t launch_logreg_simt_scratch(const float* x, const float* y, int64_t n, int p, double prior_scale,
                                       const float* Q, int npts, int row_groups, float* part_g, double* part_ll,
                                       double* PE, float* G, cudaStream_t st) {
  return launch_logreg_fp32(logreg_fp32_shape(n, npts, row_groups).variant, x, y, n, p, prior_scale, Q, npts, p,
                            logreg_fp32_row_groups(n, p, npts, row_groups), part_g, part_ll, PE, G, nullptr, st, false);
}

void horseshoe_finish_launch(const float* Q, int npts, int ld, int P, int64_t N, const float* part_gb, int splits,
                             int ldg, const double* part_rr, int ld_rr, int mtiles, int noncentred, double* PE,
                             float* G, const int32_t* pending, cudaStream_t st) {
  horseshoe_finish_kernel<<<npts, 256, 0, st>>>(Q, npts, ld, P, N, part_gb, splits, ldg, part_rr, ld_rr, mtiles,
                                                noncentred, PE, G, pending);
}

void logreg_finish_launch(const float* Q, int npts, int ld, int p, int row_groups, const float* part_g,
                          const double* part_ll, const double* lin, double prior_scale, double* PE, float* G,
                          const int32_t* pending, cudaStream_t st, const int32_t* split3, bool e_tanh) {
  float ivf;
  double pec;
  logreg_prior_consts(prior_scale, p, &ivf, &pec);
  logreg_finish_kernel<<<(npts + 7) / 8, 256, 0, st>>>(Q, npts, ld, p, row_groups, part_g, part_ll, lin, ivf, pec, PE,
                                                       G, pending, split3, e_tanh);
}
}  // namespace gbn
