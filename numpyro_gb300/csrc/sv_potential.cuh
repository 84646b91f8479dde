// sv_potential.cuh -- CTA-level potentials + adjoints of the stochastic-volatility
// family, shared by the tick-engine kernel (potentials_simt.cu) and the
// persistent engine (nuts_engine.cu) so that both produce bit-identical results.
//
//   s ~ Exponential(s_rate); nu ~ Exponential(nu_rate)        (Exp transforms, log-dets ls, lnu)
//   centred:      h ~ GaussianRandomWalk(scale=s, num_steps=T), z = [h(T), lnu, ls]
//   non-centred:  h_base ~ Normal(0, 1)^T, h = s * cumsum(h_base), z = [h_base(T), lnu, ls]
//   r_t ~ StudentT(nu, 0, exp(h_t))
// Log-densities: Exponential numpyro/distributions/continuous.py:715-726, GaussianRandomWalk
// :1104-1112, StudentT :3229-3238, Normal :2975-2989; Exp log-det transforms.py:641-644; model as
// examples/stochastic_volatility.py:58-66.
//
// Non-centred adjoint.  With S_t = sum_{k<=t} h_base_k and a_t = d log p(r_t | h_t) / d h_t,
//   dU/dh_base_k = h_base_k - s * sum_{t>=k} a_t,   dU/dls = -s * sum_t a_t S_t + s_rate * s - 1.
// Each thread owns one contiguous chunk of ceil(T/NT) steps.  The forward pass needs S_t: the
// walk is stored only at chunk starts (one checkpoint per thread, from a block-wide exclusive scan
// of the chunk totals) and recomputed inside the chunk from its checkpoint.  The reverse pass
// needs the suffix sums of a_t: a block-wide reverse exclusive scan of the chunk totals gives each
// thread its starting suffix; a_t itself stays in registers between the passes (or, for chunks
// too long for registers, is parked in the gradient row).  Running sums inside a chunk are compensated FP32
// (two-sum, Knuth TAOCP vol. 2 4.2.2); chunk totals are scanned and reduced as float-float
// pairs.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "common.cuh"

namespace gbn {

constexpr double SV_LOG_2PI = 1.8378770664093453;
constexpr double SV_LOG_PI = 1.1447298858494002;

// Scratch a CTA needs in shared memory for the SV potentials.
template <int NT>
struct SvSmem {
  double red[16];        // Group<256> reductions
  double special[9];     // lgamma(nu/2), lgamma((nu+1)/2), digamma(nu/2), digamma((nu+1)/2),
                         // nu, 1/nu, s, 1/s, log(s_rate) + log(nu_rate)
  float2 warp_tot[2][NT / 32];
};

// The scalar factors of the potential, each group on lane 0 of its own warp so they run side by
// side with the element loop; thread 0 reads them after the reductions' barriers.  The two
// log-gamma values enter U multiplied by T and grow like x log x, so they stay FP64 (in FP32,
// T * lgamma(nu/2) rounds to O(1) at large nu and roughens the energy surface).  The digammas
// enter only through a difference of order 1/nu in the gradient, and the remaining factors need
// no more than FP32 (GB300 issues FP64 at a small fraction of the FP32 rate).
template <int NT>
__device__ __forceinline__ void sv_special_functions(float lnuf, float lsf, double s_rate, double nu_rate, int tid,
                                                     double* special) {
  static_assert(NT >= 256, "needs six warps");
  if ((tid & 31) != 0) return;
  const float nu = expf(lnuf);
  switch (tid >> 5) {
    case 0: special[0] = lgamma(0.5 * (double)nu); break;
    case 1: special[1] = lgamma(0.5 * ((double)nu + 1.0)); break;
    case 2: special[2] = (double)digamma_f(0.5f * nu); break;
    case 3: special[3] = (double)digamma_f(0.5f * (nu + 1.0f)); break;
    case 4: special[4] = (double)nu; special[5] = (double)(1.0f / nu); break;
    case 5: {
      const float s = expf(lsf);
      special[6] = (double)s;
      special[7] = (double)(1.0f / s);
      special[8] = (double)(logf((float)s_rate) + logf((float)nu_rate));
      break;
    }
    default: break;
  }
}

// d/dlnu of U (both parameterisations): nu-dependent StudentT terms summed over T plus the prior.
__device__ __forceinline__ float sv_grad_lnu(double S_l1p, double S_frac, double T, double nu_rate,
                                             const double* special) {
  const double nu = special[4], inv_nu = special[5];
  double dnu = -0.5 * S_l1p + 0.5 * (nu + 1.0) * inv_nu * S_frac - 0.5 * T * inv_nu - 0.5 * T * special[2] +
               0.5 * T * special[3] - nu_rate;
  return (float)(-(dnu * nu + 1.0));
}

// One step of the centred walk: accumulates the sums and returns dU/dh_t.
__device__ __forceinline__ float sv_centred_step(int t, int T, float h, float hp, float hn, float rt, float nuf,
                                                 float inv_nuf, float inv_s2, Comp32& sdd, Comp32& sl1p,
                                                 Comp32& sfrac, Comp32& sh) {
  const float dprev = (t == 0) ? h : h - hp;
  const float dnext = (t + 1 < T) ? hn - h : 0.0f;
  const float yv = rt * expf(-h);
  const float y2 = yv * yv;
  const float q = y2 * inv_nuf;
  const float frac = __fdividef(y2, nuf + y2);
  sdd.add_fused(dprev, dprev);
  sl1p.add(log1pf(q));
  sfrac.add(frac);
  sh.add(h);
  return (dprev - dnext) * inv_s2 + 1.0f - (nuf + 1.0f) * frac;
}

// One step of the non-centred walk: extends it by e, accumulates, returns a_t = d log p(r_t | h_t) / d h_t.
// in = false (with e = 0 and rt = 0): a step past the chunk, which adds zeros.
struct SvNcSums {
  Comp32 l1p, frac, h, as, e2, atot;
};
__device__ __forceinline__ float sv_nc_step(Comp32& S, float e, float rt, float sf, float nuf, float inv_nuf,
                                            SvNcSums& a, bool in = true) {
  S.add(e);
  const float St = S.value();
  const float h = in ? __fmul_rn(sf, St) : 0.0f;
  const float yv = rt * expf(-h);
  const float y2 = yv * yv;
  const float frac = __fdividef(y2, nuf + y2);
  const float at = in ? (nuf + 1.0f) * frac - 1.0f : 0.0f;
  a.l1p.add(log1pf(y2 * inv_nuf));
  a.frac.add(frac);
  a.h.add(h);
  a.as.add_fused(at, in ? St : 0.0f);
  a.e2.add_fused(e, e);
  a.atot.add(at);
  return at;
}

// -U and dU/d log s from the sums; log_rates = log(s_rate) + log(nu_rate), lg0/lg1 = lgamma(nu / 2), lgamma((nu + 1) / 2)
__device__ __forceinline__ double sv_log_joint(bool noncentred, double S_walk, double S_l1p, double S_h, double T,
                                               double lnu, double ls, double nu, double s, double inv_s,
                                               double log_rates, double s_rate, double nu_rate, double lg0, double lg1) {
  double lp = log_rates - s_rate * s + ls - nu_rate * nu + lnu;
  if (noncentred)
    lp += -0.5 * S_walk - 0.5 * T * SV_LOG_2PI;
  else
    lp += -0.5 * S_walk * (inv_s * inv_s) - T * ls - 0.5 * T * SV_LOG_2PI;
  const double zc = 0.5 * lnu + 0.5 * SV_LOG_PI + lg0 - lg1;
  return lp + (-0.5 * (nu + 1.0) * S_l1p - S_h - T * zc);
}
__device__ __forceinline__ float sv_grad_ls(bool noncentred, double S_dd_or_as, double T, double s, double inv_s,
                                            double s_rate) {
  if (noncentred) return (float)(-s * S_dd_or_as + s_rate * s - 1.0);
  const double ds = S_dd_or_as * (inv_s * inv_s * inv_s) - T * inv_s - s_rate;
  return (float)(-(ds * s + 1.0));
}

// The potentials are compiled out of line: the tick and persistent kernels then run one and
// the same instruction sequence (inlined into different kernels, floating-point contraction
// could differ between them and break their bit-identity).
// Centred GRW.  z/g are the chain's rows; pe_out is written by thread 0.
template <int NT>
__device__ __noinline__ void sv_potential_block(const float* z, float* g, double* pe_out, int T,
                                                   const float* __restrict__ ret, double s_rate, double nu_rate,
                                                   int tid, SvSmem<NT>& sm) {
  Group<NT> grp{tid};
  // FP32 nu and 1/s^2 for the element loop; FP64 nu and s only where the scalar terms need them
  const float lnuf = z[T], lsf = z[T + 1];
  const float nuf = expf(lnuf), sf = expf(lsf);
  const float inv_s2 = 1.0f / (sf * sf), inv_nuf = 1.0f / nuf;
  sv_special_functions<NT>(lnuf, lsf, s_rate, nu_rate, tid, sm.special);
  Comp32 sdd{0.0f, 0.0f}, sl1p{0.0f, 0.0f}, sfrac{0.0f, 0.0f}, sh{0.0f, 0.0f};
  constexpr int U = 4;  // loads of U steps are issued before their gradient stores
  for (int t0 = tid; t0 < T; t0 += U * NT) {
    float hv[U], hp[U], hn[U], rv[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int t = t0 + k * NT;
      const bool in = t < T;
      hv[k] = in ? z[t] : 0.0f;
      hp[k] = (in && t > 0) ? z[t - 1] : 0.0f;
      hn[k] = (t + 1 < T) ? z[t + 1] : 0.0f;
      rv[k] = in ? ret[t] : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int t = t0 + k * NT;
      if (t >= T) continue;
      g[t] = sv_centred_step(t, T, hv[k], hp[k], hn[k], rv[k], nuf, inv_nuf, inv_s2, sdd, sl1p, sfrac, sh);
    }
  }
  FF f_dd = comp_ff(sdd), f_l1p = comp_ff(sl1p), f_frac = comp_ff(sfrac), f_h = comp_ff(sh);
  grp.sum2ff(f_dd, f_l1p, sm.red);
  grp.sum2ff(f_frac, f_h, sm.red);
  if (tid == 0) {
    const double s = sm.special[6], inv_s = sm.special[7], S_dd = ff_value(f_dd), S_l1p = ff_value(f_l1p);
    *pe_out = -sv_log_joint(false, S_dd, S_l1p, ff_value(f_h), (double)T, lnuf, lsf, sm.special[4], s, inv_s,
                            sm.special[8], s_rate, nu_rate, sm.special[0], sm.special[1]);
    g[T] = sv_grad_lnu(S_l1p, ff_value(f_frac), (double)T, nu_rate, sm.special);
    g[T + 1] = sv_grad_ls(false, S_dd, (double)T, s, inv_s, s_rate);
  }
}

// Block-wide exclusive scans of one float-float pair per thread (forward: sum over lower
// threads; reverse: sum over higher threads).  Lanes combine by shuffles, warps through `wt`
// (NT/32 pairs); each contains two barriers.
template <int NT>
__device__ __forceinline__ FF block_excl_scan(FF v, int tid, float2* wt) {
  const int lane = tid & 31, w = tid >> 5;
  FF excl{0.0f, 0.0f};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {  // inclusive lane scan of v, then shift by one lane
    FF x{__shfl_up_sync(0xffffffffu, v.hi, o), __shfl_up_sync(0xffffffffu, v.lo, o)};
    if (lane >= o) v = ff_add(x, v);
  }
  excl.hi = __shfl_up_sync(0xffffffffu, v.hi, 1);
  excl.lo = __shfl_up_sync(0xffffffffu, v.lo, 1);
  if (lane == 0) excl = FF{0.0f, 0.0f};
  if (lane == 31) wt[w] = make_float2(v.hi, v.lo);
  __syncthreads();
  FF off{0.0f, 0.0f};
  for (int k = 0; k < w; ++k) off = ff_add(off, FF{wt[k].x, wt[k].y});
  __syncthreads();
  return ff_add(off, excl);
}
template <int NT>
__device__ __forceinline__ FF block_excl_rscan(FF v, int tid, float2* wt) {
  const int lane = tid & 31, w = tid >> 5;
  FF excl{0.0f, 0.0f};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    FF x{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)};
    if (lane + o < 32) v = ff_add(v, x);
  }
  excl.hi = __shfl_down_sync(0xffffffffu, v.hi, 1);
  excl.lo = __shfl_down_sync(0xffffffffu, v.lo, 1);
  if (lane == 31) excl = FF{0.0f, 0.0f};
  if (lane == 0) wt[w] = make_float2(v.hi, v.lo);
  __syncthreads();
  FF off{0.0f, 0.0f};
  for (int k = NT / 32 - 1; k > w; --k) off = ff_add(off, FF{wt[k].x, wt[k].y});
  __syncthreads();
  return ff_add(off, excl);
}

// Non-centred GRW (h = s * cumsum(h_base)).  z/g are the chain's rows.  Chunks of at most
// SV_REG_CHUNK steps (T <= 4096 with 256 threads) are held in registers.
constexpr int SV_REG_CHUNK = 16;
// B: steps of a long walk whose loads are issued before their arithmetic.  One at a time, the potential kernel waits a
// memory latency a step: 8 take 20,000 steps x 1,024 points from 819 to 302 us and 4,097 x 256 from 25 to 21 us.  The
// engine, with fewer chains on an SM, keeps 1: with 8 it is 5 % slower at 4,350 steps where chains share SMs.
template <int NT, int B = 1>
__device__ __noinline__ void sv_nc_potential_block(const float* z, float* g, double* pe_out, int T,
                                                      const float* __restrict__ ret, double s_rate,
                                                      double nu_rate, int tid, SvSmem<NT>& sm) {
  Group<NT> grp{tid};
  const float lnuf = z[T], lsf = z[T + 1];
  const float nuf = expf(lnuf), sf = expf(lsf), inv_nuf = 1.0f / nuf;
  sv_special_functions<NT>(lnuf, lsf, s_rate, nu_rate, tid, sm.special);
  const int chunk = (T + NT - 1) / NT;
  const int t0 = min(T, tid * chunk), t1 = min(T, t0 + chunk);
  SvNcSums a{};
  // one step of the forward pass: extend the walk, accumulate, return a_t
  auto forward_step = [&](Comp32& S, float e, float r) -> float { return sv_nc_step(S, e, r, sf, nuf, inv_nuf, a); };
  if (chunk <= SV_REG_CHUNK) {
    // the chunk's h_base, returns and a_t stay in registers between the passes
    float ev[SV_REG_CHUNK], rv[SV_REG_CHUNK], av[SV_REG_CHUNK];
#pragma unroll
    for (int i = 0; i < SV_REG_CHUNK; ++i) {
      const bool in = t0 + i < t1;
      ev[i] = in ? z[t0 + i] : 0.0f;
      rv[i] = in ? ret[t0 + i] : 0.0f;
    }
    // chunk total of h_base -> checkpoint S_{t0-1} (exclusive scan)
    Comp32 tot{0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < SV_REG_CHUNK; ++i)
      if (t0 + i < t1) tot.add(ev[i]);
    const FF ck = block_excl_scan<NT>(comp_ff(tot), tid, sm.warp_tot[0]);
    Comp32 S{ck.hi, ck.lo};
#pragma unroll
    for (int i = 0; i < SV_REG_CHUNK; ++i) av[i] = (t0 + i < t1) ? forward_step(S, ev[i], rv[i]) : 0.0f;
    // reverse pass: suffix sums of a_t from the thread's starting suffix
    const FF suf = block_excl_rscan<NT>(comp_ff(a.atot), tid, sm.warp_tot[1]);
    Comp32 A{suf.hi, suf.lo};
#pragma unroll
    for (int i = SV_REG_CHUNK - 1; i >= 0; --i) {
      if (t0 + i >= t1) continue;
      A.add(av[i]);
      g[t0 + i] = ev[i] - sf * A.value();
    }
  } else {
    // long walks: a_t is parked in the gradient row between the passes
    Comp32 tot{0.0f, 0.0f};
    for (int tb = t0; tb < t1; tb += B) {
      float e[B];
#pragma unroll
      for (int i = 0; i < B; ++i) e[i] = tb + i < t1 ? z[tb + i] : 0.0f;
#pragma unroll
      for (int i = 0; i < B; ++i) tot.add(e[i]);  // adding 0 changes nothing
    }
    const FF ck = block_excl_scan<NT>(comp_ff(tot), tid, sm.warp_tot[0]);
    Comp32 S{ck.hi, ck.lo};
    for (int tb = t0; tb < t1; tb += B) {
      float e[B], r[B];
#pragma unroll
      for (int i = 0; i < B; ++i) {
        e[i] = tb + i < t1 ? z[tb + i] : 0.0f;
        r[i] = tb + i < t1 ? ret[tb + i] : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < B; ++i)
        if (tb + i < t1) g[tb + i] = forward_step(S, e[i], r[i]);
    }
    const FF suf = block_excl_rscan<NT>(comp_ff(a.atot), tid, sm.warp_tot[1]);
    Comp32 A{suf.hi, suf.lo};
    for (int tb = t1 - 1; tb >= t0; tb -= B) {
      float e[B], at[B];
#pragma unroll
      for (int i = 0; i < B; ++i) {
        e[i] = tb - i >= t0 ? z[tb - i] : 0.0f;
        at[i] = tb - i >= t0 ? g[tb - i] : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < B; ++i)
        if (tb - i >= t0) {
          A.add(at[i]);
          g[tb - i] = e[i] - sf * A.value();
        }
    }
  }
  FF f_l1p = comp_ff(a.l1p), f_frac = comp_ff(a.frac), f_h = comp_ff(a.h), f_as = comp_ff(a.as);
  grp.sum2ff(f_l1p, f_frac, sm.red);
  grp.sum2ff(f_h, f_as, sm.red);
  const FF f_e2 = grp.sumff(comp_ff(a.e2), sm.red);
  if (tid == 0) {
    const double s = sm.special[6], S_l1p = ff_value(f_l1p);
    *pe_out = -sv_log_joint(true, ff_value(f_e2), S_l1p, ff_value(f_h), (double)T, lnuf, lsf, sm.special[4], s, 0.0,
                            sm.special[8], s_rate, nu_rate, sm.special[0], sm.special[1]);
    g[T] = sv_grad_lnu(S_l1p, ff_value(f_frac), (double)T, nu_rate, sm.special);
    g[T + 1] = sv_grad_ls(true, ff_value(f_as), (double)T, s, 0.0, s_rate);
  }
}

// ------------------------------------------------ eight element warps beside scalar warps
// Pieces of the register engine (sv_engine.cuh) and of sv_potential_kernel: element thread i of 256, rows in shared
// memory with one word more every 16, so that the non-centred walk's chunk order meets few bank conflicts.
__device__ __forceinline__ int sv_pos(int d) { return d + (d >> 4); }

// folds the eight warp sums of row i, as Group<256>::sumff
__device__ __forceinline__ FF sv_fold(const float2 (*r)[8], int i) {
  FF t{r[i][0].x, r[i][0].y};
#pragma unroll
  for (int w = 1; w < 8; ++w) t = ff_add(t, FF{r[i][w].x, r[i][w].y});
  return t;
}

// block_excl_scan and block_excl_rscan over eight element warps (named barrier 2), one barrier each.
__device__ __forceinline__ FF sv_excl_scan(FF v, int lane, int warp, float2* wt) {
  FF excl{0.0f, 0.0f};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    FF x{__shfl_up_sync(0xffffffffu, v.hi, o), __shfl_up_sync(0xffffffffu, v.lo, o)};
    if (lane >= o) v = ff_add(x, v);
  }
  excl.hi = __shfl_up_sync(0xffffffffu, v.hi, 1);
  excl.lo = __shfl_up_sync(0xffffffffu, v.lo, 1);
  if (lane == 0) excl = FF{0.0f, 0.0f};
  if (lane == 31) wt[warp] = make_float2(v.hi, v.lo);
  asm volatile("bar.sync 2, 256;" ::: "memory");
  FF off{0.0f, 0.0f};
  for (int k = 0; k < warp; ++k) off = ff_add(off, FF{wt[k].x, wt[k].y});
  return ff_add(off, excl);
}
__device__ __forceinline__ FF sv_excl_rscan(FF v, int lane, int warp, float2* wt) {
  FF excl{0.0f, 0.0f};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    FF x{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)};
    if (lane + o < 32) v = ff_add(v, x);
  }
  excl.hi = __shfl_down_sync(0xffffffffu, v.hi, 1);
  excl.lo = __shfl_down_sync(0xffffffffu, v.lo, 1);
  if (lane == 31) excl = FF{0.0f, 0.0f};
  if (lane == 0) wt[warp] = make_float2(v.hi, v.lo);
  asm volatile("bar.sync 2, 256;" ::: "memory");
  FF off{0.0f, 0.0f};
  for (int k = 7; k > warp; --k) off = ff_add(off, FF{wt[k].x, wt[k].y});
  return ff_add(off, excl);
}

// The non-centred walk's elements: gradients to gs (may be rets: a thread reads its chunk before it writes it), warp
// sums of l1p, frac, h, a S and h_base^2 to r1.  K: steps a thread at most.  Steps past the chunk count as
// zeros (adding 0 to a compensated sum changes nothing), so that the steps' long operations overlap.
template <int K>
__device__ __forceinline__ void sv_nc_elements(const float* zs, const float* rets, float* gs, int T, int tid, float sf,
                                               float nuf, float inv_nuf, float2 (*r1)[8], float2 (*wt)[8]) {
  const int lane = tid & 31, warp = tid >> 5;
  const int chunk = (T + 255) / 256;
  const int t0 = min(T, tid * chunk), t1 = min(T, t0 + chunk);
  SvNcSums s{};
  float av[K];
  auto ev = [&](int i) -> float { return (t0 + i < t1) ? zs[sv_pos(t0 + i)] : 0.0f; };
  Comp32 tot{0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < K; ++i) tot.add(ev(i));
  const FF ck = sv_excl_scan(comp_ff(tot), lane, warp, wt[0]);
  Comp32 S{ck.hi, ck.lo};
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const bool in = t0 + i < t1;
    av[i] = sv_nc_step(S, ev(i), in ? rets[sv_pos(t0 + i)] : 0.0f, sf, nuf, inv_nuf, s, in);
  }
  const FF suf = sv_excl_rscan(comp_ff(s.atot), lane, warp, wt[1]);
  Comp32 A{suf.hi, suf.lo};
#pragma unroll
  for (int i = K - 1; i >= 0; --i) {
    A.add(av[i]);
    if (t0 + i < t1) gs[sv_pos(t0 + i)] = ev(i) - sf * A.value();
  }
  const FF v = warp_sum4ff(comp_ff(s.l1p), comp_ff(s.frac), comp_ff(s.h), comp_ff(s.as), lane);
  if ((lane & 7) == 0) r1[lane >> 3][warp] = make_float2(v.hi, v.lo);
  FF e2 = comp_ff(s.e2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e2 = ff_add(e2, ff_shfl_xor(e2, o));
  if (lane == 0) r1[4][warp] = make_float2(e2.hi, e2.lo);
}

}  // namespace gbn
