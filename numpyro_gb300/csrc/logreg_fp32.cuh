// logreg_fp32.cuh -- FP32 CUDA-core kernel of the logistic-regression potential.
//
//   l = X b;  U = sum_n [softplus(l_n) - y_n l_n] + prior;  dU/db = X^T (sigmoid(l) - y) + prior
// Fused per row tile: logits -> (softplus, sigmoid) -> gradient, so no logit reaches memory.  A CTA
// owns CT chains and a strided set of 64-row tiles; a thread holds 4 rows x 4 CG chains of logits.
//
// Bound: FP32 instruction issue.  A logit costs 2 p fused multiply-adds and ~60 instructions of expf, log1pf
// and reciprocal (~100 with the compiler's division: 1 + e^-|l| lies in [1, 2], so the reciprocal needs no
// range handling, recip_1_2).  The multiply-adds run as FP32x2 over pairs of chains: no more per cycle than
// scalar ones, but half the issue slots, which the epilogues of the other warps use.  Operands come from
// shared memory as 16-byte words; X tiles arrive by cp.async one tile ahead, rows swizzled by groups of
// four so that the eight lanes of a load phase meet eight bank groups.
// Measured at 581,012 x 55 x 1,024 chains: 5.52 ms (64 x 64 tile, 4 x 4 a thread, X through registers and a
// transposed copy) -> 3.65 ms = 36 TFLOP/s.  8 x 8 logits a thread with 8 warps per SM: 3.85; scalar
// multiply-adds: 3.86.
// Sums: a chain's log-likelihood of four consecutive rows in FP32, then FP64 over the thread's rows, across threads
// and across CTAs.  (Compensated FP32 pairs within a CTA leave the potential 2^-48 off instead of 2^-53 and are
// 3 % faster at 5 features, 1.72 against 1.78 ms at 581,012 x 1,024; at 55 features both take 3.68.)
#pragma once
#include <algorithm>
#include <climits>

#include "common.cuh"
#include "internal.h"

namespace gbn {

// 1 / d for d in [1, 2], rounded to nearest: one Newton-Raphson step on the approximate reciprocal with
// the residual exact in a fused multiply-add (Markstein, IBM J. Res. Dev. 34, 1990).  Equal to 1.0f / d
// for each of the 2^23 + 1 floats of the range (tests/test_gpu_reciprocal.py compares them all).
__device__ __forceinline__ float recip_1_2(float d) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return fmaf(y, fmaf(-d, y, 1.0f), y);
}

struct LogregArgs {
  const float* x;  // [n][p]
  const float* y;
  int64_t n;
  int p;
  const float* q;  // [npts][ld]
  int npts, ld;
  float* part_g;    // [gridDim.y][npts][64]
  double* part_ll;  // [gridDim.y][npts]
  const int32_t* pending;
};

__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 16 : 0)
               : "memory");
}

// CT chains, NTH threads, 4 rows x 4 CG chains a thread in the logit phase, 4 CG chains x 4 features a thread in the
// gradient phase, SP floats a row of the X tile (32 or 64), two tile buffers.
template <int CT, int NTH, int CG, int SP>
struct LogregTile {
  static constexpr int TX = CT / (4 * CG), TY = NTH / TX, RT = 4 * TY;
  static constexpr size_t bytes(int dp) {
    return sizeof(float) * (size_t)(2 * RT * SP + dp * CT + RT * CT + 2 * RT) + sizeof(double) * (NTH / 32) * CT;
  }
};

template <int CT, int NTH, int CG, int SP, int MINB>
__global__ void __launch_bounds__(NTH, MINB) logreg_fp32_kernel(const LogregArgs A) {
  using T = LogregTile<CT, NTH, CG, SP>;
  constexpr int TX = T::TX, RT = T::RT;
  extern __shared__ __align__(16) float lr_smem[];
  const int p = A.p, nc = (p + 3) >> 2;
  float* const xs = lr_smem;                 // [2][RT][SP], chunk c of row r at c ^ ((r >> 2) & 7)
  float* const es = xs + 2 * RT * SP;        // [RT][CT]
  float* const ys = es + RT * CT;            // [2][RT]
  double* const lls = reinterpret_cast<double*>(ys + 2 * RT);  // [NTH / 32][CT]
  float* const bs = reinterpret_cast<float*>(lls + (NTH / 32) * CT);  // [4 nc][CT]
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int c0 = blockIdx.x * CT, rg = blockIdx.y, groups = gridDim.y;
  const int64_t ntiles = (A.n + RT - 1) / RT;

  for (int k = tid; k < 2 * RT * SP; k += NTH) xs[k] = 0.0f;  // features past p stay zero
  __syncthreads();
  auto load_tile = [&](int64_t tile, int buf) {
    float* const dst = xs + buf * RT * SP;
    const int64_t r0 = tile * RT;
    const float* const src = A.x + r0 * p;
    const int64_t left = A.n - r0;
    if ((p & 3) == 0 && (reinterpret_cast<uintptr_t>(A.x) & 15) == 0) {
      const int q4 = p >> 2;
      for (int k = tid; k < RT * q4; k += NTH) {
        const int r = k / q4, c = k - r * q4;
        const bool in = r < left;
        cp_async16(dst + r * SP + ((c ^ ((r >> 2) & 7)) << 2), in ? src + (size_t)r * p + 4 * c : A.x, in);
      }
    } else {
      int r = tid / p, d = tid - r * p;
      const int sr = NTH / p, sd = NTH - sr * p;
      for (int k = tid; k < RT * p; k += NTH) {
        const bool in = r < left;
        cp_async4(dst + r * SP + (((d >> 2) ^ ((r >> 2) & 7)) << 2) + (d & 3), in ? src + k : A.x, in);
        r += sr;
        d += sd;
        if (d >= p) {
          d -= p;
          ++r;
        }
      }
    }
    for (int r = tid; r < RT; r += NTH) cp_async4(ys + buf * RT + r, r < left ? A.y + r0 + r : A.y, r < left);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // Gradient phase: a thread owns 4 CG chains x 4 features and takes the rows in order, so the sum of
  // an output does not depend on the tile's shape (only on which 64-row tiles a row group holds).
  const int outs = TX * nc;
  const int gc = tid % TX, gd = tid / TX;
  static_assert(TX * (SP / 4) <= NTH, "an output tile per thread");
  float2 gacc[2 * CG][4];  // pairs of chains
#pragma unroll
  for (int i = 0; i < 2 * CG; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) gacc[i][j] = make_float2(0.0f, 0.0f);
  double ll[4 * CG];
#pragma unroll
  for (int j = 0; j < 4 * CG; ++j) ll[j] = 0.0;

  int buf = 0;
  if (rg < ntiles) load_tile(rg, 0);
  tick_wait();  // the data is on its way; the positions are the previous kernel's
  tick_trigger();
  if (A.pending && *A.pending == 0) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  for (int k = tid; k < 4 * nc * CT; k += NTH) {
    const int c = k / (4 * nc), d = k % (4 * nc);
    bs[d * CT + c] = (d < p && c0 + c < A.npts) ? A.q[(size_t)(c0 + c) * A.ld + d] : 0.0f;
  }
  for (int64_t tile = rg; tile < ntiles; tile += groups, buf ^= 1) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // this tile has landed; every thread is done with the other buffer and with E
    if (tile + groups < ntiles) load_tile(tile + groups, buf ^ 1);
    const float* const xb = xs + buf * RT * SP;
    // ------------------------------------------------ logits
    float2 acc[4][2 * CG];  // pairs of chains
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2 * CG; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    for (int c = 0; c < nc; ++c) {
      float4 xv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        xv[i] = *reinterpret_cast<const float4*>(xb + (4 * ty + i) * SP + ((c ^ (ty & 7)) << 2));
#pragma unroll
      for (int dd = 0; dd < 4; ++dd) {
        float2 b[2 * CG];
#pragma unroll
        for (int h = 0; h < CG; ++h) {
          const float4 b4 = *reinterpret_cast<const float4*>(bs + (4 * c + dd) * CT + h * (CT / CG) + 4 * tx);
          b[2 * h] = make_float2(b4.x, b4.y);
          b[2 * h + 1] = make_float2(b4.z, b4.w);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float xa = dd == 0 ? xv[i].x : (dd == 1 ? xv[i].y : (dd == 2 ? xv[i].z : xv[i].w));
#pragma unroll
          for (int j = 0; j < 2 * CG; ++j) acc[i][j] = __ffma2_rn(make_float2(xa, xa), b[j], acc[i][j]);
        }
      }
    }
    // ------------------------------------------------ softplus and sigmoid
    const int64_t left = A.n - tile * RT;
    float llt[4 * CG];
#pragma unroll
    for (int j = 0; j < 4 * CG; ++j) llt[j] = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 4 * ty + i;
      const float yy = ys[buf * RT + r];
      const bool in = r < left;
      float ev[4 * CG];
#pragma unroll
      for (int j = 0; j < 4 * CG; ++j) {
        const float l = (j & 1) ? acc[i][j >> 1].y : acc[i][j >> 1].x;
        const float t = expf(-fabsf(l));
        const float sp = fmaxf(l, 0.0f) + log1pf(t);
        const float inv = recip_1_2(1.0f + t);
        const float sig = (l >= 0.0f) ? inv : t * inv;
        ev[j] = in ? sig - yy : 0.0f;
        llt[j] += in ? sp - yy * l : 0.0f;
      }
#pragma unroll
      for (int h = 0; h < CG; ++h)
        *reinterpret_cast<float4*>(es + r * CT + h * (CT / CG) + 4 * tx) =
            make_float4(ev[4 * h], ev[4 * h + 1], ev[4 * h + 2], ev[4 * h + 3]);
    }
#pragma unroll
    for (int j = 0; j < 4 * CG; ++j)  // few-chain tiles: the first sum is not added to 0
      ll[j] = CT <= 16 && tile == rg ? f2d(llt[j]) : ll[j] + f2d(llt[j]);
    __syncthreads();
    // ------------------------------------------------ gradient
    if (tid < outs) {
#pragma unroll 2
      for (int r = 0; r < RT; ++r) {
        float2 e[2 * CG];
        float xf[4];
#pragma unroll
        for (int h = 0; h < CG; ++h) {
          const float4 e4 = *reinterpret_cast<const float4*>(es + r * CT + h * (CT / CG) + 4 * gc);
          e[2 * h] = make_float2(e4.x, e4.y);
          e[2 * h + 1] = make_float2(e4.z, e4.w);
        }
        const float4 x4 = *reinterpret_cast<const float4*>(xb + r * SP + ((gd ^ ((r >> 2) & 7)) << 2));
        xf[0] = x4.x; xf[1] = x4.y; xf[2] = x4.z; xf[3] = x4.w;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 2 * CG; ++i) gacc[i][j] = __ffma2_rn(e[i], make_float2(xf[j], xf[j]), gacc[i][j]);
      }
    }
  }
  // ------------------------------------------------ the CTA's partials
  if (tid < outs) {
#pragma unroll
    for (int i = 0; i < 4 * CG; ++i) {
      const int c = c0 + (i >> 2) * (CT / CG) + 4 * gc + (i & 3);
      if (c >= A.npts) continue;
      const float2* const v = gacc[i >> 1];
      *reinterpret_cast<float4*>(A.part_g + ((size_t)rg * A.npts + c) * 64 + 4 * gd) =
          (i & 1) ? make_float4(v[0].y, v[1].y, v[2].y, v[3].y) : make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
    }
  }
  // Across the lanes of a warp that share chains.  An SM starts an FP64 instruction every 19 cycles, so the lanes first
  // deal the 4 CG sums out among themselves (lane bit o set: the upper half of those left).
  int left_sums = 4 * CG, first = 0, whole = 0;
#pragma unroll
  for (int o = 16; o >= TX; o >>= 1) {
    if (left_sums > 1) {
      left_sums >>= 1;
      const bool up = (tid & o) != 0;
      if (up) first += left_sums;
#pragma unroll
      for (int j = 0; j < 2 * CG; ++j) {
        if (j >= left_sums) break;
        const double lower = ll[j], upper = ll[j + left_sums];
        ll[j] = (up ? upper : lower) + __shfl_xor_sync(0xffffffffu, up ? lower : upper, o);
      }
    } else {
      ll[0] += __shfl_xor_sync(0xffffffffu, ll[0], o);
      whole |= o;
    }
  }
  if ((tid & whole) == 0) {
#pragma unroll
    for (int k = 0; k < 2 * CG; ++k) {
      if (k >= left_sums) break;
      const int j = first + k;
      lls[(tid >> 5) * CT + (j >> 2) * (CT / CG) + 4 * tx + (j & 3)] = ll[k];
    }
  }
  __syncthreads();
  if (tid < CT && c0 + tid < A.npts) {
    double v = lls[tid];
    for (int w = 1; w < NTH / 32; ++w) v += lls[w * CT + tid];
    A.part_ll[(size_t)rg * A.npts + c0 + tid] = v;
  }
}

// Row tiles of 64 rows: up to this many, for LR_ORDERED_POINTS points at most, every tile is a row group of its
// own and the finish adds them in order, so a small data set's gradient is one fixed sum whatever the launch
// shape.  More points would make the partials large (128 groups x 65,536 points: 2.2 GB) and their sum slow:
// 1,000 rows x 5 features x 65,536 points 492 us, 283 with two groups.
constexpr int LR_ORDERED = 128;
constexpr int LR_ORDERED_POINTS = 1024;

// The sums over row groups and the prior for one chain, a CTA of 256 threads.  By one warp the loads of
// ~150 row groups (a few-chain launch) took 29 us in dependent rounds of eight.  Where CTAs come in waves, or
// a warp has two such rounds, a warp a chain (logreg_finish_kernel, the same order up to LR_ORDERED row groups)
// is better: 200 rows x 16,384 points 76 against 45 us, x 1,024 16.4 against 14.4; 8,192 rows (128 groups) x
// 1,024 points of 55 features 97 against 104.
inline bool logreg_fp32_finish_by_warp(int npts, int groups) { return npts > 1024 || (npts > 512 && groups <= 16); }
__global__ void __launch_bounds__(256) logreg_fp32_finish_kernel(const LogregArgs A, int groups, float inv_var,
                                                                 double pe_const, double* __restrict__ pe,
                                                                 float* __restrict__ g) {
  tick_wait();
  tick_trigger();
  if (A.pending && *A.pending == 0) return;
  __shared__ float4 part[LR_ORDERED][16];
  const int c = blockIdx.x, tid = threadIdx.x, d4 = tid & 15, slice = tid >> 4;
  const float4* const src = reinterpret_cast<const float4*>(A.part_g + (size_t)c * 64) + d4;
  const bool ordered = groups <= LR_ORDERED;
  if (4 * d4 < A.p) {
    if (ordered) {
#pragma unroll 8
      for (int r = slice; r < groups; r += 16) part[r][d4] = src[(size_t)r * A.npts * 16];
    } else {  // 16 slices of the row groups, each in order
      float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
      for (int r = slice; r < groups; r += 16) {
        const float4 v = src[(size_t)r * A.npts * 16];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      part[slice][d4] = s;
    }
  }
  if (tid < 32) {  // potential and prior, in FP64 as logreg_finish_warp
    double lp = 0.0, lsum = 0.0;
    for (int d = tid; d < A.p; d += 32) {
      const double b = (double)A.q[(size_t)c * A.ld + d];
      lp += 0.5 * b * b * (double)inv_var;
    }
    for (int r = tid; r < groups; r += 32) lsum += A.part_ll[(size_t)r * A.npts + c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lp += __shfl_xor_sync(0xffffffffu, lp, o);
      lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    }
    if (tid == 0) pe[c] = lsum + lp + pe_const;
  }
  __syncthreads();
  if (tid >= 64 && tid < 128) {  // not the warp that sums in FP64
    const int d = tid - 64, rows = ordered ? groups : 16;
    if (d < A.p) {
      const float* const col = reinterpret_cast<const float*>(&part[0][0]) + d;
      float t = 0.0f;
#pragma unroll 16
      for (int k = 0; k < rows; ++k) t += col[k * 64];
      g[(size_t)c * A.ld + d] = fmaf(A.q[(size_t)c * A.ld + d], inv_var, t);
    }
  }
}

// ------------------------------------------------------------------ launch shapes
// The widest tile whose CTAs still fill the chip: 128 chains (4 x 8 logits a thread, 256 threads), 64 (4 x 4,
// 256 threads), 16 and, for the few chains of an ordinary run, 8 (a warp); 64 rows each.
constexpr int LR_SMS = 152;
struct LogregShape {
  int variant, ct;
};
// max_groups: row groups that the caller has room for (16 of 20,000 rows x 256 points x 55 features: 183 us with the
// tile of 128 chains, 117 with 64, 99 with 16)
inline LogregShape logreg_fp32_shape(int64_t n, int npts, int max_groups) {
  const int64_t tiles = std::min<int64_t>((n + 63) / 64, max_groups);
  if (npts > 64 && (npts + 127) / 128 * tiles >= 2 * LR_SMS) return {3, 128};
  if (npts > 16 && (npts + 63) / 64 * tiles >= LR_SMS) return {2, 64};
  if (npts > 8) return {1, 16};
  return {0, 8};
}
// Row groups (CTAs of a chain group) by a rule on the sizes, as they set the order of FP32 sums: picked by timing, a
// model's draws differed between processes.  One a tile for small data sets of up to LR_ORDERED_POINTS points, else
// the same number of tiles in every group where that can be, and of the counts that put one CTA on each SM or k = 1
// to 8 on the busiest the largest (with the shortest sums) within 1 % of the least cost:
//   64 and 128 chains   k (tiles of a CTA + 0.4) + 0.006 for each group (the finish).  In the tick loop the CTAs start beside
//                       the state machine's, eight chains each, and go to the other SMs first: as many CTAs as
//                       those have one each, f = 1.3 + 4 / p (1.5 at most) times as slow as two that overlap their
//                       phases; more, up to one an SM, meet on one SM, k = 2 (45,000 rows x 50 features x 100 chains:
//                       141 CTAs beside 13 take 5.8 ms for 60 ticks, 235 4.1; 60,000: 134 4.6, 235 5.1).
//   8 chains            k (tiles + 0.15) (1 + 0.8 / k) + 0.004 a group, k = 4 at least: a CTA is a warp, fewer leave
//                       schedulers idle and more overlap better.  16 chains, and 8 with many features: 4 CTAs an SM.
// Against the best of up to 20 counts a potential alone is 1.1 % slower on average (900 shapes of 8,193 to 581,012
// rows, 5 to 55 features, 1 to 1,024 chains; the best of three timed ones, as before: 1.8 %), a run 0.5 % (520
// shapes of 8,256 to 90,000 rows, 20 to 1,024 chains).  want > 0: at most that many.
inline int logreg_fp32_row_groups(int64_t n, int p, int npts, int want) {
  const int64_t tiles = (n + 63) / 64;
  if (tiles <= LR_ORDERED && want > 0) return (int)std::min<int64_t>(want, tiles);
  if (tiles <= LR_ORDERED && npts <= LR_ORDERED_POINTS) return (int)tiles;
  const LogregShape s = logreg_fp32_shape(n, npts, INT_MAX);
  const int cgroups = (npts + s.ct - 1) / s.ct;
  auto even = [&](int64_t groups) {  // the same number of tiles each
    const int64_t g = std::min<int64_t>(std::max<int64_t>(groups, 1), tiles), per = (tiles + g - 1) / g;
    return (tiles + per - 1) / per;
  };
  if (want > 0) return (int)even(want);
  if (s.variant == 1 || (s.variant == 0 && p > 32)) return (int)even(4 * LR_SMS / cgroups);
  const bool few = s.variant == 0;
  const int64_t beside = LR_SMS - std::min(LR_SMS, (npts + 7) / 8);  // SMs without a CTA of the state machine
  const double alone = std::min(1.5, 1.3 + 4.0 / p);
  int64_t pick = 1;
  double least = 1e300;
  for (int k = few ? 1 : 0; k <= 8; ++k) {
    const int64_t room = k == 0 ? beside : (int64_t)k * LR_SMS;
    if (k == 0 && room < cgroups) continue;
    const int64_t g = even(room / cgroups), per = (tiles + g - 1) / g, ctas = g * cgroups;
    const double busiest = (double)((ctas + LR_SMS - 1) / LR_SMS);
    double cost;
    if (few) {
      const double b = std::max(busiest, 4.0);
      cost = b * ((double)per + 0.15) * (1.0 + 0.8 / b) + 0.004 * (double)g;
    } else {
      cost = (ctas <= beside ? alone : std::max(busiest, 2.0)) * ((double)per + 0.4) + 0.006 * (double)g;
    }
    if (cost < 1.01 * least) pick = g;
    least = std::min(least, cost);
  }
  return (int)pick;
}
// Whether the tick loop's kernels of such a model start while the one before them ends.  That takes 4 to 20 % off a run
// of up to 512 chains.  With more the early CTAs crowd the SMs that the state machine's leave free: 1,000 rows x 1,024
// chains take 1.36 ms for 60 ticks against 1.12, 5,000 x 2,000 3.43 against 3.25; from 2,000 rows up to 1,024 chains still gain
// (1.50 against 1.60).
inline bool logreg_fp32_dependent(int64_t n, int npts) { return npts <= 512 || (npts <= 1024 && n > 1024); }

template <int CT, int NTH, int CG, int MINB>
static cudaError_t logreg_fp32_launch_variant(const LogregArgs& A, int row_groups, bool attr, cudaStream_t st,
                                              bool dependent) {
  const int dp = (A.p + 3) / 4 * 4;
  const dim3 grid((A.npts + CT - 1) / CT, row_groups);
  if (attr) {  // the shared-memory limit, at the most features each instance takes
    cudaError_t e = cudaFuncSetAttribute(logreg_fp32_kernel<CT, NTH, CG, 32, MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)LogregTile<CT, NTH, CG, 32>::bytes(32));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(logreg_fp32_kernel<CT, NTH, CG, 64, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)LogregTile<CT, NTH, CG, 64>::bytes(64));
    return e;
  }
  if (dp <= 32)
    return launch_tick(logreg_fp32_kernel<CT, NTH, CG, 32, MINB>, grid, NTH, LogregTile<CT, NTH, CG, 32>::bytes(dp), st,
                       dependent, A);
  return launch_tick(logreg_fp32_kernel<CT, NTH, CG, 64, MINB>, grid, NTH, LogregTile<CT, NTH, CG, 64>::bytes(dp), st,
                     dependent, A);
}

// variant < 0: sets every variant's shared-memory limit on the current device
static cudaError_t logreg_fp32_launch(int variant, const LogregArgs& A, int row_groups, cudaStream_t st, bool dependent) {
  const bool attr = variant < 0;
  cudaError_t e = cudaSuccess;
  if (attr || variant == 0) e = logreg_fp32_launch_variant<8, 32, 1, 6>(A, row_groups, attr, st, dependent);
  if ((attr && e == cudaSuccess) || variant == 1)
    e = logreg_fp32_launch_variant<16, 64, 1, 5>(A, row_groups, attr, st, dependent);
  if ((attr && e == cudaSuccess) || variant == 2)
    e = logreg_fp32_launch_variant<64, 256, 1, 2>(A, row_groups, attr, st, dependent);
  if ((attr && e == cudaSuccess) || variant == 3)
    e = logreg_fp32_launch_variant<128, 256, 2, 2>(A, row_groups, attr, st, dependent);
  return e;
}

}  // namespace gbn
