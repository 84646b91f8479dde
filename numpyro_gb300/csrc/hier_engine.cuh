// hier_engine.cuh -- the persistent NUTS engine of the hierarchical family with the chain in registers.
//
// One warp runs one chain; lane l holds the elements d = l + 32 k of the position, momentum,
// gradient, inverse mass and subtree momentum sum (K registers each), and a leaf -- both
// half-kicks, the drift, the potential, the energy, the multinomial choice, the U-turn checks --
// touches memory only for the data (y, 1/sigma) and the checkpoints.  It is the arithmetic of
// Chain<32> (nuts_engine.cu) and hier_nc_potential_warp, term for term and in the same order, so
// its draws are bit-identical to the tick engine's.
//
// What bounds it: the dependent instructions of one leaf for a few chains (4,300 cycles with its share of the
// transition's end), the FP64 pipe and instruction fetch for thousands.  The sums of a leaf (potential 3, kinetic energy 1, U-turn
// 2 per check) are float-float: a butterfly costs 5 x (2 shuffles + 11 FP32 adds).  Summed together,
// the values are dealt to lane groups in the first two steps (warp_sum3ff), so three of them cost 6
// additions instead of 15, in two rounds per leaf (the potential's sums, then the energy with the
// first U-turn check) instead of four.  The pairs that meet at each step, and so the bits, are those
// of the butterfly (ff_add commutes).  The uniforms of a transition's first 31 leaves come from one
// Philox evaluation (a lane each).
// Measured against the state machine over memory (persistent_hier_kernel): eight schools, 4 chains,
// 200 transitions 10.3 -> 4.8 ms; 16,384 chains of 4 to 256 groups, 5 transitions 8.2 -> 4.2 ms a call;
// dense mass matrices (M^-1 in shared memory, one row broadcast by shuffle a step), 64 chains of 32 dimensions,
// 100 warmup transitions 25.6 -> 9.4 ms, half of it from a warp per SM instead of eight.
#pragma once

namespace gbn {

__device__ __forceinline__ FF ff_from_lane(FF v, int src) {
  return FF{__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src)};
}

// Out of line: one copy of the generator per kernel instead of K + 3.  With 12 warps of an SM at
// different places of the tree, the size of the leaf loop's code is what the instruction cache sees.
__device__ __noinline__ uint4 hier_draw(Seed s, uint32_t chain, uint32_t n, uint32_t purpose, int idx, int sub) {
  return draw(s, chain, n, purpose, (uint32_t)idx, (uint32_t)sub);
}
__device__ __noinline__ float hier_momentum(Seed s, uint32_t chain, uint32_t n, int d) {
  return normal_at(s, chain, n, P_MOMENTUM, d, 0);
}

// The end of a transition (state, collection, adaptation and its step-size searches) through the
// generic state machine, out of line: it runs once per tree and its registers stay out of the leaf
// loop.  Returns how many transitions the chain has left.
template <bool DM>
__device__ __noinline__ int hier_end_transition(const AdvParams& P, const HierView& hv, int c, int m, int D, int lane,
                                                double pe, double energy, int num_steps, double accept_prob,
                                                int diverging, const float* znew, const float* gnew) {
  Chain<32, DM> ch{P, Group<32>{lane}, nullptr, c, D, P.D, P.e.ctl[c], nullptr};
  __syncwarp();  // ctl read by every lane before lane 0 writes it back
  const size_t row = (size_t)c * P.D;
  if (ch.finish_transition(pe, energy, num_steps, accept_prob, diverging, znew, gnew)) {
    const int j0 = hv.off[m], J = hv.off[m + 1] - j0;
    do {
      __syncwarp();  // Q written by other lanes
      hier_nc_potential_warp(P.e.Q + row, P.e.G + row, P.e.PE + c, J, hv.y + j0, hv.sinv + j0, hv.cmodel[m],
                             hv.inv_ms2, hv.inv_ts, lane);
      __syncwarp();  // G and PE written by other lanes
    } while (!ch.heur_finish());
    ch.heur_done();
  }
  ch.ctl.phase = ch.ctl.iters_left > 0 ? PH_START : PH_DONE;
  if (lane == 0) P.e.ctl[c] = ch.ctl;
  __syncwarp();
  return ch.ctl.iters_left;
}

// Every transition of chain c, of latent dimension at most 32 K.  ck_warp: ck_floats floats of
// shared memory for the shallowest (most used) of its U-turn checkpoints (momentum and momentum sum).
// DM: dense mass matrices; minv then holds 32 K floats of shared memory for each row of M^-1.
template <int K, bool DM>
__device__ __forceinline__ void hier_run_chain(const AdvParams& P, const HierView& hv, int c, int m, int D, int lane,
                                               float* ck_warp, int ck_floats, float* minv) {
  const uint32_t FULL = 0xffffffffu;
  const int ck_slots = ck_floats / (64 * K);
  const int j0 = hv.off[m], J = hv.off[m + 1] - j0;
  const float* __restrict__ y = hv.y + j0;
  const float* __restrict__ sinv = hv.sinv + j0;
  const double cmodel = hv.cmodel[m];
  const int kc = (D + 31) >> 5;
  const size_t row = (size_t)c * P.D;
  float* const r_ck = P.e.r_ck + row * P.maxd;
  float* const rs_ck = P.e.rs_ck + row * P.maxd;
  int iters_left = P.e.ctl[c].iters_left;
  while (iters_left > 0) {
    // ---------------------------------------------------------- start of a transition
    const uint32_t n = P.s.rng_key[2 * c + 1], cid = P.s.rng_key[2 * c];
    float z[K], r[K], g[K], mi[DM ? 1 : K], rss[K];
    float kin0f = 0.0f;
    // v = M^-1 x, terms in the order of Chain::sym_matvec
    auto matvec = [&](const float* x, float* v) {
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = 0.0f;
#pragma unroll
      for (int kb = 0; kb < K; ++kb) {
        const int rows = min(32, D - 32 * kb);
#pragma unroll 8
        for (int j = 0; j < rows; ++j) {
          const float xj = __shfl_sync(FULL, x[kb], j);
          const float* const a = minv + (32 * kb + j) * (32 * K) + lane;
#pragma unroll
          for (int k = 0; k < K; ++k) v[k] = fmaf(a[32 * k], xj, v[k]);
        }
      }
    };
    if (DM) {  // M^-1 may have changed at a window end
      const float* const src = P.s.inverse_mass_matrix + row * P.D;
      constexpr int B = 8;  // rows in flight: one at a time, 96 rows took 33 us, half of a transition of one leaf
      __syncwarp();
      for (int j = 0; j < D; j += B) {
        float a[B][K];
#pragma unroll
        for (int i = 0; i < B; ++i)
#pragma unroll
          for (int k = 0; k < K; ++k)
            a[i][k] = j + i < D && lane + 32 * k < D ? src[(size_t)(j + i) * P.D + lane + 32 * k] : 0.0f;
#pragma unroll
        for (int i = 0; i < B; ++i)
#pragma unroll
          for (int k = 0; k < K; ++k)
            if (j + i < D) minv[(j + i) * (32 * K) + 32 * k + lane] = a[i][k];
      }
      __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int d = lane + 32 * k;
      const bool in = d < D;
      z[k] = in ? P.s.z[row + d] : 0.0f;
      g[k] = in ? P.s.z_grad[row + d] : 0.0f;
      if (!DM) mi[DM ? 0 : k] = in ? P.s.inverse_mass_matrix[row + d] : 0.0f;
      r[k] = 0.0f;
      rss[k] = 0.0f;
      if (k < kc) {
        const float e = hier_momentum(P.seed, cid, n, d);
        if (DM) {
          if (in) P.e.tmp[row + d] = e;
        } else if (in) {
          r[k] = P.s.mass_matrix_sqrt[row + d] * e;
          kin0f = fmaf(mi[DM ? 0 : k] * r[k], r[k], kin0f);
          P.e.r_l[row + d] = r[k];
          P.e.rsum[row + d] = r[k];
        }
      }
    }
    if (DM) {  // r = S eps, as Chain::dense_momentum
      __syncwarp();
      const float* const eps = P.e.tmp + row;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int d = lane + 32 * k;
        if (d < D) {
          const float* const Si = P.s.mass_matrix_sqrt + (row + d) * P.D;
          float acc = 0.0f;
#pragma unroll 4
          for (int j = 0; j < D; ++j) acc = fmaf(Si[j], eps[j], acc);
          r[k] = acc;
          P.e.r_l[row + d] = acc;
          P.e.rsum[row + d] = acc;
        }
      }
      float v[K];
      matvec(r, v);
#pragma unroll
      for (int k = 0; k < K; ++k) kin0f = fmaf(v[k], r[k], kin0f);
    }
    FF kff = ff_from(kin0f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) kff = ff_add(kff, ff_shfl_xor(kff, o));
    const double pe0 = P.s.potential_energy[c];
    const double energy0 = pe0 + 0.5 * ff_value(kff);
    const float step = P.s.step_size[c];
    const int max_depth = (P.s.i[c] < P.num_warmup) ? P.mtd_warmup : P.mtd;
    // lane l: the doubling's draws at depth l; the leaf uniform of leaf l - 2^depth at depth
    // floor(log2 l)
    const uint4 wd = hier_draw(P.seed, cid, n, P_DOUBLING, lane, 0);
    uint32_t wl = 0;
    {
      const int dl = 31 - __clz(lane | 1);
      wl = hier_draw(P.seed, cid, n, P_LEAF, dl, lane - (1 << dl)).x;
    }
    int depth = 0, side = 0, prop = -1;  // prop: proposal rows (-1: the starting state)
    bool other_is_start = true;          // the inactive frontier's position is still the starting one
    double tree_w = 0.0, tree_acc = 0.0, pe_p = pe0, energy_p = energy0;
    int num_prop = 0;
    bool tree_div = false, tree_turning = false;
    // The inactive frontier lives in the rows z_l, r_l, g_l (whichever side it is).
    do {
      // -------------------------------------------------------- one doubling
      const int dir = u01f(__shfl_sync(FULL, wd.x, depth)) < 0.5f ? 1 : 0;
      const float u_take = u01f(__shfl_sync(FULL, wd.y, depth));
      if (depth > 0 && dir != side) {  // swap the frontiers
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int d = lane + 32 * k;
          if (d >= D) continue;
          const float zo = other_is_start ? P.s.z[row + d] : P.e.z_l[row + d];
          const float go = other_is_start ? P.s.z_grad[row + d] : P.e.g_l[row + d];
          const float ro = P.e.r_l[row + d];
          P.e.z_l[row + d] = z[k];
          P.e.r_l[row + d] = r[k];
          P.e.g_l[row + d] = g[k];
          z[k] = zo;
          r[k] = ro;
          g[k] = go;
        }
        other_is_start = false;
      }
      side = dir;
      const float eps = dir ? step : -step;
      const int sprop = prop == 0 ? 1 : 0;
      float* const zsp = (sprop ? P.e.z_sp : P.e.z_p) + row;
      float* const gsp = (sprop ? P.e.g_sp : P.e.g_p) + row;
      double sub_w = -INFINITY, sub_acc = 0.0, pe_sp = 0.0, energy_sp = 0.0;
      int leaf = 0;
      bool sub_div = false, sub_turning = false;
      do {
        if (depth > 4 && (leaf == 1 || ((leaf & 31) == 0 && leaf > 0)))  // lane l: leaf l of this block of 32
          wl = hier_draw(P.seed, cid, n, P_LEAF, depth, (leaf & ~31) + lane).x;
        // ------------------------------------------------------ leapfrog to the new position
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float rh = r[k] - 0.5f * eps * g[k];
          if (!DM) z[k] = z[k] + eps * (mi[DM ? 0 : k] * rh);
          r[k] = rh;
        }
        float v[K];
        if (DM) {
          matvec(r, v);
#pragma unroll
          for (int k = 0; k < K; ++k) z[k] = z[k] + eps * v[k];
        }
        // ------------------------------------------------------ potential (hier_potential.cuh)
        // group j = lane + 32 k is element j + 2: two lanes up
        const float mu = __shfl_sync(FULL, z[0], 0), lt = __shfl_sync(FULL, z[0], 1);
        const float tau = expf(lt);
        float lpf = 0.0f, swf = 0.0f, swef = 0.0f;
        float gj[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
          gj[k] = 0.0f;
          if (k >= kc) continue;
          const float zup = k + 1 < K ? z[k + 1 < K ? k + 1 : k] : 0.0f;
          const float eta = __shfl_sync(FULL, lane < 2 ? zup : z[k], (lane + 2) & 31);
          const int j = lane + 32 * k;
          if (j < J) {
            const float is = sinv[j];
            const float th = fmaf(tau, eta, mu);
            const float rr = (y[j] - th) * is;
            lpf += -0.5f * eta * eta - 0.5f * rr * rr;
            const float w = rr * is;
            swf += w;
            swef = fmaf(w, eta, swef);
            gj[k] = eta - tau * w;
          }
        }
        const FF ps = warp_sum3ff(ff_from(swf), ff_from(lpf), ff_from(swef), lane);
        const FF fsw = ff_from_lane(ps, 0), fswe = ff_from_lane(ps, 16), flp = ff_from_lane(ps, 8);
        const float sw = fsw.hi + fsw.lo, swe = fswe.hi + fswe.lo;
        const float u = tau * hv.inv_ts;
        const float u2 = u * u;
        const float lp_prior = -0.5f * mu * mu * hv.inv_ms2 - log1pf(u2) + lt;
        const double pe = -(ff_value_int(flp) + f2d(lp_prior) - cmodel);
        const float g0 = mu * hv.inv_ms2 - sw;
        const float g1 = 2.0f * u2 / (1.0f + u2) - 1.0f - tau * swe;
        // ------------------------------------------------------ second half-kick, energy, momentum sum
        float kinf = 0.0f;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (k >= kc) continue;
          const float dn = k > 0 ? gj[k > 0 ? k - 1 : 0] : 0.0f;
          float gn = __shfl_sync(FULL, lane >= 30 ? dn : gj[k], (lane + 30) & 31);
          if (k == 0) gn = lane == 0 ? g0 : (lane == 1 ? g1 : gn);
          const float rn = r[k] - 0.5f * eps * gn;
          r[k] = rn;
          g[k] = gn;
          if (!DM) kinf = fmaf(mi[DM ? 0 : k] * rn, rn, kinf);
          rss[k] = leaf == 0 ? rn : rss[k] + rn;
        }
        if (DM) {
          matvec(r, v);
#pragma unroll
          for (int k = 0; k < K; ++k) kinf = fmaf(v[k], r[k], kinf);
        }
        // ------------------------------------------------------ checkpoints and U-turn checks
        const int idx_max = __popc((unsigned)(leaf >> 1));
        const bool odd = (leaf & 1) != 0;
        const int idx_min = odd ? idx_max + 1 - __popc((unsigned)((~leaf & (leaf + 1)) - 1)) : idx_max;
        FF kin{0.0f, 0.0f};
        // one pass per check (an even leaf: one pass that stores its checkpoint instead); the first
        // pass also sums the kinetic energy
        for (int idx = idx_max; idx >= idx_min && !sub_turning; --idx) {
          const bool on_chip = idx < ck_slots;
          float* const rc = on_chip ? ck_warp + idx * (64 * K) : r_ck + idx * P.D;
          float* const rsc = on_chip ? rc + 32 * K : rs_ck + idx * P.D;
          float ax = odd ? 0.0f : 1.0f, ay = ax;  // 1: no turn
          float left[K], mid[K];  // DM: the checkpoint's momentum, the subtree's sum less the end points' mean
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int d = lane + 32 * k;
            if (DM) left[k] = mid[k] = 0.0f;
            if (d >= D) continue;
            if (odd) {
              const float av = rc[d];
              const float sv = (rss[k] - rsc[d]) + av;
              const float s = sv - 0.5f * (av + r[k]);
              if (DM) {
                left[k] = av;
                mid[k] = s;
              } else {
                ax = fmaf(mi[DM ? 0 : k] * av, s, ax);
                ay = fmaf(mi[DM ? 0 : k] * r[k], s, ay);
              }
            } else {
              rc[d] = r[k];
              rsc[d] = rss[k];
            }
          }
          if (DM && odd) {
            matvec(mid, v);
#pragma unroll
            for (int k = 0; k < K; ++k) {
              ax = fmaf(left[k], v[k], ax);
              ay = fmaf(r[k], v[k], ay);
            }
          }
          const FF sums = warp_sum3ff(ff_from(kinf), ff_from(ax), ff_from(ay), lane);
          if (idx == idx_max) kin = ff_from_lane(sums, 0);
          sub_turning = (__ballot_sync(FULL, ff_le0(sums)) & ((1u << 8) | (1u << 16))) != 0u;
        }
        // ------------------------------------------------------ energy, divergence, multinomial choice
        const double e_new = pe + ff_half(kin);
        double dE = e_new - energy0;
        if (d_isnan(dE)) dE = INFINITY;
        const double w = -dE;
        sub_div = d_gt_pos(dE, P.max_dE);
        sub_acc += f2d(exp_min1_f(w));
        // sigmoid_f(w - sub_w) and logaddexp_mixed(sub_w, w) from one difference; the first leaf
        // meets an empty subtree of weight -infinity
        const double dw = w - sub_w;
        const float x = (float)dw;
        const float ul = u01f(__shfl_sync(FULL, wl, depth <= 4 ? (1 << depth) + leaf : leaf & 31));
        const bool take = leaf == 0 || ul < 1.0f / (1.0f + expf(-x));
        sub_w = logaddexp_diff(sub_w, w, dw, x);
        if (take) {
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int d = lane + 32 * k;
            if (d < D) {
              zsp[d] = z[k];
              gsp[d] = g[k];
            }
          }
          pe_sp = pe;
          energy_sp = e_new;
        }
        ++leaf;
      } while (leaf < (1 << depth) && !sub_turning && !sub_div);
      // -------------------------------------------------------- combine the subtree (biased)
      float p = 0.0f;
      const double dw = sub_w - tree_w;
      const float x = (float)dw;
      if (!(sub_turning || sub_div)) p = fminf(expf(x), 1.0f);
      float ax = 0.0f, ay = 0.0f;
      float lr[K], rr[K], mid[K], v[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int d = lane + 32 * k;
        if (DM) lr[k] = rr[k] = mid[k] = 0.0f;
        if (d < D) {
          const float sv = P.e.rsum[row + d] + rss[k];
          P.e.rsum[row + d] = sv;
          const float ro = P.e.r_l[row + d];
          const float av = dir ? ro : r[k], bv = dir ? r[k] : ro;  // left, right
          const float s = sv - 0.5f * (av + bv);
          if (DM) {
            lr[k] = av;
            rr[k] = bv;
            mid[k] = s;
          } else {
            ax = fmaf(mi[DM ? 0 : k] * av, s, ax);
            ay = fmaf(mi[DM ? 0 : k] * bv, s, ay);
          }
        }
      }
      if (DM) {
        matvec(mid, v);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          ax = fmaf(lr[k], v[k], ax);
          ay = fmaf(rr[k], v[k], ay);
        }
      }
      tree_turning = sub_turning;
      if (!tree_turning) {
        const FF sums = warp_sum3ff(ff_from(ax), ff_from(ay), FF{1.0f, 0.0f}, lane);
        tree_turning = (__ballot_sync(FULL, ff_le0(sums)) & ((1u << 0) | (1u << 8))) != 0u;
      }
      if (u_take < p) {
        prop = sprop;
        pe_p = pe_sp;
        energy_p = energy_sp;
      }
      depth += 1;
      tree_w = logaddexp_diff(tree_w, sub_w, dw, x);
      tree_div = sub_div;
      tree_acc += sub_acc;
      num_prop += leaf;
    } while (depth < max_depth && !tree_turning && !tree_div);
    // ---------------------------------------------------------- end of the transition
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (lane + 32 * k < D) P.e.Q[row + lane + 32 * k] = z[k];  // the last queried position
    const float* znew = prop < 0 ? P.s.z + row : (prop ? P.e.z_sp : P.e.z_p) + row;
    const float* gnew = prop < 0 ? P.s.z_grad + row : (prop ? P.e.g_sp : P.e.g_p) + row;
    iters_left = hier_end_transition<DM>(P, hv, c, m, D, lane, pe_p, energy_p, num_prop, tree_acc / (double)num_prop,
                                     tree_div, znew, gnew);
  }
}

// 12 warps per SM with up to 168 registers each: 16 warps with 128 took 4.0 against 3.8 ms (4,096
// models of 4 to 256 groups, 16,384 chains, 5 transitions), 20 took 4.4.  One K per launch: letting
// each chain run the smallest instance that holds it was no faster (several loops share the
// instruction caches then).
template <int K, bool DM>
__global__ void __launch_bounds__(128, 3)
    persistent_hier_reg_kernel(const AdvParams* __restrict__ Pp, const __grid_constant__ HierView hv,
                               int32_t* queue_head, const int32_t* __restrict__ order, int ck_floats) {
  __shared__ __align__(16) AdvParams sp;
  extern __shared__ float ck_smem[];
  const AdvParams& P = stage_params(Pp, &sp);
  const int lane = threadIdx.x & 31;
  const int mass_floats = DM ? P.D * (32 * K) : 0;
  float* const minv = ck_smem + (size_t)(threadIdx.x >> 5) * (ck_floats + mass_floats);
  float* const ck_warp = minv + mass_floats;
  for (;;) {
    int q = 0;
    if (lane == 0) q = atomicAdd(queue_head, 1);
    q = __shfl_sync(0xffffffffu, q, 0);
    if (q >= P.C) break;
    const int c = order ? order[q] : q;
    int m = c / hv.cpm;
    if (m >= hv.num_models) m = hv.num_models - 1;
    const int D = P.e.chain_dim ? P.e.chain_dim[c] : P.D;
    hier_run_chain<K, DM>(P, hv, c, m, D, lane, ck_warp, ck_floats, minv);
  }
}

}  // namespace gbn
