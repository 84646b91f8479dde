// sv_engine.cuh -- the persistent NUTS engine of the stochastic-volatility family with the chain on chip.
//
// One CTA runs one chain: eight element warps and two scalar warps.  Element thread i owns the
// coordinates d = i + 256 k; momentum, inverse mass and subtree momentum sum are in its registers,
// position, gradient and the newest U-turn checkpoint in shared memory (index d + d / 16, so that
// the non-centred walk's chunk order meets few bank conflicts).  A leaf touches global memory only
// for the returns (cached), the older checkpoints and the proposal.
//
// What bounds a leaf is its chain of block-wide steps.  The state machine over memory
// (persistent_sv_kernel) had about a dozen barriers and memory round trips, its FP64 (64 cycles a
// dependent operation, one warp instruction per 19 cycles and SM) ran in all eight warps, and the
// log-gammas (1,700 to 3,100 cycles) in front of two warps' elements.  Here a leaf has two
// barriers, and everything scalar runs beside the element warps: in warp 8 the digammas and the previous
// leaf's energy, multinomial choice and U-turn verdict beside the potential's elements, the tail of the
// gradient beside the second half-kick; in warp 9 the log-gammas beside the elements and the potential
// beside the half-kick (one scalar warp for both took 14,400 cycles a leaf, T = 1,001).  A leaf's verdict so arrives one leaf late; as a turn or a
// divergence ends the whole tree, the leaf computed too far is just left out.  Each leaf's position
// and gradient go to one of three proposal rows, and the choice only names the row.
//
// The arithmetic is that of Chain<256> and sv_potential.cuh, term for term and in the same order (the
// group sums fold the same warp sums), so draws are bit-identical to the tick engine's.
// Measured, one NUTS run each: T = 4,096 centred, 256 chains, 1,023 leaves 22.2 -> 12.0 ms; T = 1,001
// non-centred, 16 chains, 380 leaves 5.0 -> 2.4 ms.  Two chains per SM keep the issue slots 58 % busy; FP32x2
// compensated sums were no faster (the pairs cost the moves they save).
#pragma once

namespace gbn {

// The 256 element threads as a group: as Group<256>, on a named barrier, for the end of a transition.  It has no sums,
// which only step-size searches need there: runs of a handle that has them take persistent_sv_kernel.
struct SvGroup {
  static constexpr bool searches = false;
  int tid;
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync 2, 256;" ::: "memory"); }
};

struct SvEngineSmem {
  float2 r1[5][8];    // potential sums per warp
  float2 r2[42][8];   // kinetic energy and U-turn sums per warp
  float2 wt[2][8];    // scans of the non-centred walk
  float gtail[2];     // dU/d log nu, dU/d log s
  double pe;          // potential of the newest leaf
  int take, stop;     // verdict on a leaf
  int next_chain, iters_left, tree_more, tree_take;
};

constexpr int SV_MASS_REGS = 9;  // more coordinates per thread than this: the inverse mass in shared memory
inline size_t sv_engine_smem(int D, bool noncentred, int K) {
  const size_t row = sizeof(float) * (size_t)(D + D / 16 + 1);
  return row * (4 + (noncentred ? 1 : 0) + (K > SV_MASS_REGS ? 1 : 0));
}

// The end of a transition through the generic state machine (element threads only).
__device__ __noinline__ int sv_end_transition(const AdvParams& P, int c, int tid, double pe, double energy,
                                              int num_steps, double accept_prob, int diverging, const float* znew,
                                              const float* gnew) {
  Chain<256, false, SvGroup> ch{P, SvGroup{tid}, nullptr, c, P.D, P.D, P.e.ctl[c], nullptr};
  ch.g.sync();  // every thread has read ctl before thread 0 writes it back
  ch.finish_transition(pe, energy, num_steps, accept_prob, diverging, znew, gnew);
  ch.ctl.phase = ch.ctl.iters_left > 0 ? PH_START : PH_DONE;
  if (tid == 0) P.e.ctl[c] = ch.ctl;
  return ch.ctl.iters_left;
}

// K: coordinates per element thread (D <= 256 K).  Two CTAs an SM leave 96 registers: ptxas spills (bytes of stores /
// loads) 144 / 290 at K = 17 centred, 496 / 922 non-centred, 348 / 610 at 13 non-centred, 256 / 378 at 9, 80 / 84 at 4.
template <int K, bool NC>
__global__ void __launch_bounds__(320, 2)
    persistent_sv_reg_kernel(const AdvParams* __restrict__ Pp, SvView sv, int32_t* queue_head) {
  __shared__ __align__(16) AdvParams sp;
  __shared__ SvEngineSmem sm;
  extern __shared__ float rows[];
  const AdvParams& P = stage_params(Pp, &sp);
  const uint32_t FULL = 0xffffffffu;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool scalar = warp == 8, element = warp < 8;
  const int D = P.D, T = sv.T, rowlen = D + D / 16 + 1;
  float* const zs = rows;
  float* const gs = zs + rowlen;
  float* const ckr = gs + rowlen;   // the newest checkpoint: momentum and momentum sum
  float* const cks = ckr + rowlen;
  float* const rets = cks + rowlen;  // NC: the returns
  constexpr bool MREG = K <= SV_MASS_REGS;
  float* const ms = rets + (NC ? rowlen : 0);  // the inverse mass where registers do not hold it
  // element k of this thread: d = tid + 256 k at position p0 + 272 k; it has kd of them
  const int p0 = sv_pos(tid), kd = !element ? 0 : (D - tid + 255) >> 8;
  const int below = (tid & 15) == 0 ? 2 : 1, above = (tid & 15) == 15 ? 2 : 1;
  const bool owner = element && (warp == ((T & 255) >> 5) || warp == (((T + 1) & 255) >> 5));  // of log nu, log s
  const int tail_threads = 32 + (((T & 255) >> 5) == (((T + 1) & 255) >> 5) ? 32 : 64);
  const double log_rates = (double)(logf((float)sv.s_rate) + logf((float)sv.nu_rate));
  if (NC)
    for (int t = tid; t < T; t += 320) rets[sv_pos(t)] = sv.ret[t];
  for (;;) {
    __syncthreads();
    if (tid == 0) sm.next_chain = atomicAdd(queue_head, 1);
    __syncthreads();
    const int c = sm.next_chain;
    if (c >= P.C) break;
    const size_t row = (size_t)c * D;
    int iters_left = P.e.ctl[c].iters_left;
    while (iters_left > 0) {
      // ---------------------------------------------------------------- start of a transition
      const uint32_t n = P.s.rng_key[2 * c + 1], cid = P.s.rng_key[2 * c];
      const float step = P.s.step_size[c];
      const int max_depth = (P.s.i[c] < P.num_warmup) ? P.mtd_warmup : P.mtd;
      const double pe0 = P.s.potential_energy[c];
      const uint4 wd = hier_draw(P.seed, cid, n, P_DOUBLING, lane, 0);  // lane l: the doubling at depth l
      float r[K], mi[MREG ? K : 1], rss[K];
      auto mass = [&](int k) -> float { return MREG ? mi[MREG ? k : 0] : ms[p0 + 272 * k]; };
      if (element) {
        float kinf = 0.0f;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const int d = tid + 256 * k;
          r[k] = 0.0f;
          rss[k] = 0.0f;
          if (k < kd) {
            zs[p0 + 272 * k] = P.s.z[row + d];
            gs[p0 + 272 * k] = P.s.z_grad[row + d];
            const float m = P.s.inverse_mass_matrix[row + d];
            if (MREG)
              mi[MREG ? k : 0] = m;
            else
              ms[p0 + 272 * k] = m;
            r[k] = P.s.mass_matrix_sqrt[row + d] * hier_momentum(P.seed, cid, n, d);
            kinf = fmaf(m * r[k], r[k], kinf);
            P.e.r_l[row + d] = r[k];
            P.e.rsum[row + d] = r[k];
          }
        }
        FF v = ff_from(kinf);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = ff_add(v, ff_shfl_xor(v, o));
        if (lane == 0) sm.r2[0][warp] = make_float2(v.hi, v.lo);
      }
      __syncthreads();
      // scalar warp: the state of the tree
      double energy0 = 0.0, tree_w = 0.0, tree_acc = 0.0, pe_p = pe0, energy_p = 0.0;
      uint32_t wl = 0;
      if (scalar) {
        const FF k0 = sv_fold(sm.r2, 0);
        energy0 = pe0 + 0.5 * ff_value(k0);
        energy_p = energy0;
        const int dl = 31 - __clz(lane | 1);  // leaf uniforms of depths 0 to 4, as in hier_run_chain
        wl = hier_draw(P.seed, cid, n, P_LEAF, dl, lane - (1 << dl)).x;
      }
      int depth = 0, side = 0, prop = -1, num_prop = 0;
      bool other_is_start = true, tree_div = false;
      for (;;) {
        // -------------------------------------------------------------- one doubling
        const int dir = u01f(__shfl_sync(FULL, wd.x, depth)) < 0.5f ? 1 : 0;
        if (element && depth > 0 && dir != side) {  // swap the frontiers
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int d = tid + 256 * k;
            if (k >= kd) continue;
            const float zo = other_is_start ? P.s.z[row + d] : P.e.z_l[row + d];
            const float go = other_is_start ? P.s.z_grad[row + d] : P.e.g_l[row + d];
            const float ro = P.e.r_l[row + d];
            P.e.z_l[row + d] = zs[p0 + 272 * k];
            P.e.g_l[row + d] = gs[p0 + 272 * k];
            P.e.r_l[row + d] = r[k];
            zs[p0 + 272 * k] = zo;
            gs[p0 + 272 * k] = go;
            r[k] = ro;
          }
        }
        if (depth > 0 && dir != side) other_is_start = false;
        side = dir;
        const float eps = dir ? step : -step;
        int sprop = -1, cur = -1;  // rows of the subtree's proposal and of the newest leaf
        double sub_w = -INFINITY, sub_acc = 0.0, pe_sp = 0.0, energy_sp = 0.0;
        bool sub_div = false, sub_turning = false;
        int leaf = 0;
        // scalar warp: energy, divergence, choice and U-turn verdict of leaf `at`
        auto decide = [&](int at) {
          const int checks = (at & 1) ? __popc((unsigned)((~at & (at + 1)) - 1)) : 0;
          const FF v = sv_fold(sm.r2, lane <= 2 * checks ? lane : 0);
          bool turn = lane > 0 && lane <= 2 * checks && ff_le0(v);
          for (int i = lane + 32; i <= 2 * checks; i += 32) turn = turn || ff_le0(sv_fold(sm.r2, i));
          sub_turning = __any_sync(FULL, turn);
          const FF kin = ff_from_lane(v, 0);
          const double pe_leaf = sm.pe, e_new = pe_leaf + ff_half(kin);
          double dE = e_new - energy0;
          if (d_isnan(dE)) dE = INFINITY;
          const double w = -dE;
          sub_div = d_gt_pos(dE, P.max_dE);
          sub_acc += f2d(exp_min1_f(w));
          if (depth > 4 && (at == 1 || ((at & 31) == 0 && at > 0)))  // lane l: leaf l of this block of 32
            wl = hier_draw(P.seed, cid, n, P_LEAF, depth, (at & ~31) + lane).x;
          const double dw = w - sub_w;
          const float x = (float)dw;
          const float ul = u01f(__shfl_sync(FULL, wl, depth <= 4 ? (1 << depth) + at : at & 31));
          const bool take = at == 0 || ul < 1.0f / (1.0f + expf(-x));
          sub_w = logaddexp_diff(sub_w, w, dw, x);
          if (take) {
            pe_sp = pe_leaf;
            energy_sp = e_new;
          }
          if (lane == 0) {
            sm.take = take;
            sm.stop = sub_div || sub_turning;
          }
        };
        for (;;) {
          // ------------------------------------------------------------ leapfrog to the new position
          if (element) {
#pragma unroll
            for (int k = 0; k < K; ++k) {
              if (k >= kd) continue;
              const float rh = r[k] - 0.5f * eps * gs[p0 + 272 * k];
              zs[p0 + 272 * k] = zs[p0 + 272 * k] + eps * (mass(k) * rh);
              r[k] = rh;
            }
          }
          __syncthreads();  // positions of this leaf, sums of the one before
          const float lnuf = zs[sv_pos(T)], lsf = zs[sv_pos(T + 1)];
          const float nuf = expf(lnuf), sf = expf(lsf), inv_nuf = 1.0f / nuf;
          float dg0 = 0.0f, dg1 = 0.0f;
          double lg0 = 0.0, lg1 = 0.0;
          if (warp == 9) {
            const double nu = (double)nuf;
            const double lg = lgamma(0.5 * (lane == 1 ? nu + 1.0 : nu));
            lg0 = __shfl_sync(FULL, lg, 0);
            lg1 = __shfl_sync(FULL, lg, 1);
          } else if (scalar) {
            const float dg = digamma_f(0.5f * (lane == 1 ? nuf + 1.0f : nuf));
            dg0 = __shfl_sync(FULL, dg, 0);
            dg1 = __shfl_sync(FULL, dg, 1);
            if (leaf > 0) decide(leaf - 1);
          } else if (!NC) {
            const float inv_s2 = 1.0f / (sf * sf);
            Comp32 sdd{0.0f, 0.0f}, sl1p{0.0f, 0.0f}, sfrac{0.0f, 0.0f}, sh{0.0f, 0.0f};
#pragma unroll 4
            for (int t = tid, q = p0; t < T; t += 256, q += 272) {
              // the neighbours' positions: one further where t is the last or the first of 16
              const float hp = t > 0 ? zs[q - below] : 0.0f;
              gs[q] = sv_centred_step(t, T, zs[q], hp, zs[q + above], __ldg(sv.ret + t), nuf, inv_nuf, inv_s2, sdd,
                                      sl1p, sfrac, sh);
            }
            const FF v = warp_sum4ff(comp_ff(sdd), comp_ff(sl1p), comp_ff(sfrac), comp_ff(sh), lane);
            if ((lane & 7) == 0) sm.r1[lane >> 3][warp] = make_float2(v.hi, v.lo);
          } else {
            sv_nc_elements<K>(zs, rets, gs, T, tid, sf, nuf, inv_nuf, sm.r1, sm.wt);
          }
          __syncthreads();  // sums of the potential, gradients, verdict on the leaf before
          if (leaf > 0) {
            if (sm.take) sprop = cur;
            if (sm.stop) break;  // the tree ends with the leaf before; this one is left out
          }
          if (!element) {
            const FF v = sv_fold(sm.r1, lane < (NC ? 5 : 4) ? lane : 0);
            const double sums = ff_value(v);
            const double nu = (double)nuf, inv_nu = (double)inv_nuf, s = (double)sf, inv_s = (double)(1.0f / sf);
            const double S0 = __shfl_sync(FULL, sums, 0), S1 = __shfl_sync(FULL, sums, 1),
                         S2 = __shfl_sync(FULL, sums, 2), S3 = __shfl_sync(FULL, sums, 3);
            const double S_l1p = NC ? S0 : S1, S_frac = NC ? S1 : S2, S_h = NC ? S2 : S3;
            if (scalar) {
              const double special[6] = {0.0, 0.0, (double)dg0, (double)dg1, nu, inv_nu};
              const float gl = sv_grad_lnu(S_l1p, S_frac, (double)T, sv.nu_rate, special);
              const float gsv = sv_grad_ls(NC, NC ? S3 : S0, (double)T, s, inv_s, sv.s_rate);
              if (lane == 0) {
                sm.gtail[0] = gl;
                sm.gtail[1] = gsv;
              }
              __syncwarp();
              asm volatile("bar.arrive 1, %0;" ::"r"(tail_threads) : "memory");
            } else {  // only the verdict, a leaf later, needs the potential
              const double S_walk = NC ? __shfl_sync(FULL, sums, 4) : S0;
              const double pe = -sv_log_joint(NC, S_walk, S_l1p, S_h, (double)T, lnuf, lsf, nu, s, inv_s, log_rates,
                                              sv.s_rate, sv.nu_rate, lg0, lg1);
              if (lane == 0) sm.pe = pe;
            }
          } else {
            if (owner) asm volatile("bar.sync 1, %0;" ::"r"(tail_threads) : "memory");
            // ---------------------------------------------------------- second half-kick, momentum sum, proposal row
            cur = 0;
            while (cur == prop || cur == sprop) ++cur;
            float* const zrow = (cur == 0 ? P.e.z_p : (cur == 1 ? P.e.z_sp : P.e.z_r)) + row;
            float* const grow = (cur == 0 ? P.e.g_p : (cur == 1 ? P.e.g_sp : P.e.g_r)) + row;
            float kinf = 0.0f;
            auto finish = [&](int k) {  // element k: momentum at the leaf, its sum, the proposal row
              const int d = tid + 256 * k;
              float gn = gs[p0 + 272 * k];
              if (d >= T) {
                gn = sm.gtail[d - T];
                gs[p0 + 272 * k] = gn;
              }
              const float rn = r[k] - 0.5f * eps * gn;
              r[k] = rn;
              kinf = fmaf(mass(k) * rn, rn, kinf);
              rss[k] = leaf == 0 ? rn : rss[k] + rn;
              zrow[d] = zs[p0 + 272 * k];
              grow[d] = gn;
            };
            // ---------------------------------------------------------- checkpoints and U-turn sums
            const int idx_max = __popc((unsigned)(leaf >> 1));
            if ((leaf & 1) == 0) {
              // the next leaf's first check reads the newest checkpoint; older ones are read again only
              // where the leaf number is a multiple of 4
              const bool keep = (leaf & 2) == 0;
              float* const rc = P.e.r_ck + (row * P.maxd + (size_t)idx_max * D) + tid;
              float* const rsc = P.e.rs_ck + (row * P.maxd + (size_t)idx_max * D) + tid;
#pragma unroll
              for (int k = 0; k < K; ++k) {
                if (k >= kd) continue;
                finish(k);
                ckr[p0 + 272 * k] = r[k];
                cks[p0 + 272 * k] = rss[k];
                if (keep) {
                  rc[256 * k] = r[k];
                  rsc[256 * k] = rss[k];
                }
              }
              FF kin = ff_from(kinf);
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) kin = ff_add(kin, ff_shfl_xor(kin, o));
              if (lane == 0) sm.r2[0][warp] = make_float2(kin.hi, kin.lo);
            } else {
              const int checks = __popc((unsigned)((~leaf & (leaf + 1)) - 1));
              float ax = 0.0f, ay = 0.0f;
              auto turn = [&](int k, float av, float minus) {  // one element of a check
                const float s = ((rss[k] - minus) + av) - 0.5f * (av + r[k]);
                const float m = mass(k);
                ax = fmaf(m * av, s, ax);
                ay = fmaf(m * r[k], s, ay);
              };
#pragma unroll
              for (int k = 0; k < K; ++k) {
                if (k >= kd) continue;
                finish(k);
                turn(k, ckr[p0 + 272 * k], cks[p0 + 272 * k]);
              }
              FF v = warp_sum3ff(ff_from(kinf), ff_from(ax), ff_from(ay), lane);
              if ((lane & 7) == 0 && lane < 24) sm.r2[lane >> 3][warp] = make_float2(v.hi, v.lo);
              for (int j = 1; j < checks; ++j) {
                const float* const rc = P.e.r_ck + (row * P.maxd + (size_t)(idx_max - j) * D) + tid;
                const float* const rsc = P.e.rs_ck + (row * P.maxd + (size_t)(idx_max - j) * D) + tid;
                ax = 0.0f;
                ay = 0.0f;
                constexpr int B = K < 6 ? K : 6;  // loads in flight: one memory round trip a batch
#pragma unroll
                for (int k0 = 0; k0 < K; k0 += B) {
                  float a[B], b[B];
#pragma unroll
                  for (int k = 0; k < B; ++k) {
                    const bool in = k0 + k < K && k0 + k < kd;
                    a[k] = in ? rc[256 * (k0 + k)] : 0.0f;
                    b[k] = in ? rsc[256 * (k0 + k)] : 0.0f;
                  }
#pragma unroll
                  for (int k = 0; k < B; ++k)
                    if (k0 + k < K && k0 + k < kd) turn(k0 + k < K ? k0 + k : 0, a[k], b[k]);
                }
                v = warp_sum3ff(ff_from(ax), ff_from(ay), FF{0.0f, 0.0f}, lane);
                if (lane == 0 || lane == 8) sm.r2[1 + 2 * j + (lane >> 3)][warp] = make_float2(v.hi, v.lo);
              }
            }
          }
          ++leaf;
          if (leaf == (1 << depth)) {  // the subtree is full: its last verdict
            __syncthreads();
            if (scalar) decide(leaf - 1);
            __syncthreads();
            if (sm.take) sprop = cur;
            break;
          }
        }
        // -------------------------------------------------------------- combine the subtree (biased)
        // (leaf counts the leaves the subtree took: a stop is seen at the leaf after, before it counts)
        if (element) {
          float ax = 0.0f, ay = 0.0f;
#pragma unroll
          for (int k = 0; k < K; ++k) {
            const int d = tid + 256 * k;
            if (k >= kd) continue;
            const float sv_ = P.e.rsum[row + d] + rss[k];
            P.e.rsum[row + d] = sv_;
            const float ro = P.e.r_l[row + d];
            const float av = dir ? ro : r[k], bv = dir ? r[k] : ro;  // left, right
            const float s = sv_ - 0.5f * (av + bv);
            ax = fmaf(mass(k) * av, s, ax);
            ay = fmaf(mass(k) * bv, s, ay);
          }
          const FF v = warp_sum3ff(ff_from(ax), ff_from(ay), FF{1.0f, 0.0f}, lane);
          if (lane == 0) sm.r2[0][warp] = make_float2(v.hi, v.lo);
          if (lane == 8) sm.r2[1][warp] = make_float2(v.hi, v.lo);
        }
        __syncthreads();
        if (scalar) {
          const double dw = sub_w - tree_w;
          const float x = (float)dw;
          float p = 0.0f;
          if (!(sub_turning || sub_div)) p = fminf(expf(x), 1.0f);
          const bool turn = lane < 2 && ff_le0(sv_fold(sm.r2, lane & 1));
          const bool tree_turning = sub_turning || __any_sync(FULL, turn);
          const bool take = u01f(__shfl_sync(FULL, wd.y, depth)) < p;
          if (take) {
            pe_p = pe_sp;
            energy_p = energy_sp;
          }
          tree_w = logaddexp_diff(tree_w, sub_w, dw, x);
          tree_div = sub_div;
          tree_acc += sub_acc;
          if (lane == 0) {
            sm.tree_take = take;
            sm.tree_more = depth + 1 < max_depth && !tree_turning && !tree_div;
          }
        }
        __syncthreads();
        if (sm.tree_take) prop = sprop;
        depth += 1;
        num_prop += leaf;
        if (!sm.tree_more) break;
      }
      // ---------------------------------------------------------------- end of the transition
      // the scalar warp's results reach the element threads through the rows of the partial sums
      double* const out = reinterpret_cast<double*>(&sm.r2[0][0]);
      if (scalar && lane == 0) {
        out[0] = pe_p;
        out[1] = energy_p;
        out[2] = tree_acc / (double)num_prop;
        out[3] = tree_div ? 1.0 : 0.0;
      }
      __syncthreads();
      if (element) {
        for (int d = tid; d < D; d += 256) P.e.Q[row + d] = zs[sv_pos(d)];  // the last queried position
        const float* znew = prop < 0 ? P.s.z : (prop == 0 ? P.e.z_p : (prop == 1 ? P.e.z_sp : P.e.z_r));
        const float* gnew = prop < 0 ? P.s.z_grad : (prop == 0 ? P.e.g_p : (prop == 1 ? P.e.g_sp : P.e.g_r));
        const int left = sv_end_transition(P, c, tid, out[0], out[1], num_prop, out[2], out[3] != 0.0, znew + row, gnew + row);
        if (tid == 0) sm.iters_left = left;
      }
      __syncthreads();
      iters_left = sm.iters_left;
    }
  }
}

}  // namespace gbn
