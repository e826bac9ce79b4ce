// Per-step force kernel and integrator kernels.
//
// k_forces reproduces forceCalculation (src/forces.cpp:13-171) for a run of subunits per CTA:
//   stretching   BEAD::update_stretching_force (src/bead.cpp:17-23) via EDGE::update_length
//                (src/edge.cpp:35-49)
//   bending      EDGE::update_bending_forces + get_gradS/get_grad0/get_grad1
//                (src/edge.cpp:69-188) over FACE::update_area_normal (src/face.cpp:11-17)
//   pair terms   the neighbour loop of src/forces.cpp:67-145: Debye-Hueckel for charged pairs,
//                then attractive LJ (directed table) or WCA for pairs in different subunits.
//   big beads    forceCalculation_bigbead (src/forces.cpp:174-236) when the system has
//                encapsulation big beads: added to the bead's total in the per-bead phase.
// Forces are evaluated in FP32 from exact integer coordinate differences (force_core.cuh); partial
// sums are combined in 64-bit fixed point (2^-32 units), so the total does not depend on summation
// order.  In MD mode the kernel applies the second half-kick
// (src/bead.h:113-117, src/md.cpp:450-455) in integer arithmetic, reduces kinetic energy and
// momentum exactly (int64), and the last CTA of each system (or k_step_end) runs the Nose-Hoover chain
// (src/md.cpp:456-460, 401-406; src/functions.cpp:33-58) and the centre-of-mass velocity
// (src/md.cpp:505-514).  No FP64 instruction runs per bead: GB300's FP64 rate is a small
// fraction of its FP32 rate, so velocities, forces and positions are 64-bit fixed point and
// FP64 is used only for the per-system thermostat scalars.
#include <cuda_runtime.h>

#include <algorithm>

#include "force_core.cuh"
#include "kernels.cuh"
#include "launch.cuh"
#include "thermostat.cuh"

namespace souffle {

// int64 warp sum with a fixed xor tree (exact, so any order gives the same bits)
__device__ __forceinline__ long long warp_sum_ll(long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Encapsulation big beads (forceCalculation_bigbead, src/forces.cpp:192-227) on one subunit bead
// at high words pi (DH weight wl, diameter sl): for each big bead (those flagged in mask, or all),
// r = big - subunit; screened Coulomb q_big q_j lb e^(-kappa r) / r^2 (kappa + 1/r) times the
// Yukawa size factor, and WCA with hard-core distance shc shifted by delta = (sigma_big +
// sigma_j)/2 - shc; the subunit bead takes minus their sum.  Out of line: it runs only for
// systems with big beads and keeps the force kernel's registers for the common path.
__device__ __noinline__ float3 bigbead_force(const ForceArgs& a, const SysParams& P, int4 pi, float wl, float sl,
                                             float unit, const unsigned int* mask) {
  const float kappa = P.kappa;
  const float delta = 0.5f * (P.bb_sigma + sl) - P.bb_shc;
  const float wc = delta + 1.12246205f * P.bb_shc;
  const float s3 = P.bb_shc * P.bb_shc * P.bb_shc, shc6 = s3 * s3;
  float3 fb = f3(0.f, 0.f, 0.f);
  for (int k = 0; k < P.nbb; k++) {
    if (mask) {  // next big bead within reach of the CTA
      const unsigned int m = mask[k >> 5] >> (k & 31);
      if (!m) {
        k |= 31;
        continue;
      }
      k += __ffs(m) - 1;
      if (k >= P.nbb) break;
    }
    const float3 d = dvec(__ldg(&a.bb_pos32[P.bb0 + k]), pi, unit);
    const float r2 = dot3(d, d);
    const float r = sqrtf(r2);
    float c = 0.f;
    if (wl != 0.f && r2 < P.bb_dh_cut2) c = P.bb_w * wl * __expf(-kappa * r) / r2 * (kappa + 1.0f / r);
    if (r2 < wc * wc) {
      const float x = r - delta;
      const float x3 = x * x * x, s6 = shc6 / (x3 * x3);
      c += 48.0f * s6 * (s6 - 0.5f) / r / x;
    }
    fb = fb - d * c;
  }
  return fb;
}

constexpr int kBBWords = 8;   // per-subunit flags for up to 256 big beads (more: all visited)

// Flags the big beads within reach of each of the CTA's nsub subunits (bit k of mask[s * kBBWords
// ...]): a subunit's beads lie within R of its centre bead (R from the coordinates relative to
// the centre bead, packed by twos), and a big bead farther than R + the reach of every big-bead pair term
// (bb_reach2, with a 1 % margin) acts on none of them.  A warp per subunit; all threads of the
// CTA call it.
__device__ __noinline__ void bigbead_mask(const ForceArgs& a, const SysParams& P, const int4* s_pos,
                                          const float* s_rel, int nsub, int np, float unit, unsigned int* mask) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float reach = sqrtf(P.bb_reach2);
  for (int s = wid; s < nsub; s += nw) {
    float r2 = 0.f;
    for (int l = lane; l < np; l += 32) {
      const float* q = s_rel + 8 * (s * ((np + 1) >> 1) + (l >> 1)) + (l & 1);
      r2 = fmaxf(r2, q[0] * q[0] + q[2] * q[2] + q[4] * q[4]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    const float lim = sqrtf(r2) * 1.01f + reach;
    const int4 c = s_pos[s * np + P.center_local];
    for (int k = lane; k < P.nbb; k += 32) {
      const float3 d = dvec(__ldg(&a.bb_pos32[P.bb0 + k]), c, unit);
      if (dot3(d, d) < lim * lim) atomicOr(&mask[s * kBBWords + (k >> 5)], 1u << (k & 31));
    }
  }
}

// Four int64 sums over the warp: halved among the lanes while they are added (12 exchanges instead
// of 40).  Lane l < 4 returns the total of value warp_sum4_index(l).
__device__ __forceinline__ int warp_sum4_index(int lane) { return 2 * (lane & 1) + ((lane >> 1) & 1); }
__device__ __forceinline__ long long warp_sum4_ll(long long v0, long long v1, long long v2, long long v3) {
  const int lane = threadIdx.x & 31;
  const bool b0 = lane & 1, b1 = lane & 2;
  const long long k0 = (b0 ? v2 : v0) + __shfl_xor_sync(0xffffffffu, b0 ? v0 : v2, 1);
  const long long k1 = (b0 ? v3 : v1) + __shfl_xor_sync(0xffffffffu, b0 ? v1 : v3, 1);
  long long x = (b1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2);
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// The end of a step (mode 1) or of the initial forces (mode 2) for one system, from its kinetic
// energy and momentum sums (2^-32 and 2^-40 units) into its state S in shared memory: warp 0 runs
// the thermostat chain, warp 1 the centre-of-mass velocity.  The caller's barrier ends it.
// chain_pre: warp 0's nhc_pre_warp of this step has run with this result, else ~0.
template <bool kChain64>
__device__ __forceinline__ void step_tail(const ForceArgs& a, const SysParams& P, int sys, SysState& S, const long long* sum,
                                          dfloat* chain_scratch, unsigned int chain_pre = ~0u) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int vcom_warp = nw > 1 ? 1 : 0;
  if (wid == 0) {
    if (lane == 0) {
      S.done = 0;
      S.ke = df_from_fixed(sum[0], 2.3283064365386963e-10f);  // 2^-32
      if (a.mode == 1) S.steps += 1;
      if (P.brownian && a.mode == 1) {  // this step's draws are used: next step's generator state
        S.fran_sum[0] = S.fran_sum[1] = S.fran_sum[2] = 0;
        S.lcg = lcg_mul(S.lcg, P.lcg_step);
      }
    }
    __syncwarp();
    if constexpr (kChain64) {  // FP64 validation variant, one thread
      if (lane == 0) {
        Chain64& c = a.chain64[sys];
        if (!chain64_tail(c, (double)sum[0] * 2.3283064365386963e-10, a.mode == 1, S))  // KE: 2^-32 units
          atomicOr(a.err, kErrNonFinite);
      }
      __syncwarp();
    } else {
      const bool forward = a.mode == 1;
      unsigned int active = chain_pre;
      if (!forward) active = __ballot_sync(0xffffffffu, lane < S.m && nhc_active(S, lane));
      else if (chain_pre == ~0u) active = nhc_pre_warp(S, lane, chain_scratch);
      if (!nhc_post_warp(S, lane, chain_scratch, active, forward)) atomicOr(a.err, kErrNonFinite);
    }
  }
  if (wid == vcom_warp && lane == 0) {
    const long long x = sum[1], y = sum[2], z = sum[3];
    if (a.mode == 1) {
      // mean velocity, removed from every bead before the next kick (src/md.cpp:505-514)
      const double vx = (double)x * S.inv_n, vy = (double)y * S.inv_n, vz = (double)z * S.inv_n;
      S.vcom_fx[0] = __double2ll_rn(vx);
      S.vcom_fx[1] = __double2ll_rn(vy);
      S.vcom_fx[2] = __double2ll_rn(vz);
      S.vsum[0] = x;  // (its magnitude is an output: formed on the host, an FP64 root takes 2 us here)
      S.vsum[1] = y;
      S.vsum[2] = z;
    } else {
      S.vcom_fx[0] = S.vcom_fx[1] = S.vcom_fx[2] = 0;
    }
  }
}

// The end of a step of one system by a whole CTA: the system's state and its sums (cleared for the next
// launch) come into shared memory, step_tail, the state goes back, and the per-bead kick coefficients
// c0 / m follow, one template bead per thread.  smem: the state and the chain's scratch.  wait: called
// between the state, with the part of the chain that needs no sums, and the sums.
template <bool kChain64, class Wait>
__device__ __forceinline__ void step_end(const ForceArgs& a, int sys, unsigned char* smem, long long* s_sum, Wait wait) {
  const int np = a.L.np;
  unsigned long long* acc = reinterpret_cast<unsigned long long*>(a.partial) + 4 * (size_t)sys;
  static_assert(sizeof(SysState) % 16 == 0, "SysState is copied as int4");
  constexpr int kStateVecs = (int)(sizeof(SysState) / 16);
  SysState& S = *reinterpret_cast<SysState*>(smem);
  dfloat* chain_scratch = reinterpret_cast<dfloat*>(smem + sizeof(SysState));  // 3 kMaxChain
  const int4* st_src = reinterpret_cast<const int4*>(a.state + sys);
  int4* st_dst = reinterpret_cast<int4*>(&S);
  for (int q = threadIdx.x; q < kStateVecs; q += blockDim.x) st_dst[q] = __ldcg(st_src + q);  // L2 (coherent), not L1
  __syncthreads();
  unsigned int chain_pre = ~0u;
  if (!kChain64 && a.mode == 1 && threadIdx.x < 32) chain_pre = nhc_pre_warp(S, threadIdx.x, chain_scratch);
  wait();
  if (threadIdx.x < 4) {
    s_sum[threadIdx.x] = (long long)__ldcg(acc + threadIdx.x);
    acc[threadIdx.x] = 0;
  }
  __syncthreads();
  step_tail<kChain64>(a, a.sys[sys], sys, S, s_sum, chain_scratch, chain_pre);
  __syncthreads();
  for (int q = threadIdx.x; q < kStateVecs; q += blockDim.x) reinterpret_cast<int4*>(a.state + sys)[q] = st_dst[q];
  long long* kc = a.kick_c + (size_t)sys * np;
  for (int l = threadIdx.x; l < np; l += blockDim.x) {
    long long c = 0;
    if (!nhc_kick_coefficient(S.kick_c0, a.inv_mass[l], c)) atomicOr(a.err, kErrNonFinite);
    kc[l] = c;
  }
}

// One system per CTA, after a force kernel whose CTAs took several work items.  It starts while that
// kernel ends.
template <bool kChain64>
__global__ void __launch_bounds__(64) k_step_end(ForceArgs a) {
  __shared__ __align__(16) unsigned char smem[sizeof(SysState) + 3 * kMaxChain * sizeof(dfloat)];
  __shared__ long long s_sum[4];
  step_end<kChain64>(a, blockIdx.x, smem, s_sum, [] {
    pdl_wait();
    pdl_launch();
  });
}

// One item per CTA (kRun false), 5 CTAs of 256 threads per SM (<= 51 registers) so that 3-subunit
// work items fit one wave of 152 x 5 CTAs at the 2000-subunit workload.  Items beyond one wave
// (kRun): a wave of CTAs that draw items from a counter, 4 per SM with 64 registers.  The tables are
// then loaded once, the upper warps fetch the next item while the lower ones finish the beads of
// one, an item has three barriers instead of six, and the sums leave the CTA once per run of items of
// one system, not with each item and a fence and a ticket behind them; k_step_end ends the step.
// Those serial stretches were a third of the time: 840,000 beads 160 -> 141 us.
// kChain64: the tail runs the FP64 validation chain (souffle_options.chain_fp64) instead of the
// double-float one; a separate instantiation, so that the default kernel's code is untouched.
template <bool kChain64, bool kRun>
__global__ void __launch_bounds__(256, kRun ? 4 : 5) k_forces(ForceArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TplLayout& L = a.L;
  const int np = L.np;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // a thread's place when an item's beads are fetched: with kRun the upper half of the warps first
  const int fetch = kRun ? 32 * (wid >= (nw >> 1) ? wid - (nw >> 1) : wid + nw - (nw >> 1)) + lane : threadIdx.x;
  // (the tail of a system's last CTA reuses the first region for the system state)
  const ForceSmem m = force_smem(smem, a, nw);
  const float* s_mass = m.tpl_f + L.o_mass;
  __shared__ ForceQueue s_queue;
  __shared__ WorkItem s_work;                       // the item in work, then the next one
  __shared__ int s_next;
  __shared__ long long s_sum[4];                    // kinetic energy and momentum of this CTA's beads
  __shared__ unsigned int s_bbm[16 * kBBWords];     // big beads within reach of each of the item's subunits
  if (threadIdx.x == 0) s_queue = ForceQueue{0, 0, 0, 0};
  if (threadIdx.x < 4) s_sum[threadIdx.x] = 0;
  force_setup(a, m);
  for (int t = threadIdx.x; t < 9 * a.max_sub * np; t += blockDim.x) m.F[t] = 0u;  // the beads' force limbs
  pdl_wait();
  if (kRun && a.mode != 0) pdl_launch();  // (k_step_end, which waits for this kernel's end)
  int sys = -1;
  auto flush = [&]() {  // this CTA's sums of system `sys`: exact int64 adds, order-independent
    unsigned long long* acc = reinterpret_cast<unsigned long long*>(a.partial) + 4 * (size_t)sys;
    if (threadIdx.x < 4) {
      atomicAdd(acc + threadIdx.x, (unsigned long long)s_sum[threadIdx.x]);
      s_sum[threadIdx.x] = 0;
    }
  };
  if (threadIdx.x == 0) s_work = a.work[blockIdx.x];
  __syncthreads();
  for (;;) {
    const WorkItem w = s_work;
    const SysParams& P = a.sys[w.sys];
    const int nbead = w.nsub * np;
    const int bead0 = w.sub_begin * np;  // global index of the first bead
    const float unit = P.unit32;
    const RunBeads bead{bead0};
    force_rows(a, m, bead, nbead, fetch, &s_queue);
    for (int t = fetch; t < nbead; t += blockDim.x) {
      const int4 p = a.pos32[bead0 + t];
      const int s = fast_div(t, a.div_np), l = t - s * np;
      const int4 c = __ldg(&a.pos32[bead0 + s * np + P.center_local]);
      m.pos[t] = p;
      force_rel(m, np, s, l, p, c, __ldg(&a.dh_w[w.sys * np + l]), unit);
    }
    if (w.sys != sys)
      for (int l = fetch; l < np; l += blockDim.x) m.w[l] = __ldg(&a.dh_w[w.sys * np + l]);
    const bool bb_filter = P.nbb > 0 && P.nbb <= 32 * kBBWords && w.nsub <= 16;
    if (bb_filter)  // (CTAs of 64 threads and items of 16 subunits: more words than threads)
      for (int t = threadIdx.x; t < w.nsub * kBBWords; t += blockDim.x) s_bbm[t] = 0u;
    __syncthreads();
    if (w.sys != sys) {
      if (kRun && sys >= 0 && a.mode != 0) flush();
      sys = w.sys;
    }
    if (kRun && wid == nw - 1 && lane == 0) {  // the next item, while the others begin
      // (items are drawn in order, every CTA's last draw past the end: the last of all clears the counter)
      const unsigned int v = atomicAdd(a.ticket, 1u);
      if (v == (unsigned int)a.n_items - 1) *a.ticket = 0;
      s_next = (int)(gridDim.x + v);
      if (s_next < a.n_items) s_work = a.work[s_next];
    }
    force_terms<false, kRun ? 4 : 8>(a, P, m, w, nbead, bead, &s_queue, [] {});
    __syncthreads();
    if (kRun && threadIdx.x == 0) s_queue = ForceQueue{0, 0, 0, 0};
    force_gather<1>(a, m, nbead, bead);
    if (bb_filter) bigbead_mask(a, P, m.pos, m.rel, w.nsub, np, unit, s_bbm);
    __syncthreads();

    // The bead's total force, the second half kick and the kinetic-energy and momentum sums, one
    // thread per bead; nothing here reads what the next item's fetch writes
    const SysState& st = a.state[w.sys];
    const long long delta_fx = st.delta_fx;
    const long long* kick_c = a.kick_c + (size_t)w.sys * np;
    long long ke_acc = 0, px_acc = 0, py_acc = 0, pz_acc = 0;
    const bool bd = P.brownian && a.mode == 1;  // Brownian MD step
    for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
      const int sub = fast_div(t, a.div_np), l = t - sub * np, g = bead0 + t;
      unsigned int* F = m.F + 9 * t;
      long long Fx = limbs_value(F), Fy = limbs_value(F + 3), Fz = limbs_value(F + 6);
      if (kRun)
#pragma unroll
        for (int k = 0; k < 9; k++) F[k] = 0u;
      if (P.nbb) {
        const float3 fb = bigbead_force(a, P, m.pos[t], m.w[l], m.tpl_f[L.o_sigma + l], unit,
                                        bb_filter ? s_bbm + sub * kBBWords : nullptr);
        if (!(isfinite(fb.x) && isfinite(fb.y) && isfinite(fb.z)) ||
            fmaxf(fmaxf(fabsf(fb.x), fabsf(fb.y)), fabsf(fb.z)) > 1.0e9f)
          atomicOr(a.err, kErrNonFinite);
        Fx += f32_to_fx32(fb.x);
        Fy += f32_to_fx32(fb.y);
        Fz += f32_to_fx32(fb.z);
      }
      if (bd) {
        // Brownian: tforce + (fran - mean fran over the system) + fdrag (src/md.cpp:468-494,
        // src/bead.h:147-149)
        const long long N = a.n_beads_total;
        Fx += a.fran[g] - __double2ll_rn((double)st.fran_sum[0] * st.inv_n) + a.fdrag[g];
        Fy += a.fran[N + g] - __double2ll_rn((double)st.fran_sum[1] * st.inv_n) + a.fdrag[N + g];
        Fz += a.fran[2 * N + g] - __double2ll_rn((double)st.fran_sum[2] * st.inv_n) + a.fdrag[2 * N + g];
      }
      a.fx[g] = Fx;
      a.fy[g] = Fy;
      a.fz[g] = Fz;
      if (a.mode == 1 || a.mode == 2) {
        long long vx = a.vx[g], vy = a.vy[g], vz = a.vz[g];
        if (a.mode == 1) {  // v <- v exp(-dt xi/2) + F dt sqrt(expfac)/(2m)  (src/bead.h:113-117)
          const long long c = kick_c[l];
          vx = vx - mul_shr(vx, delta_fx, 62) + mul_shr(Fx, c, 56);
          vy = vy - mul_shr(vy, delta_fx, 62) + mul_shr(Fy, c, 56);
          vz = vz - mul_shr(vz, delta_fx, 62) + mul_shr(Fz, c, 56);
          a.vx[g] = vx;
          a.vy[g] = vy;
          a.vz[g] = vz;
          px_acc += vx;
          py_acc += vy;
          pz_acc += vz;
        }
        const float ux = vel_to_f32(vx), uy = vel_to_f32(vy), uz = vel_to_f32(vz);
        const float v2 = ux * ux + uy * uy + uz * uz;
        if (!(v2 < 1.0e12f)) atomicOr(a.err, kErrNonFinite);  // |v| beyond 1e6: a blown-up run
        ke_acc += f32_to_fx32(0.5f * s_mass[l] * v2);
      }
    }
    if (a.mode != 0 && wid * 32 < nbead) {
      const long long x = warp_sum4_ll(ke_acc, px_acc, py_acc, pz_acc);
      if (lane < 4) atomicAdd(reinterpret_cast<unsigned long long*>(s_sum + warp_sum4_index(lane)), (unsigned long long)x);
    }
    if (!kRun) break;
    if (P.nbb) __syncthreads();  // (the big beads' pass reads the item's positions and weights)
    if (s_next >= a.n_items) break;
  }
  if (a.mode == 0) return;
  __syncthreads();
  if (kRun) {  // k_step_end follows
    flush();
    return;
  }

  // one item per CTA: the last CTA of a system ends its step
  __shared__ bool last;
  if (wid == 0) {
    flush();
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      const unsigned int prev = atomicAdd(&a.state[sys].done, 1u);
      last = (prev == (unsigned int)a.sys_slots[sys].y - 1);
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  step_end<kChain64>(a, sys, smem, s_sum, [] {});
}

// Half-kick and drift of one bead (src/md.cpp:409-414, src/bead.h:72-81,113-117), with the
// pending centre-of-mass velocity subtracted first; integer arithmetic only (x += v dt is an
// exact multiply into the fixed-point box).
__device__ __forceinline__ void drift_bead(int g, int l, long long c, long long delta_fx, long long vcx, long long vcy,
                                           long long vcz, long long dx_fx, const long long* fx, const long long* fy,
                                           const long long* fz, long long* vxp, long long* vyp, long long* vzp,
                                           long long* px, long long* py, long long* pz, int4* pos32) {
  long long vx = vxp[g] - vcx, vy = vyp[g] - vcy, vz = vzp[g] - vcz;
  vx = vx - mul_shr(vx, delta_fx, 62) + mul_shr(fx[g], c, 56);
  vy = vy - mul_shr(vy, delta_fx, 62) + mul_shr(fy[g], c, 56);
  vz = vz - mul_shr(vz, delta_fx, 62) + mul_shr(fz[g], c, 56);
  vxp[g] = vx;
  vyp[g] = vy;
  vzp[g] = vz;
  const long long X = (long long)((unsigned long long)px[g] + (unsigned long long)mul_shr(vx, dx_fx, 40));
  const long long Y = (long long)((unsigned long long)py[g] + (unsigned long long)mul_shr(vy, dx_fx, 40));
  const long long Z = (long long)((unsigned long long)pz[g] + (unsigned long long)mul_shr(vz, dx_fx, 40));
  px[g] = X;
  py[g] = Y;
  pz[g] = Z;
  pos32[g] = make_int4(hi_word(X), hi_word(Y), hi_word(Z), l);
}

// Drag and random force of one bead for a Brownian step (src/md.cpp:415-421, 461-467), from its
// velocity after the last centre-of-mass removal and the generator's state before the step: bead k
// of the system takes draws 6k+1 .. 6k+6 (x, y, z: two draws each).  Both are stored for the force
// kernel; r returns the random force.
__device__ __forceinline__ void brownian_drag(const DriftArgs& a, int sys, int g, int l, long long vx, long long vy, long long vz) {
  const long long N = a.n_total;
  const long long dc = a.bd_drag[(size_t)sys * a.np + l];
  a.fdrag[g] = -mul_shr(vx, dc, 48);
  a.fdrag[N + g] = -mul_shr(vy, dc, 48);
  a.fdrag[2 * N + g] = -mul_shr(vz, dc, 48);
}
// component k of bead g's random force alone
__device__ __forceinline__ long long brownian_draw(const DriftArgs& a, const SysParams& P, unsigned int lcg, int sys, int g, int l,
                                                   int k) {
  unsigned int x = lcg_mul(lcg_mul(lcg, a.lcg_table[g - P.bead0]), 16807u);
  for (int i = 0; i < 2 * k; i++) x = lcg_mul(x, 16807u);
  const double sc = a.bd_noise[(size_t)sys * a.np + l];
  const long long r = __double2ll_rn(__dmul_rn(sc, lcg_uniform_half(x, lcg_mul(x, 16807u))) * 4294967296.0);
  a.fran[k * (long long)a.n_total + g] = r;
  return r;
}
__device__ __forceinline__ void brownian_draws(const DriftArgs& a, const SysParams& P, unsigned int lcg, int sys, int g, int l,
                                               long long vx, long long vy, long long vz, long long* r) {
  const long long N = a.n_total;
  brownian_drag(a, sys, g, l, vx, vy, vz);
  unsigned int x = lcg_mul(lcg, a.lcg_table[g - P.bead0]);
  unsigned int d[6];
#pragma unroll
  for (int k = 0; k < 6; k++) d[k] = x = lcg_mul(x, 16807u);
  const double sc = a.bd_noise[(size_t)sys * a.np + l];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    r[k] = __double2ll_rn(__dmul_rn(sc, lcg_uniform_half(d[2 * k], d[2 * k + 1])) * 4294967296.0);
    a.fran[k * N + g] = r[k];
  }
}

// A bead's three force components kept in the first six words of its limbs between steps.
__device__ __forceinline__ void put_fx(unsigned int* F, long long x, long long y, long long z) {
  F[0] = (unsigned int)x;
  F[1] = (unsigned int)(x >> 32);
  F[2] = (unsigned int)y;
  F[3] = (unsigned int)(y >> 32);
  F[4] = (unsigned int)z;
  F[5] = (unsigned int)(z >> 32);
}
__device__ __forceinline__ void get_fx(const unsigned int* F, long long& x, long long& y, long long& z) {
  x = (long long)((unsigned long long)F[1] << 32 | F[0]);
  y = (long long)((unsigned long long)F[3] << 32 | F[2]);
  z = (long long)((unsigned long long)F[5] << 32 | F[4]);
}

__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// First half-kick and drift with periodic wrap (src/md.cpp:409-414, src/bead.h:72-81,113-117),
// with the pending centre-of-mass velocity of the previous step subtracted first.  Integer
// arithmetic only: x += v dt is an exact multiply into the fixed-point box.
__global__ void __launch_bounds__(256) k_drift(DriftArgs a) {
  const WorkItem w = a.work[blockIdx.x];
  const SysParams& P = a.sys[w.sys];
  SysState& S = a.state[w.sys];
  pdl_wait();
  pdl_launch();
  const long long delta_fx = S.delta_fx;
  const long long vcx = S.vcom_fx[0], vcy = S.vcom_fx[1], vcz = S.vcom_fx[2];
  const long long dx_fx = P.drift_fx;
  const long long* kick_c = a.kick_c + (size_t)w.sys * a.np;
  const int n = w.nsub * a.np;
  const int bead0 = w.sub_begin * a.np;
  const int half = blockDim.x >> 1;
  if (P.brownian) {
    // Brownian step, first half (src/md.cpp:415-421): drag -m v / damp from the velocity after
    // the last centre-of-mass removal, half-kick with the stored total force, drift; then this
    // step's random forces (src/md.cpp:461-467): bead k of the system takes draws 6k+1 .. 6k+6
    // of the generator after the previous steps' draws (x, y, z: two draws each)
    long long sx = 0, sy = 0, sz = 0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
      const int g = bead0 + t, l = t % a.np;
      long long r[3];
      brownian_draws(a, P, S.lcg, w.sys, g, l, a.vx[g] - vcx, a.vy[g] - vcy, a.vz[g] - vcz, r);
      drift_bead(g, l, kick_c[l], 0, vcx, vcy, vcz, dx_fx, a.fx, a.fy, a.fz, a.vx, a.vy, a.vz, a.px, a.py, a.pz,
                 a.pos32);
      sx += r[0];
      sy += r[1];
      sz += r[2];
    }
    sx = warp_sum_ll(sx);
    sy = warp_sum_ll(sy);
    sz = warp_sum_ll(sz);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(reinterpret_cast<unsigned long long*>(&S.fran_sum[0]), (unsigned long long)sx);
      atomicAdd(reinterpret_cast<unsigned long long*>(&S.fran_sum[1]), (unsigned long long)sy);
      atomicAdd(reinterpret_cast<unsigned long long*>(&S.fran_sum[2]), (unsigned long long)sz);
    }
    return;
  }
  if (a.inter_ids && n <= half && (int)threadIdx.x >= half) {
    // Idle half of the CTA: bring into L2 what k_forces of this work item reads next step, the
    // used part of each bead's inter-subunit row and the subunits' intra-pair masks (cold after
    // anything has evicted L2 since the last step).
    const int k0 = threadIdx.x - half;
    for (int t = k0; t < n; t += half) {
      const int g = bead0 + t;
      const int cnt = a.inter_count[g];
      const char* row = reinterpret_cast<const char*>(a.inter_ids + (size_t)g * a.inter_cap);
      for (int off = 0; off < cnt * 4; off += 128) prefetch_l2(row + off);
    }
    const char* mk = reinterpret_cast<const char*>(a.intra_mask + (size_t)bead0 * a.words);
    for (int off = k0 * 128; off < n * a.words * 4; off += half * 128) prefetch_l2(mk + off);
    return;
  }
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int l = t % a.np;
    drift_bead(bead0 + t, l, kick_c[l], delta_fx, vcx, vcy, vcz, dx_fx, a.fx, a.fy, a.fz, a.vx, a.vy, a.vz, a.px, a.py,
               a.pz, a.pos32);
  }
}

// Deals a system's subunits to the window kernel's CTAs after a rebuild, so that crowded ones do not
// meet: every CTA of a step waits for the one with the most inter-subunit pairs, and subunits differ
// (2,000 of them, a tenth in contact: 94 pairs on average, 1,600 at most; runs of three: 3,150).  A
// warp per subunit sums its list lengths; the last CTA sorts the subunits by them (counting sort, most
// first) and deals them out in rounds, back and forth, the first round starting at the items with the
// fewest places.  Any order gives the same bits.  100 steps 3,526 -> 3,192 us.
__global__ void __launch_bounds__(1024) k_deal(DealArgs a) {
  __shared__ int s_bin[kDealBins], s_warp[kDealBins / 32];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int sub = blockIdx.x * 32 + wid;
  if (sub < a.n_sub) {
    int n = 0;
    for (int l = lane; l < a.np; l += 32) n += __ldg(a.inter_count + (size_t)sub * a.np + l);
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) a.key[sub] = kDealBins - 1 - min(n / kDealPairs, kDealBins - 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    if (s_last) *a.ticket = 0u;
  }
  if (threadIdx.x < kDealBins) s_bin[threadIdx.x] = 0;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int s = threadIdx.x; s < a.n_sub; s += blockDim.x) atomicAdd(&s_bin[__ldcg(a.key + s)], 1);
  __syncthreads();
  int mine = 0, incl = 0;
  if (threadIdx.x < kDealBins) {
    incl = mine = s_bin[threadIdx.x];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[wid] = incl;
  }
  __syncthreads();
  if (threadIdx.x < kDealBins) {
    int off = incl - mine;
    for (int k = 0; k < wid; k++) off += s_warp[k];
    s_bin[threadIdx.x] = off;
  }
  __syncthreads();
  const int per = a.n_sub / a.items, more = a.n_sub - per * a.items;  // items of per + 1 subunits first
  for (int s = threadIdx.x; s < a.n_sub; s += blockDim.x) {
    const int rank = atomicAdd(&s_bin[__ldcg(a.key + s)], 1);
    const int round = rank / a.items, k = rank - round * a.items;
    const int item = round < per && !(round & 1) ? a.items - 1 - k : k;
    a.deal[item * per + min(item, more) + round] = s;
  }
}

// ---- the window kernel ------------------------------------------------------------------------
// A run of MD or Brownian steps between two pair-list rebuilds in one launch, for handles whose
// work items all fit the GPU at once (one CTA per item, cooperative launch).  The CTA keeps its
// beads' positions, velocities and forces, the template tables and the system's thermostat state
// in shared memory; only the high words of the positions pass through global memory.  A step is
//   drift      own beads; publish the new high words and count the arrival
//   terms      own subunits' rows, quads and edges, then (the others having long arrived) the
//              inter-subunit pairs
//   finish     totals, second half kick, kinetic energy and momentum; send the sums and wait for
//              the others'; every CTA runs the thermostat chain itself, which costs the same
//              3 us once per SM instead of in one CTA, and saves handing its result around
// The same operations as k_drift and k_forces, so the results are the same bits.  What it removes
// is latency, which is all a small system's step consists of: two launches per step, the reload of
// tables, state and tile (about 3 us), and the serial hand-over to the last CTA.  Per step, rebuilds
// included and no subunits in contact: 19.6 -> 10.2 us at 200 beads, 23.3 -> 11.9 at 2,688, 24.8 ->
// 14.5 at 13,986, 36.2 -> 25.6 at 84,000.  What is left there: the chain (2.7 us), the two waits (1.2
// us) and, with subunits in contact, the wait for the CTA with the most pairs.
// A step has two waits, both among the CTAs of one system.  The first (positions published) counts
// arrivals behind a fence.  The second needs none: the sums themselves count.  A sum's 64 bits are
// added as two words of 32 with 1 << kSumCount on top, so whoever reads as many counts as the system
// has CTAs reads complete sums, one trip through L2 after they were sent (with a fence and a counter
// behind them, two: 20 subunits 1,256 -> 1,196 us per 100 steps, 333 Brownian ones 1,242 -> 1,172 per
// 50).  A CTA without inter-subunit pairs does not wait at the first; it cannot get further than the
// second, so arrivals of two steps never mix.
constexpr int kSumCount = 50;     // fewer than 2^14 CTAs (kWindowMaxCtas), sums of up to 2^18 32-bit words
constexpr int kWinWords = 16;     // a system's words per step: 8 of sums, 3 of random forces
struct GridBarrier {
  unsigned int* count;    // arrivals, zero between launches
  unsigned int* err;
  unsigned int polls;     // tries of a wait before it gives up
  unsigned int target;    // arrivals that complete the barrier in progress
  // thread 0 of the CTA, after a CTA barrier behind the writes to publish
  __device__ __forceinline__ void arrive() const {
    __threadfence();
    atomicAdd(count, 1u);
  }
  // any thread; false when the wait ran out
  __device__ __forceinline__ bool wait(volatile int* abort_flag) const {
    for (unsigned int i = 0; i < polls; i++) {
      unsigned int v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
      if ((int)(v - target) >= 0) return true;
      if ((i & 255u) == 255u && *abort_flag) return false;
    }
    *abort_flag = 1;
    atomicOr(err, kErrWindow);
    return false;
  }
};

// kWide: 512 threads and 64 registers (two CTAs per SM) instead of 256 and 48, for grids that fit.
template <bool kWide>
__global__ void __launch_bounds__(kWide ? 512 : 256, kWide ? 2 : 5) k_window(ForceArgs a, DriftArgs d, WindowArgs q) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TplLayout& L = a.L;
  const WorkItem w = a.work[blockIdx.x];
  const SysParams& P = a.sys[w.sys];
  const int np = L.np, nbead = w.nsub * np;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const ForceSmem m = force_smem(smem, a, nw);
  // behind the force kernel's shared memory: velocities, kick coefficients, the state, the low words of
  // the positions (the high words are the tile's)
  const int nmax = a.max_sub * np;
  long long* s_v = reinterpret_cast<long long*>(smem + q.force_bytes);  // [3][nmax]
  long long* s_kc = s_v + ((3 * nmax + 1) & ~1);                        // [np] (16-byte aligned, as the state)
  dfloat* s_im = reinterpret_cast<dfloat*>(s_kc + ((np + 1) & ~1));     // [np] 1 / m
  SysState& S = *reinterpret_cast<SysState*>(s_im + ((np + 1) & ~1));
  dfloat* chain_scratch = reinterpret_cast<dfloat*>(&S + 1);
  unsigned int* s_lo = reinterpret_cast<unsigned int*>(chain_scratch + 3 * kMaxChain);  // [3][nmax]
  int* s_first = reinterpret_cast<int*>(s_lo + 3 * nmax);                               // [max_sub]
  const auto bead = [&] {  // (wide grids are one subunit per item, or asked for: nothing to deal)
    if constexpr (kWide) return RunBeads{w.sub_begin * np};
    else return DealtBeads{s_first};
  }();
  // (high words are rounded, so the low ones are signed offsets from them)
  auto whole = [](int hi, unsigned int lo) {
    return (long long)(((unsigned long long)(unsigned int)hi << 32) + (unsigned long long)(long long)(int)lo);
  };
  __shared__ ForceQueue s_queue;
  __shared__ unsigned int s_active;     // the chain's active links
  __shared__ long long s_draw[3];       // sums of the random forces drawn ahead
  __shared__ int s_abort;
  __shared__ long long s_sum[7];  // kinetic energy, momentum; Brownian: mean random force
  GridBarrier moved{q.count + 1 + w.sys, a.err, q.polls, 0u};  // positions published
  const int n_cta = a.sys_slots[w.sys].y;             // CTAs of the system
  const bool first_cta = w.sub_begin == P.sub0;       // of them, the one with the first subunit
  const float unit = P.unit32;
  const bool bd = P.brownian;
  if (threadIdx.x == 0) {
    // a window queued behind one that gave up leaves at once: the counters stand where that one left them
    s_abort = (*(volatile unsigned int*)a.err & kErrWindow) != 0;
    s_queue = ForceQueue{0, 0, 0, 0};
  }
  for (int s = threadIdx.x; !kWide && s < w.nsub; s += blockDim.x)
    s_first[s] = ((q.deal ? q.deal[w.sub_begin + s] : w.sub_begin + s) - s) * np;
  __syncthreads();
  if (s_abort) return;
  force_rows(a, m, bead, nbead, threadIdx.x, &s_queue);
  force_setup(a, m);
  for (int t = threadIdx.x; t < np; t += blockDim.x) m.w[t] = __ldg(&a.dh_w[w.sys * np + t]);
  {
    const int4* src = reinterpret_cast<const int4*>(a.state + w.sys);
    int4* dst = reinterpret_cast<int4*>(&S);
    for (int t = threadIdx.x; t < (int)(sizeof(SysState) / 16); t += blockDim.x) dst[t] = __ldcg(src + t);
    for (int l = threadIdx.x; l < np; l += blockDim.x) {
      s_kc[l] = a.kick_c[(size_t)w.sys * np + l];
      s_im[l] = a.inv_mass[l];
    }
  }
  const bool own_c = nbead <= (int)blockDim.x;
  long long my_c = 0;
  dfloat inv_m = {0.f, 0.f};
  if (own_c && (int)threadIdx.x < nbead) {
    const int l = threadIdx.x - fast_div(threadIdx.x, a.div_np) * np;
    my_c = a.kick_c[(size_t)w.sys * np + l];
    inv_m = a.inv_mass[l];
  }
  for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
    const int g = bead(fast_div(t, a.div_np), t);
    const long long X = d.px[g], Y = d.py[g], Z = d.pz[g];
    s_lo[t] = (unsigned int)X;
    s_lo[nmax + t] = (unsigned int)Y;
    s_lo[2 * nmax + t] = (unsigned int)Z;
    m.pos[t] = make_int4(hi_word(X), hi_word(Y), hi_word(Z), t - fast_div(t, a.div_np) * np);
    s_v[t] = a.vx[g];
    s_v[nmax + t] = a.vy[g];
    s_v[2 * nmax + t] = a.vz[g];
    unsigned int* F = m.F + 9 * t;
    if (q.forces_first) {  // the first step's drift is done: no forces yet
#pragma unroll
      for (int k = 0; k < 9; k++) F[k] = 0u;
    } else {
      put_fx(F, a.fx[g], a.fy[g], a.fz[g]);
    }
  }
  __syncthreads();
  const float* s_mass = m.tpl_f + L.o_mass;
  bool drawn = false;  // the step's random forces have been drawn in the one before
  for (int step = 0; step < q.steps; step++) {
    unsigned long long* acc = q.acc + (size_t)(step % 3) * q.acc_stride + (size_t)kWinWords * w.sys;
    const bool drift = step > 0 || !q.forces_first;
    // The next step's sums start from zero: their words were last read two steps ago, and every CTA of
    // the system has sent the last step's sums since.  (Seen before this step's sums complete.)
    if (first_cta && threadIdx.x < kWinWords) {
      q.acc[(size_t)((step + 1) % 3) * q.acc_stride + (size_t)kWinWords * w.sys + threadIdx.x] = 0;
      __threadfence();
    }
    if (threadIdx.x == 0) s_queue.next = 0;
    // the part of the chain that needs no sums, by a warp that has no beads (in small systems)
    if (wid == nw - 1) {
      const unsigned int active = nhc_pre_warp(S, lane, chain_scratch);
      if (lane == 0) s_active = active;
    }
    const unsigned int lcg = S.lcg;
    if (drift) {
      long long rx = 0, ry = 0, rz = 0;
      for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
        const int s = fast_div(t, a.div_np), l = t - s * np, g = bead(s, t);
        const long long c = own_c ? my_c : s_kc[l], del = bd ? 0 : S.delta_fx;
        unsigned int* F = m.F + 9 * t;
        long long Fx, Fy, Fz;
        get_fx(F, Fx, Fy, Fz);
        long long vx = s_v[t] - S.vcom_fx[0], vy = s_v[nmax + t] - S.vcom_fx[1], vz = s_v[2 * nmax + t] - S.vcom_fx[2];
        if (bd && drawn) {
          brownian_drag(d, w.sys, g, l, vx, vy, vz);
        } else if (bd) {
          long long r[3];
          brownian_draws(d, P, lcg, w.sys, g, l, vx, vy, vz, r);
          rx += r[0];
          ry += r[1];
          rz += r[2];
        }
        vx = vx - mul_shr(vx, del, 62) + mul_shr(Fx, c, 56);
        vy = vy - mul_shr(vy, del, 62) + mul_shr(Fy, c, 56);
        vz = vz - mul_shr(vz, del, 62) + mul_shr(Fz, c, 56);
        s_v[t] = vx;
        s_v[nmax + t] = vy;
        s_v[2 * nmax + t] = vz;
        const int4 old = m.pos[t];
        const long long X = (long long)((unsigned long long)whole(old.x, s_lo[t]) + (unsigned long long)mul_shr(vx, P.drift_fx, 40));
        const long long Y = (long long)((unsigned long long)whole(old.y, s_lo[nmax + t]) + (unsigned long long)mul_shr(vy, P.drift_fx, 40));
        const long long Z = (long long)((unsigned long long)whole(old.z, s_lo[2 * nmax + t]) + (unsigned long long)mul_shr(vz, P.drift_fx, 40));
        s_lo[t] = (unsigned int)X;
        s_lo[nmax + t] = (unsigned int)Y;
        s_lo[2 * nmax + t] = (unsigned int)Z;
        const int4 p = make_int4(hi_word(X), hi_word(Y), hi_word(Z), l);
        m.pos[t] = p;
        __stcg(&d.pos32[g], p);
#pragma unroll
        for (int k = 0; k < 9; k++) F[k] = 0u;
      }
      if (bd && drawn) {
        if (threadIdx.x < 3) atomicAdd(acc + 8 + threadIdx.x, (unsigned long long)s_draw[threadIdx.x]);
        __threadfence();
      } else if (bd) {
        rx = warp_sum_ll(rx);
        ry = warp_sum_ll(ry);
        rz = warp_sum_ll(rz);
        if (lane == 0 && wid * 32 < nbead) {
          atomicAdd(acc + 8, (unsigned long long)rx);
          atomicAdd(acc + 9, (unsigned long long)ry);
          atomicAdd(acc + 10, (unsigned long long)rz);
        }
        __threadfence();
      }
      moved.target += n_cta;
      __syncthreads();
      if (threadIdx.x == 0) moved.arrive();
    }
    for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
      const int s = fast_div(t, a.div_np), l = t - s * np;
      force_rel(m, np, s, l, m.pos[t], m.pos[s * np + P.center_local], m.w[l], unit);
    }
    __syncthreads();
    force_terms<true, 8>(a, P, m, w, nbead, bead, &s_queue, [&] {
      if (drift) {
        if (lane == 0) moved.wait(&s_abort);
        __syncwarp();
      }
    });
    if (bd) {  // the step's random forces: their sum over the system
      if (threadIdx.x < 3) {
        s_draw[threadIdx.x] = 0;  // (sent before this step's first wait)
        if (drift) {
          moved.wait(&s_abort);
          s_sum[4 + threadIdx.x] = (long long)__ldcg(acc + 8 + threadIdx.x);
        } else {
          s_sum[4 + threadIdx.x] = S.fran_sum[threadIdx.x];
        }
        s_sum[4 + threadIdx.x] = __double2ll_rn((double)s_sum[4 + threadIdx.x] * S.inv_n);  // mean
      }
    }
    __syncthreads();
    if (s_abort) return;  // uniform: nothing sets it between the barrier and here but a failed wait
    force_gather<kWide ? 4 : 1>(a, m, nbead, bead);
    __syncthreads();
    long long ke_acc = 0, px_acc = 0, py_acc = 0, pz_acc = 0;
    for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
      const int s = fast_div(t, a.div_np), l = t - s * np, g = bead(s, t);
      unsigned int* F = m.F + 9 * t;
      long long Fx = limbs_value(F), Fy = limbs_value(F + 3), Fz = limbs_value(F + 6);
      if (bd) {
        const long long N = a.n_beads_total;
        Fx += a.fran[g] - s_sum[4] + a.fdrag[g];
        Fy += a.fran[N + g] - s_sum[5] + a.fdrag[N + g];
        Fz += a.fran[2 * N + g] - s_sum[6] + a.fdrag[2 * N + g];
      }
      put_fx(F, Fx, Fy, Fz);
      const long long c = own_c ? my_c : s_kc[l], del = S.delta_fx;
      long long vx = s_v[t], vy = s_v[nmax + t], vz = s_v[2 * nmax + t];
      vx = vx - mul_shr(vx, del, 62) + mul_shr(Fx, c, 56);
      vy = vy - mul_shr(vy, del, 62) + mul_shr(Fy, c, 56);
      vz = vz - mul_shr(vz, del, 62) + mul_shr(Fz, c, 56);
      s_v[t] = vx;
      s_v[nmax + t] = vy;
      s_v[2 * nmax + t] = vz;
      px_acc += vx;
      py_acc += vy;
      pz_acc += vz;
      const float ux = vel_to_f32(vx), uy = vel_to_f32(vy), uz = vel_to_f32(vz);
      const float v2 = ux * ux + uy * uy + uz * uz;
      if (!(v2 < 1.0e12f)) atomicOr(a.err, kErrNonFinite);  // |v| beyond 1e6: a blown-up run
      ke_acc += f32_to_fx32(0.5f * s_mass[l] * v2);
    }
    // the CTA's sums by its working warps, then the system's
    if (wid * 32 < nbead) {
      const long long x = warp_sum4_ll(ke_acc, px_acc, py_acc, pz_acc);
      if (lane < 4) m.red[wid * 4 + warp_sum4_index(lane)] = x;
    }
    __syncthreads();
    unsigned int chain_pre = 0;
    if (wid == 0) {
      if (lane < 8) {
        long long x = 0;
        for (int k = 0; k < nw && k * 32 < nbead; k++) x += m.red[4 * k + (lane >> 1)];
        const unsigned long long part = lane & 1 ? (unsigned long long)((x >> 32) + 2147483648ll) : (unsigned long long)(unsigned int)x;
        atomicAdd(acc + lane, (1ull << kSumCount) + part);
      }
      chain_pre = s_active;
      unsigned long long v = 0;
      bool done = false;
      for (unsigned int i = 0; i < q.polls; i++) {
        if (lane < 8) asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(acc + lane) : "memory");
        done = __all_sync(0xffffffffu, lane >= 8 || (v >> kSumCount) == (unsigned long long)n_cta);
        if (done || ((i & 255u) == 255u && *(volatile int*)&s_abort)) break;
      }
      if (!done && lane == 0) {
        s_abort = 1;
        atomicOr(a.err, kErrWindow);
      }
      v &= (1ull << kSumCount) - 1;
      const unsigned long long hi = __shfl_down_sync(0xffffffffu, v, 1) - ((unsigned long long)n_cta << 31);
      if (lane < 8 && !(lane & 1)) s_sum[lane >> 1] = (long long)(v + (hi << 32));
    } else if (bd && step + 1 < q.steps) {
      // Meanwhile the other warps draw the next step's random forces (this step's are used up), a
      // component per thread: their FP64 operations took 8,000 cycles before each drift.
      const unsigned int next = lcg_mul(lcg, P.lcg_step);
      long long r[3] = {0, 0, 0};
      for (int u = threadIdx.x - 32; u < 3 * nbead; u += blockDim.x - 32) {
        const int k = u >= 2 * nbead ? 2 : u >= nbead ? 1 : 0, t = u - k * nbead;
        const int s = fast_div(t, a.div_np), l = t - s * np;
        const long long f = brownian_draw(d, P, next, w.sys, bead(s, t), l, k);
        if (k == 0) r[0] += f;
        else if (k == 1) r[1] += f;
        else r[2] += f;
      }
      const long long x = warp_sum4_ll(r[0], r[1], r[2], 0);
      if (lane < 4 && warp_sum4_index(lane) < 3)
        atomicAdd(reinterpret_cast<unsigned long long*>(s_draw + warp_sum4_index(lane)), (unsigned long long)x);
    }
    __syncthreads();
    if (s_abort) return;
    drawn = bd && nw > 1 && step + 1 < q.steps;
    step_tail<false>(a, P, w.sys, S, s_sum, chain_scratch, chain_pre);
    __syncthreads();
    // the next kicks' coefficients: a thread's only bead's stays in its register
    if (own_c) {
      if ((int)threadIdx.x < nbead && !nhc_kick_coefficient(S.kick_c0, inv_m, my_c)) atomicOr(a.err, kErrNonFinite);
    } else {
      for (int l = threadIdx.x; l < np; l += blockDim.x) {
        long long c = 0;
        if (!nhc_kick_coefficient(S.kick_c0, s_im[l], c)) atomicOr(a.err, kErrNonFinite);
        s_kc[l] = c;
      }
      __syncthreads();
    }
  }
  if (own_c) {
    if ((int)threadIdx.x < np) s_kc[threadIdx.x] = my_c;  // (np <= nbead: the first subunit's beads)
    __syncthreads();
  }
  // results back to global memory
  for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
    const int g = bead(fast_div(t, a.div_np), t);
    const int4 p = m.pos[t];
    d.px[g] = whole(p.x, s_lo[t]);
    d.py[g] = whole(p.y, s_lo[nmax + t]);
    d.pz[g] = whole(p.z, s_lo[2 * nmax + t]);
    a.vx[g] = s_v[t];
    a.vy[g] = s_v[nmax + t];
    a.vz[g] = s_v[2 * nmax + t];
    long long Fx, Fy, Fz;
    get_fx(m.F + 9 * t, Fx, Fy, Fz);
    a.fx[g] = Fx;
    a.fy[g] = Fy;
    a.fz[g] = Fz;
  }
  if (first_cta) {
    int4* dst = reinterpret_cast<int4*>(a.state + w.sys);
    const int4* src = reinterpret_cast<const int4*>(&S);
    for (int t = threadIdx.x; t < (int)(sizeof(SysState) / 16); t += blockDim.x) dst[t] = src[t];
    for (int l = threadIdx.x; l < np; l += blockDim.x) a.kick_c[(size_t)w.sys * np + l] = s_kc[l];
  }
  // the last CTA to leave clears the counters and sums for the next launch
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(q.count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (s_last) {
    for (int k = threadIdx.x; k < (int)(3 * q.acc_stride); k += blockDim.x) q.acc[k] = 0;
    for (int k = threadIdx.x; k < q.n_sys; k += blockDim.x) q.count[1 + k] = 0u;
    if (threadIdx.x == 0) {
      q.count[0] = 0u;
    }
  }
}

// Host state in: double positions to 64-bit fixed point, the high-word copy, velocities to
// 2^-40 fixed point.
__global__ void k_state_in(StateArgs a) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.n) return;
  const SysParams& P = a.sys[a.bead_sys[g]];
  const double invL = 1.0 / P.box;
  long long X = fixed_from_fraction(a.pos_in[3 * g] * invL);
  long long Y = fixed_from_fraction(a.pos_in[3 * g + 1] * invL);
  long long Z = fixed_from_fraction(a.pos_in[3 * g + 2] * invL);
  a.px[g] = X;
  a.py[g] = Y;
  a.pz[g] = Z;
  a.pos32[g] = make_int4(hi_word(X), hi_word(Y), hi_word(Z), g % a.np);
  if (a.vel_in) {
    a.vx[g] = __double2ll_rn(a.vel_in[3 * g] * kVelScale);
    a.vy[g] = __double2ll_rn(a.vel_in[3 * g + 1] * kVelScale);
    a.vz[g] = __double2ll_rn(a.vel_in[3 * g + 2] * kVelScale);
  } else {
    a.vx[g] = a.vy[g] = a.vz[g] = 0;
  }
}

// Device state out, with any pending COM velocity subtracted (what the reference holds after
// src/md.cpp:513-514); optionally the force in double.
__global__ void k_state_out(StateArgs a) {
  int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= a.n) return;
  const int sy = a.bead_sys[g];
  const SysParams& P = a.sys[sy];
  const SysState& S = a.state[sy];
  const double inv = 1.0 / kTwo32;
  if (a.pos_out) {
    a.pos_out[3 * g] = (double)a.px[g] * P.fx_to_len;
    a.pos_out[3 * g + 1] = (double)a.py[g] * P.fx_to_len;
    a.pos_out[3 * g + 2] = (double)a.pz[g] * P.fx_to_len;
  }
  if (a.vel_out) {
    const double iv = 1.0 / kVelScale;
    a.vel_out[3 * g] = (double)(a.vx[g] - S.vcom_fx[0]) * iv;
    a.vel_out[3 * g + 1] = (double)(a.vy[g] - S.vcom_fx[1]) * iv;
    a.vel_out[3 * g + 2] = (double)(a.vz[g] - S.vcom_fx[2]) * iv;
  }
  if (a.force_out) {
    a.force_out[3 * g] = (double)a.fx_in[g] * inv;
    a.force_out[3 * g + 1] = (double)a.fy_in[g] * inv;
    a.force_out[3 * g + 2] = (double)a.fz_in[g] * inv;
  }
  const long long N = a.n;
  for (int k = 0; k < 2; k++) {  // the parts, when asked for
    double* out = k == 0 ? a.sforce_out : a.bforce_out;
    if (!out) continue;
    const float* in = a.sb_in + 3 * k * N + g;
    out[3 * g] = (double)in[0];
    out[3 * g + 1] = (double)in[N];
    out[3 * g + 2] = (double)in[2 * N];
  }
}

}  // namespace souffle

namespace souffle {
// Where CTAs draw items, the kernels of a step start while the one before them ends: the force kernel loads
// its tables, k_step_end the state and the part of the chain that needs no sums (840,000 beads 7,369 ->
// 7,143 us per 40 steps, 64 replicas 5,586 -> 5,504 per 20).  A step of one wave of CTAs is 2 % slower
// that way (84,000 beads, L2 flushed before each step: 44.6 against 43.6 us).
void launch_forces(const ForceArgs& a, int n_sys, int grid, int block, size_t smem, cudaStream_t s) {
  if (grid == a.n_items) {
    if (a.chain64)
      k_forces<true, false><<<grid, block, smem, s>>>(a);
    else
      k_forces<false, false><<<grid, block, smem, s>>>(a);
    return;
  }
  launch_pdl(a.chain64 ? k_forces<true, true> : k_forces<false, true>, grid, block, smem, s, a);
  if (a.mode != 0) launch_pdl(a.chain64 ? k_step_end<true> : k_step_end<false>, n_sys, 64, 0, s, a);
}
void launch_drift(const DriftArgs& a, bool overlap, int grid, int block, cudaStream_t s) {
  if (overlap)
    launch_pdl(k_drift, grid, block, 0, s, a);
  else
    k_drift<<<grid, block, 0, s>>>(a);
}
// shared memory of k_window: the force kernel's, then per-bead state, kick coefficients, system state
size_t window_smem_bytes(size_t force_bytes, int subs, int np) {
  const size_t vel = (3 * (size_t)subs * np + 1) & ~(size_t)1;
  return ((force_bytes + 15) & ~(size_t)15) + sizeof(long long) * (vel + 2 * (size_t)((np + 1) & ~1)) +
         sizeof(SysState) + 3 * kMaxChain * sizeof(dfloat) + sizeof(unsigned int) * (3 * (size_t)subs * np + subs);
}
cudaError_t launch_window(const ForceArgs& a, const DriftArgs& d, const WindowArgs& q, int grid, int block, size_t smem,
                          cudaStream_t s) {
  void* args[] = {const_cast<ForceArgs*>(&a), const_cast<DriftArgs*>(&d), const_cast<WindowArgs*>(&q)};
  return cudaLaunchCooperativeKernel(q.wide ? (const void*)k_window<true> : (const void*)k_window<false>, dim3(grid), dim3(block),
                                     args, smem, s);
}
cudaError_t window_wave_ctas(bool wide, int threads, size_t smem, int* ctas) {
  *ctas = 0;
  const void* fn = wide ? (const void*)k_window<true> : (const void*)k_window<false>;
  cudaError_t e = raise_smem_limit(fn, smem);
  if (e != cudaSuccess) return e;
  if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100)) != cudaSuccess) return e;
  int per_sm = 0, dev = 0, sms = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem)) != cudaSuccess) return e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  *ctas = per_sm * sms;
  return cudaSuccess;
}
void launch_deal(const DealArgs& a, cudaStream_t s) { k_deal<<<(a.n_sub + 31) / 32, 1024, 0, s>>>(a); }
void launch_state_in(const StateArgs& a, int grid, int block, cudaStream_t s) {
  k_state_in<<<grid, block, 0, s>>>(a);
}
void launch_state_out(const StateArgs& a, int grid, int block, cudaStream_t s) {
  k_state_out<<<grid, block, 0, s>>>(a);
}
namespace {
// Ask for a shared-memory carveout that holds as many force CTAs as the registers allow (the
// default may be smaller, which splits a one-wave grid into two waves).
template <class Kernel>
cudaError_t set_force_smem(Kernel* fn, size_t smem, int threads, int regs_sm, int smem_sm) {
  cudaError_t e = raise_smem_limit((const void*)fn, smem);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa{};
  if ((e = cudaFuncGetAttributes(&fa, fn)) != cudaSuccess) return e;
  const int warp_regs = ((fa.numRegs * 32 + 255) / 256) * 256;
  const int ctas = regs_sm / (warp_regs * ((threads + 31) / 32));
  const size_t need = (size_t)ctas * (smem + fa.sharedSizeBytes + 1024);
  const int percent = (int)std::min<size_t>(100, (need * 100 + smem_sm - 1) / (size_t)smem_sm);
  return cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, percent);
}
}  // namespace

cudaError_t set_kernel_smem(size_t force_smem, int force_threads, size_t pair_smem) {
  cudaError_t e;
  int dev = 0, regs_sm = 0, smem_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess) return e;
  if ((e = set_force_smem(k_forces<false, false>, force_smem, force_threads, regs_sm, smem_sm)) != cudaSuccess ||
      (e = set_force_smem(k_forces<false, true>, force_smem, force_threads, regs_sm, smem_sm)) != cudaSuccess ||
      (e = set_force_smem(k_forces<true, false>, force_smem, force_threads, regs_sm, smem_sm)) != cudaSuccess ||
      (e = set_force_smem(k_forces<true, true>, force_smem, force_threads, regs_sm, smem_sm)) != cudaSuccess)
    return e;
  return set_pairs_smem(pair_smem);
}

// CTAs of the force kernel resident at once: one item each, or (run) drawing items
cudaError_t force_wave_ctas(bool run, int threads, size_t smem, int* ctas) {
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t e = run ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_forces<false, true>, threads, smem)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_forces<false, false>, threads, smem);
  if (e != cudaSuccess) return e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  *ctas = per_sm * sms;
  return cudaSuccess;
}
}  // namespace souffle
