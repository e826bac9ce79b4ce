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
// momentum exactly (int64), and the last CTA of each system runs the Nose-Hoover chain
// (src/md.cpp:456-460, 401-406; src/functions.cpp:33-58) and the centre-of-mass velocity
// (src/md.cpp:505-514).  No FP64 instruction runs per bead: GB300's FP64 rate is a small
// fraction of its FP32 rate, so velocities, forces and positions are 64-bit fixed point and
// FP64 is used only for the per-system thermostat scalars.
#include <cuda_runtime.h>

#include <algorithm>

#include "force_core.cuh"
#include "kernels.cuh"
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

// 5 CTAs of 256 threads per SM (<= 51 registers) so 3-subunit work items fit one wave of
// 152 x 5 CTAs at the 2000-subunit workload.
// kChain64: the tail runs the FP64 validation chain (souffle_options.chain_fp64) instead of the
// double-float one; a separate instantiation, so that the default kernel's code is untouched.
template <bool kChain64>
__global__ void __launch_bounds__(256, 5) k_forces(ForceArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const TplLayout& L = a.L;
  const WorkItem w = a.work[blockIdx.x];
  const SysParams& P = a.sys[w.sys];
  const int np = L.np;
  const int nbead = w.nsub * np;
  const int bead0 = w.sub_begin * np;  // global index of the first bead
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // (the tail of the system's last CTA reuses the first region for the system state)
  const ForceSmem m = force_smem(smem, a, nw);
  int4* s_pos = m.pos;
  long long* s_red = m.red;
  unsigned int* s_F = m.F;
  const float* tpl_f = m.tpl_f;
  const float* s_w = m.w;
  const float unit = P.unit32;
  __shared__ int s_counter;
  if (threadIdx.x == 0) s_counter = 0;
  force_setup(a, w, m);
  for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
    const int4 p = a.pos32[bead0 + t];
    const int s = fast_div(t, a.div_np), l = t - s * np;
    const int4 c = __ldg(&a.pos32[bead0 + s * np + P.center_local]);
    s_pos[t] = p;
    force_rel(m, np, s, l, p, c, __ldg(&a.dh_w[w.sys * np + l]), unit);
  }
  for (int t = threadIdx.x; t < 9 * nbead; t += blockDim.x) s_F[t] = 0u;  // the beads' force limbs
  // big beads within reach of each of the CTA's subunits (s_bbm), flagged before phase 3
  __shared__ unsigned int s_bbm[16 * kBBWords];
  const bool bb_filter = P.nbb > 0 && P.nbb <= 32 * kBBWords && w.nsub <= 16;
  if (threadIdx.x < 16 * kBBWords) s_bbm[threadIdx.x] = 0u;
  force_prefix(a, m, bead0, nbead);  // (its barrier makes the tile visible)
  __syncthreads();               // the prefix sums
  force_terms<false>(a, P, m, w, nbead, bead0, &s_counter);
  __syncthreads();
  const float* s_mass = tpl_f + L.o_mass;
  const SysState& st = a.state[w.sys];
  const long long delta_fx = st.delta_fx;
  const long long* kick_c = a.kick_c + (size_t)w.sys * np;
  long long ke_acc = 0, px_acc = 0, py_acc = 0, pz_acc = 0;
  const bool bd = P.brownian && a.mode == 1;  // Brownian MD step
  force_gather(a, m, nbead, bead0);
  if (bb_filter) bigbead_mask(a, P, s_pos, m.rel, w.nsub, np, unit, s_bbm);
  __syncthreads();

  // Phase 3: the bead's total force, the second half kick and the kinetic-energy and momentum
  // sums, one thread per bead
  for (int t = threadIdx.x; t < nbead; t += blockDim.x) {
    const int sub = fast_div(t, a.div_np), l = t - sub * np, g = bead0 + t;
    long long Fx = limbs_value(s_F + 9 * t), Fy = limbs_value(s_F + 9 * t + 3), Fz = limbs_value(s_F + 9 * t + 6);
    if (P.nbb) {
      const float3 fb = bigbead_force(a, P, s_pos[t], s_w[l], tpl_f[L.o_sigma + l], unit,
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
  if (a.mode == 0) return;

  // exact CTA reduction in int64
  ke_acc = warp_sum_ll(ke_acc);
  px_acc = warp_sum_ll(px_acc);
  py_acc = warp_sum_ll(py_acc);
  pz_acc = warp_sum_ll(pz_acc);
  if (lane == 0) {
    s_red[wid * 4 + 0] = ke_acc;
    s_red[wid * 4 + 1] = px_acc;
    s_red[wid * 4 + 2] = py_acc;
    s_red[wid * 4 + 3] = pz_acc;
  }
  __syncthreads();
  __shared__ bool last;
  // the system's running sums (kinetic energy, momentum) for this launch: exact int64 adds,
  // order-independent; the last CTA reads them and clears them for the next launch
  unsigned long long* acc = reinterpret_cast<unsigned long long*>(a.partial) + 4 * (size_t)w.sys;
  if (threadIdx.x == 0) {
    long long k = 0, x = 0, y = 0, z = 0;
    for (int q = 0; q < nw; q++) {
      k += s_red[q * 4];
      x += s_red[q * 4 + 1];
      y += s_red[q * 4 + 2];
      z += s_red[q * 4 + 3];
    }
    atomicAdd(acc + 0, (unsigned long long)k);
    atomicAdd(acc + 1, (unsigned long long)x);
    atomicAdd(acc + 2, (unsigned long long)y);
    atomicAdd(acc + 3, (unsigned long long)z);
    __threadfence();
    const int2 sl = a.sys_slots[w.sys];
    unsigned int prev = atomicAdd(&a.state[w.sys].done, 1u);
    last = (prev == (unsigned int)sl.y - 1);
  }
  __syncthreads();
  if (!last) return;

  // Last CTA of this system: the running sums and the system's state come into shared memory
  // (the tile area, free by now) in one round of loads; then warp 0 runs the thermostat chain
  // and warp 1 the centre-of-mass velocity.
  __threadfence();
  static_assert(sizeof(SysState) % 16 == 0, "SysState is copied as int4");
  constexpr int kStateVecs = (int)(sizeof(SysState) / 16);
  SysState& S = *reinterpret_cast<SysState*>(smem);
  dfloat* chain_scratch = reinterpret_cast<dfloat*>(smem + sizeof(SysState));  // 3 kMaxChain
  const int4* st_src = reinterpret_cast<const int4*>(a.state + w.sys);
  int4* st_dst = reinterpret_cast<int4*>(&S);
  long long sum = 0;
  if (threadIdx.x < 4) {
    sum = (long long)__ldcg(acc + threadIdx.x);  // L2 (coherent), not L1
    acc[threadIdx.x] = 0;
  }
  for (int q = threadIdx.x; q < kStateVecs; q += blockDim.x) st_dst[q] = __ldcg(st_src + q);
  if (threadIdx.x < 4) s_red[threadIdx.x] = sum;
  __syncthreads();
  const int vcom_warp = nw > 1 ? 1 : 0;
  if (wid == 0) {
    if (lane == 0) {
      S.done = 0;
      S.ke = df_from_fixed(s_red[0], 2.3283064365386963e-10f);  // 2^-32
      if (a.mode == 1) S.steps += 1;
      if (P.brownian && a.mode == 1) {  // this step's draws are used: next step's generator state
        S.fran_sum[0] = S.fran_sum[1] = S.fran_sum[2] = 0;
        S.lcg = lcg_mul(S.lcg, P.lcg_step);
      }
    }
    __syncwarp();
    if constexpr (kChain64) {  // FP64 validation variant, one thread
      if (lane == 0) {
        Chain64& c = a.chain64[w.sys];
        if (!chain64_tail(c, (double)s_red[0] * 2.3283064365386963e-10, a.mode == 1, S))  // KE: 2^-32 units
          atomicOr(a.err, kErrNonFinite);
      }
      __syncwarp();
    } else {
      if (a.mode == 1) nhc_forward_warp(S, lane, chain_scratch);
      if (!nhc_backward_warp(S, lane, chain_scratch + 2 * kMaxChain)) atomicOr(a.err, kErrNonFinite);
    }
  }
  if (wid == vcom_warp && lane == 0) {
    const long long x = s_red[1], y = s_red[2], z = s_red[3];
    if (a.mode == 1) {
      // mean velocity, removed from every bead before the next kick (src/md.cpp:505-514)
      const double vx = (double)x * S.inv_n, vy = (double)y * S.inv_n, vz = (double)z * S.inv_n;
      S.vcom_fx[0] = __double2ll_rn(vx);
      S.vcom_fx[1] = __double2ll_rn(vy);
      S.vcom_fx[2] = __double2ll_rn(vz);
      S.vcom_mag = sqrt(vx * vx + vy * vy + vz * vz) * (1.0 / kVelScale);
    } else {
      S.vcom_fx[0] = S.vcom_fx[1] = S.vcom_fx[2] = 0;
    }
  }
  __syncthreads();
  for (int q = threadIdx.x; q < kStateVecs; q += blockDim.x) reinterpret_cast<int4*>(a.state + w.sys)[q] = st_dst[q];
  // per-bead kick coefficients c0 / m, one template bead per thread
  long long* kc = a.kick_c + (size_t)w.sys * np;
  for (int l = threadIdx.x; l < np; l += blockDim.x) {
    long long c = 0;
    if (!nhc_kick_coefficient(S.kick_c0, a.inv_mass[l], c)) atomicOr(a.err, kErrNonFinite);
    kc[l] = c;
  }
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
    const long long N = a.n_total;
    long long sx = 0, sy = 0, sz = 0;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
      const int g = bead0 + t, l = t % a.np;
      const long long dc = a.bd_drag[(size_t)w.sys * a.np + l];
      const long long vx = a.vx[g] - vcx, vy = a.vy[g] - vcy, vz = a.vz[g] - vcz;
      a.fdrag[g] = -mul_shr(vx, dc, 48);
      a.fdrag[N + g] = -mul_shr(vy, dc, 48);
      a.fdrag[2 * N + g] = -mul_shr(vz, dc, 48);
      drift_bead(g, l, kick_c[l], 0, vcx, vcy, vcz, dx_fx, a.fx, a.fy, a.fz, a.vx, a.vy, a.vz, a.px, a.py, a.pz,
                 a.pos32);
      unsigned int x = lcg_mul(S.lcg, a.lcg_table[g - P.bead0]);
      unsigned int d[6];
#pragma unroll
      for (int k = 0; k < 6; k++) d[k] = x = lcg_mul(x, 16807u);
      const double sc = a.bd_noise[(size_t)w.sys * a.np + l];
      const long long rx = __double2ll_rn(__dmul_rn(sc, lcg_uniform_half(d[0], d[1])) * 4294967296.0);
      const long long ry = __double2ll_rn(__dmul_rn(sc, lcg_uniform_half(d[2], d[3])) * 4294967296.0);
      const long long rz = __double2ll_rn(__dmul_rn(sc, lcg_uniform_half(d[4], d[5])) * 4294967296.0);
      a.fran[g] = rx;
      a.fran[N + g] = ry;
      a.fran[2 * N + g] = rz;
      sx += rx;
      sy += ry;
      sz += rz;
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

// Host state in: double positions to 64-bit fixed point, the high-word copy, velocities to
// 2^-32 fixed point.
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
}

}  // namespace souffle

namespace souffle {
void launch_forces(const ForceArgs& a, int grid, int block, size_t smem, cudaStream_t s) {
  if (a.chain64)
    k_forces<true><<<grid, block, smem, s>>>(a);
  else
    k_forces<false><<<grid, block, smem, s>>>(a);
}
void launch_drift(const DriftArgs& a, int grid, int block, cudaStream_t s) {
  k_drift<<<grid, block, 0, s>>>(a);
}
void launch_state_in(const StateArgs& a, int grid, int block, cudaStream_t s) {
  k_state_in<<<grid, block, 0, s>>>(a);
}
void launch_state_out(const StateArgs& a, int grid, int block, cudaStream_t s) {
  k_state_out<<<grid, block, 0, s>>>(a);
}
cudaError_t set_kernel_smem(size_t force_smem, int force_threads, size_t pair_smem) {
  cudaError_t e = cudaFuncSetAttribute(k_forces<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)force_smem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(k_forces<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)force_smem);
  if (e != cudaSuccess) return e;
  // Ask for a shared-memory carveout that holds as many force CTAs as the registers allow (the
  // default may be smaller, which splits a one-wave grid into two waves).
  cudaFuncAttributes fa{};
  if ((e = cudaFuncGetAttributes(&fa, k_forces<false>)) != cudaSuccess) return e;
  int dev = 0, regs_sm = 0, smem_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess) return e;
  const int warp_regs = ((fa.numRegs * 32 + 255) / 256) * 256;
  const int ctas = regs_sm / (warp_regs * ((force_threads + 31) / 32));
  const size_t need = (size_t)ctas * (force_smem + fa.sharedSizeBytes + 1024);
  const int percent = (int)std::min<size_t>(100, (need * 100 + smem_sm - 1) / (size_t)smem_sm);
  if ((e = cudaFuncSetAttribute(k_forces<false>, cudaFuncAttributePreferredSharedMemoryCarveout, percent)) != cudaSuccess ||
      (e = cudaFuncSetAttribute(k_forces<true>, cudaFuncAttributePreferredSharedMemoryCarveout, percent)) != cudaSuccess)
    return e;
  return set_pairs_smem(pair_smem);
}

cudaError_t force_wave_ctas(int threads, size_t smem, int* ctas) {
  int per_sm = 0, dev = 0, sms = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_forces<false>, threads, smem);
  if (e != cudaSuccess) return e;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  *ctas = per_sm * sms;
  return cudaSuccess;
}
}  // namespace souffle
