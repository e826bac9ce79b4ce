// Energy block of run_simulation (src/md.cpp:553-605), evaluated in FP64.
//
//   k_energy_sub      the bonded terms (BEAD::update_stretching_energy, src/bead.cpp:9-14;
//                     EDGE::update_bending_energy, src/edge.cpp:51-67), kinetic energies
//                     (BEAD::update_kinetic_energy, src/bead.h:129-131) and intra-subunit pairs of a
//                     few subunits per CTA, and every subunit's bounding sphere
//   k_energy_inter    pairs j > i of beads in different subunits, CTA per subunit, over the
//                     subunits whose spheres come within the reach of the pair terms
//   k_energy_pairs    update_LJ_ES_energies_simplified (src/energies.cpp:24-93) without a DH
//                     cut-off: every pair j > i of the system
//   k_energy_bigbeads update_LJ_ES_energies_bigbeads (src/energies.cpp:96-137) when the system
//                     has encapsulation big beads
//   k_energy_totals   per-system sums with a fixed tree (src/md.cpp:586-594).
// The reference visits every pair j > i (no pair list, no prefilter) and credits it to i: shifted
// Debye-Hueckel, WCA (+1 shift), and attractive LJ shifted at ecut with sbar^6 and epsilon = -E.
// Pairs beyond every cut-off add exactly nothing to its sums and are not visited here.
//
// What bounds this file is FP64 issue: GB300 runs two FP64 lanes per cycle and SM, so a warp
// instruction holds the pipe for 16 cycles, and the pair terms are cut to about 27 of them: the
// inverse distance from an FP32 seed and one third-order Newton step instead of a square root and
// a division, the exponential by a table of 2^(j/64) and a degree-5 polynomial (Tang's scheme),
// the distance-independent factors as one weight per bead.  Every edge and bending quad is
// evaluated once per subunit instead of once per bead that it touches.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"
#include "launch.cuh"

namespace souffle {


__device__ __forceinline__ void ddiff(const EnergyArgs& a, double fx, int i, int j, double& x,
                                      double& y, double& z) {
  x = fixed_diff(a.px[i], a.px[j], fx);
  y = fixed_diff(a.py[i], a.py[j], fx);
  z = fixed_diff(a.pz[i], a.pz[j], fx);
}

// 2^(j/64), j = 0 .. 63, correctly rounded.
__device__ const double kExp2Tab[64] = {
    1.0, 1.0108892860517005, 1.0218971486541166, 1.0330248790212284,
    1.0442737824274138, 1.0556451783605572, 1.0671404006768237, 1.0787607977571199,
    1.0905077326652577, 1.102382583307841, 1.1143867425958924, 1.1265216186082418,
    1.1387886347566916, 1.1511892299529827, 1.1637248587775775, 1.1763969916502812,
    1.189207115002721, 1.202156731452703, 1.215247359980469, 1.22848053610687,
    1.241857812073484, 1.255380757024691, 1.2690509571917332, 1.2828700160787783,
    1.2968395546510096, 1.3109612115247644, 1.3252366431597413, 1.339667524053303,
    1.3542555469368927, 1.3690024229745905, 1.383909881963832, 1.3989796725383112,
    1.4142135623730951, 1.42961333839197, 1.4451808069770467, 1.460917794180647,
    1.4768261459394993, 1.4929077282912648, 1.5091644275934228, 1.5255981507445384,
    1.5422108254079407, 1.559004400237837, 1.5759808451078865, 1.593142151342267,
    1.6104903319492543, 1.6280274218573478, 1.645755478153965, 1.6636765803267364,
    1.681792830507429, 1.7001063537185235, 1.718619298122478, 1.7373338352737062,
    1.7562521603732995, 1.7753764925265212, 1.7947090750031072, 1.8142521755003989,
    1.8340080864093424, 1.8539791250833855, 1.8741676341103, 1.8945759815869656,
    1.9152065613971474, 1.9360617934922943, 1.9571441241754002, 1.978456026387951,
};

// 2^(u / 64) for |u| < 2^16 as u = k + f with k the nearest integer and |f| <= 1/2: the table's
// 2^(k / 64) times e^(f ln2 / 64), the latter by its series through the fifth power (truncation
// below (ln2 / 128)^6 / 720 < 4e-17).  u comes as r c, c = -kappa 64 / ln2, and f = r c - k is
// formed by one fused multiply-add, so only c's own rounding enters, as the rounding of kappa r
// would.
__device__ __forceinline__ double exp_rc(double r, double c, const double* tab) {
  const double big = 6755399441055744.0;  // 1.5 2^52: adding it rounds to an integer
  const double kd = fma(r, c, big);
  const int k = __double2loint(kd);
  const double f = fma(r, c, big - kd);
  const double p = f * fma(f, fma(f, fma(f, fma(f, 1.2417843701716925e-12, 5.732851688640402e-10), 2.1173137155464776e-07), 5.86490495505617e-05), 0.010830424696249145);
  const double T = tab[k & 63];
  const double s = __hiloint2double(__double2hiint(T) + ((k >> 6) << 20), __double2loint(T));
  return fma(s, p, s);
}
constexpr float kExpMaxArg = 690.0f;  // e^-x is taken as 0 beyond

// 1 / sqrt(r2) from the FP32 estimate of r2: one third-order step from rsqrt(r2f), e = 1 - r2 y^2,
// y (1 + e (1/2 + 3/8 e)); the FP32 value is off by a few 1e-7 for r > 0.1, so the remaining error
// (5/16 e^3) is far below a rounding.  Closer pairs take the square root and the division.
__device__ __forceinline__ double inv_sqrt(double r2, float r2f) {
  if (r2f < 0.01f) return 1.0 / sqrt(r2);
  const unsigned int f = __float_as_uint(rsqrtf(r2f));
  const double y = __hiloint2double((int)((f >> 3) + 0x38000000u), (int)(f << 29));
  const double e = fma(-(r2 * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// a difference of fixed-point coordinates in FP32 from its high word (within L / 2^32)
__device__ __forceinline__ float diff_f(long long d, float unit) { return (float)(int)(d >> 32) * unit; }

// dx^2 + dy^2 + dz^2 of fixed-point differences, in their units: the 128-bit integer sum, rounded once to
// FP64 by shifting its leading bits into place.  About 70 integer instructions, which this FP64-bound
// code has to spare, for nine FP64 ones (three of them conversions).
__device__ __forceinline__ double fixed_r2(const long long* d) {
  unsigned long long hi = 0, lo = 0;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const unsigned long long u = d[k] < 0 ? 0ull - (unsigned long long)d[k] : (unsigned long long)d[k];
    const unsigned long long l = u * u;
    lo += l;
    hi += __umul64hi(u, u) + (lo < l ? 1 : 0);
  }
  int s = __clzll((long long)hi);
  if (hi == 0) {
    hi = lo;
    lo = 0;
    s = 64 + __clzll((long long)hi);
    if (hi == 0) return 0.0;
  }
  const int n = s & 63;
  const unsigned long long m = n ? hi << n | lo >> (64 - n) : hi;  // leading bit 63, worth 2^(127 - s)
  const unsigned long long r = (m >> 11) + (m >> 10 & 1);          // 53 bits, the leading one at 52 (53 when rounding carries)
  return __longlong_as_double((long long)(((unsigned long long)(1022 + 127 - s) << 52) + r));
}

// The screened Coulomb term e^(-kappa r) / r minus its value at the cut-off, 0 beyond the cut-off,
// from exact fixed-point differences.  The cut-off is decided in FP32 except within a margin of it.
struct PairCut {
  float unit, cut2_lo, cut2_hi, kappa_f;
  double fx2, c, cut, shift;
  __device__ PairCut(const EnergyArgs& a, const SysParams& P) {
    unit = P.unit32;
    fx2 = P.fx_to_len * P.fx_to_len;
    cut = a.ecut_el;
    shift = a.el_shift;
    c = a.exp_scale;
    kappa_f = (float)a.kappa;
    const float c2 = (float)(cut * cut);
    cut2_lo = cut > 0 ? c2 * 0.999f - 1e-3f : -1.0f;
    cut2_hi = cut > 0 ? c2 * 1.001f + 1e-3f : -1.0f;
  }
  __device__ __forceinline__ float r2f(const long long* d) const {
    const float x = diff_f(d[0], unit), y = diff_f(d[1], unit), z = diff_f(d[2], unit);
    return x * x + y * y + z * z;
  }
  __device__ __forceinline__ double r2(const long long* d) const { return fixed_r2(d) * fx2; }
  __device__ __forceinline__ double term_r(double r, double ir, float f, const double* tab) const {
    const double e = kappa_f * sqrtf(f) < kExpMaxArg ? exp_rc(r, c, tab) : 0.0;
    const double v = fma(e, ir, -shift);
    if (f < cut2_lo) return v;
    return f <= cut2_hi && r < cut ? v : 0.0;
  }
  __device__ __forceinline__ double term(const long long* d, float f, const double* tab) const {
    const double q = r2(d), ir = inv_sqrt(q, f);
    return term_r(f < 0.01f ? sqrt(q) : q * ir, ir, f, tab);
  }
};

// Bonded terms, kinetic energies, intra-subunit Debye-Hueckel pairs and bounding spheres of
// a.spc consecutive subunits per CTA.  The edges (BEAD::update_stretching_energy,
// src/bead.cpp:9-14) and bending quads (EDGE::update_bending_energy, src/edge.cpp:51-67) are
// evaluated once each into shared memory and summed per bead in the bead's own order; the
// kinetic energy is BEAD::update_kinetic_energy (src/bead.h:129-131).  Pairs inside a subunit
// are nearly all within the cut-off, so they are walked densely: rows p and np - 1 - p together
// have np - 1 partners j > i, and two threads share such a pair of rows (even and odd partners),
// which keeps every lane of the FP64 loop busy.  At 84,000 beads (2000 x 42)
// 115 us, 80 % of the FP64 pipe while a CTA is resident (142 with separations formed in FP64: fixed_r2);
// one thread per bead over every edge and quad
// that touches it took 203 us for the bonded terms alone, the former pair kernel 1786.
__global__ void __launch_bounds__(256) k_energy_sub(EnergyArgs a) {
  extern __shared__ __align__(16) unsigned char esm[];
  const TplLayout& L = a.L;
  const SysParams& P = a.sys[a.sysid];
  const SysState& S = a.state[a.sysid];
  const int np = L.np, ne = L.ne, nb = L.nbend;
  const int s0 = blockIdx.x * a.spc, nsub = min(a.spc, a.n / np - s0), n = nsub * np;
  long long* sx = reinterpret_cast<long long*>(esm);
  long long* sy = sx + a.spc * np;
  long long* sz = sy + a.spc * np;
  double* s_edge = reinterpret_cast<double*>(sz + a.spc * np);  // [spc * ne]
  double* s_quad = s_edge + a.spc * ne;                         // [spc * nb]
  double* s_face = s_quad + a.spc * nb;                         // [spc * nf][4] area vector, magnitude (a.faces)
  double* s_part = s_face + (a.faces ? 4 * a.spc * L.nf : 0);   // [2][spc * np]
  double* s_w = s_part + 2 * a.spc * np;                        // [np]
  double* s_tab = s_w + np;                                     // [64]
  const int g0 = a.n0 + s0 * np;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    sx[t] = a.px[g0 + t];
    sy[t] = a.py[g0 + t];
    sz[t] = a.pz[g0 + t];
  }
  for (int t = threadIdx.x; t < np; t += blockDim.x) s_w[t] = a.w[t];
  if (threadIdx.x < 64) s_tab[threadIdx.x] = kExp2Tab[threadIdx.x];
  __syncthreads();
  const double fx = P.fx_to_len;
  auto diff = [&](int i, int j, double* d) {
    d[0] = fixed_diff(sx[i], sx[j], fx);
    d[1] = fixed_diff(sy[i], sy[j], fx);
    d[2] = fixed_diff(sz[i], sz[j], fx);
  };
  // the root of r2 to within a rounding: r2 times the inverse root, then one correction by the residual
  auto length = [](double r2) {
    const float r2f = (float)r2;
    if (!(r2f >= 0.01f && r2f < 1e30f)) return sqrt(r2);
    const double ir = inv_sqrt(r2, r2f), r = r2 * ir;
    return fma(0.5 * ir, fma(-r, r, r2), r);
  };
  for (int t = threadIdx.x; t < nsub * ne; t += blockDim.x) {
    const int s = t / ne, e = t - s * ne, pk = a.tpl_i[L.o_edge + e];
    const int i = s * np + (pk & 0xffff), j = s * np + (pk >> 16);
    const long long d[3] = {sx[i] - sx[j], sy[i] - sy[j], sz[i] - sz[j]};
    const double x = a.len0[e] - length(fixed_r2(d) * (fx * fx));
    s_edge[t] = 0.25 * P.ks_d * x * x;
  }
  auto area = [&](int s, int f, double* A) {  // area vector 1/2 (b1 - b0) x (b2 - b1) and its magnitude
    const int* fb = a.tpl_i + L.o_face + 3 * f;
    double u[3], v[3];
    diff(s * np + fb[1], s * np + fb[0], u);
    diff(s * np + fb[2], s * np + fb[1], v);
    A[0] = 0.5 * (u[1] * v[2] - u[2] * v[1]);
    A[1] = 0.5 * (u[2] * v[0] - u[0] * v[2]);
    A[2] = 0.5 * (u[0] * v[1] - u[1] * v[0]);
    A[3] = length(A[0] * A[0] + A[1] * A[1] + A[2] * A[2]);
  };
  for (int t = threadIdx.x; a.faces && t < nsub * L.nf; t += blockDim.x) area(t / L.nf, t % L.nf, s_face + 4 * t);
  __syncthreads();
  for (int t = threadIdx.x; t < nsub * nb; t += blockDim.x) {
    const int s = t / nb, k = t - s * nb, base = s * np;
    const double beta0 = (double)a.tpl_f[L.o_beta0 + k];
    double e;
    if (beta0 != 0.0) {  // rest-angle option: kb/4 (1 - cos(beta - beta0)) per quad bead
      const int* bq = a.tpl_i + L.o_bend + 4 * k;
      double v1[3], v2[3], v3[3];
      diff(base + bq[0], base + bq[2], v1);
      diff(base + bq[1], base + bq[0], v2);
      diff(base + bq[3], base + bq[1], v3);
      const double m[3] = {v1[1] * v2[2] - v1[2] * v2[1], v1[2] * v2[0] - v1[0] * v2[2], v1[0] * v2[1] - v1[1] * v2[0]};
      const double q[3] = {v2[1] * v3[2] - v2[2] * v3[1], v2[2] * v3[0] - v2[0] * v3[2], v2[0] * v3[1] - v2[1] * v3[0]};
      const double l2 = sqrt(v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2]);
      const double beta = atan2(-l2 * (v1[0] * q[0] + v1[1] * q[1] + v1[2] * q[2]), -(m[0] * q[0] + m[1] * q[1] + m[2] * q[2]));
      e = P.kb_d * 0.25 * (1.0 - cos(beta - beta0));
    } else {
      const int* bf = a.tpl_i + L.o_bendf + 2 * k;
      auto cosine = [](const double* A, const double* B) {
        return (A[0] * B[0] + A[1] * B[1] + A[2] * B[2]) / (A[3] * B[3]);
      };
      double c;
      if (a.faces) {
        c = cosine(s_face + 4 * (s * L.nf + bf[0]), s_face + 4 * (s * L.nf + bf[1]));
      } else {
        double A[4], B[4];
        area(s, bf[0], A);
        area(s, bf[1], B);
        c = cosine(A, B);
      }
      e = P.kb_d * 0.25 * (1.0 - fabs(c));
    }
    s_quad[t] = e;
  }
  // intra-subunit pairs (Debye-Hueckel only, src/energies.cpp:40-55)
  const int R = (np + 1) >> 1, per = 2 * R;
  if ((int)threadIdx.x < nsub * per) {
    const int s = threadIdx.x / per, u = threadIdx.x - s * per, p = u >> 1, h = u & 1, pb = np - 1 - p;
    const int n0 = np - 1 - p, total = pb != p ? np - 1 : n0;  // partners of row p, of both rows
    const int base = s * np;
    const PairCut pc(a, P);
    // partner number `it` of the two rows (row p first): its screened Coulomb term over w_i
    auto coords = [&](int it, int& i, int& j) {
      const bool first = it < n0;
      i = first ? p : pb;
      j = first ? p + 1 + it : pb + 1 + it - n0;
    };
    auto near = [&](int i, int j, long long* d, float& r2f) {
      d[0] = sx[base + i] - sx[base + j];
      d[1] = sy[base + i] - sy[base + j];
      d[2] = sz[base + i] - sz[base + j];
      r2f = pc.r2f(d);
      return r2f <= pc.cut2_hi;  // false without a cut-off: k_energy_pairs
    };
    double acc = 0.0, acc_p = 0.0;
    bool second = false;
    for (int it = h; it < total; it += 4) {
      const int it1 = it + 2;
      int i0, j0, i1, j1;
      long long d0[3], d1[3];
      float f0, f1;
      coords(it, i0, j0);
      coords(min(it1, total - 1), i1, j1);
      const bool in0 = near(i0, j0, d0, f0), in1 = near(i1, j1, d1, f1) && it1 < total;
      double v0 = 0.0, v1 = 0.0, w0 = 0.0, w1 = 0.0;
      if (in0 || in1) {
        v0 = pc.term(d0, f0, s_tab);
        v1 = pc.term(d1, f1, s_tab);
        w0 = in0 ? s_w[j0] : 0.0;
        w1 = in1 ? s_w[j1] : 0.0;
        if (__double2hiint(w0) == 0) v0 = 0.0;  // (an uncharged bead, w = 0; no FP64 comparison)
        if (__double2hiint(w1) == 0) v1 = 0.0;
      }
      if (!second && it >= n0) {  // row p is complete
        acc_p = acc;
        acc = 0.0;
        second = true;
      }
      acc = fma(w0, v0, acc);
      if (!second && it1 >= n0) {
        acc_p = acc;
        acc = 0.0;
        second = true;
      }
      acc = fma(w1, v1, acc);
    }
    if (!second) {
      acc_p = acc;
      acc = 0.0;
    }
    s_part[h * a.spc * np + base + p] = s_w[p] != 0.0 ? acc_p * s_w[p] : 0.0;
    if (pb != p) s_part[h * a.spc * np + base + pb] = s_w[pb] != 0.0 ? acc * s_w[pb] : 0.0;
  }
  // bounding spheres about the centre bead (FP32, padded), warp per subunit
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int s = wid; s < nsub; s += nw) {
    const int c = s * np + P.center_local;
    float r2 = 0.f;
    for (int l = lane; l < np; l += 32) {
      const int i = s * np + l;
      const float x = diff_f(sx[i] - sx[c], P.unit32), y = diff_f(sy[i] - sy[c], P.unit32), z = diff_f(sz[i] - sz[c], P.unit32);
      r2 = fmaxf(r2, x * x + y * y + z * z);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
    if (lane == 0) {
      const float rad = sqrtf(r2) * 1.001f + 1e-3f;
      a.sph[s0 + s] = make_int4(hi_word(sx[c]), hi_word(sy[c]), hi_word(sz[c]), __float_as_int(rad));
      atomicMax(a.rmax, __float_as_int(rad));  // positive floats order like their bits
    }
  }
  __syncthreads();
  const double inv = 1.0 / kVelScale;
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int s = t / np, l = t - s * np, g = g0 + t;
    double se = 0.0, be = 0.0;
    for (int k = 0; k < L.maxdeg; k++) {
      const int e = a.tpl_i[L.o_bead_edges + l * L.maxdeg + k];
      if (e < 0) break;
      se += s_edge[s * ne + (e & 0xffff)];
    }
    for (int k = 0; k < L.maxrole; k++) {
      const int r = a.tpl_i[L.o_bead_roles + l * L.maxrole + k];
      if (r < 0) break;
      be += s_quad[s * nb + (r >> 2)];
    }
    const double vx = (double)(a.vx[g] - S.vcom_fx[0]) * inv, vy = (double)(a.vy[g] - S.vcom_fx[1]) * inv,
                 vz = (double)(a.vz[g] - S.vcom_fx[2]) * inv;
    const int o = s0 * np + t;
    a.se[o] = se;
    a.be[o] = be;
    a.ke[o] = 0.5 * a.mass[l] * (vx * vx + vy * vy + vz * vz);
    a.ne[o] = 0.0;
    a.ce[o] = s_part[t] + s_part[a.spc * np + t];
  }
}

// Pairs of beads in different subunits, CTA (four warps) per half of the beads (rows) of subunit i
// (all of them up to 16 beads): partners in subunits j > i
// whose bounding spheres come within the reach of the pair terms.  Candidate subunits come from a
// scan of all j > i (threads along j, 16 coalesced bytes each) up to kEnergyScan subunits, and from the
// cells of the subunit centres within reach beyond.  A call with the scan against one with the cells (four
// launches to build them): 153 and 179 us at 1,000 subunits, 213 and 242 at 2,000, 341 and 362 at 4,000, 490
// and 500 at 6,000, 638 and 617 at 8,000, 972 and 870 at 12,000, 1,353 and 1,121 at 16,000; so the lines
// cross near 7,000, below where kEnergyScan has the change.  A candidate's beads are staged in shared memory;
// every (row, 32 partners) item of the block passes an FP32 test with a margin at once, the hits
// are listed row by row, and the FP64 terms run 128 listed pairs at a time, each row's terms then
// summed with a fixed tree: deterministic.  Few pairs (147,000 at 84,000 beads) behind long
// chains of loads and FP64 latency, the longest in subunits with several contacts: one warp per
// subunit took 257 us there, four warps with a queue each 157, a CTA per subunit 68, two CTAs 63 (four: 75); 60 with fixed_r2.
constexpr int kEnergyCand = 1280;    // candidate subunits held per CTA
constexpr int kEnergyScan = 16384;   // subunits up to which all are scanned
constexpr int kScanBatch = 8;        // subunits per thread and round of the scan
__host__ __device__ inline size_t energy_inter_bytes(int np) { return 64 * (size_t)np; }
__global__ void __launch_bounds__(128) k_energy_inter(EnergyArgs a) {
  extern __shared__ __align__(16) unsigned char esm[];
  __shared__ double s_tab[64];
  __shared__ double s_val[2][128];
  __shared__ int s_cand[kEnergyCand];
  __shared__ unsigned short s_list[128 * 32];  // row | partner << 8
  __shared__ int s_item[129];                  // list offset of each item of the pass
  __shared__ int s_wsum[4];
  __shared__ unsigned int s_word[4 * kScanBatch];
  __shared__ int s_off[4 * kScanBatch + 1];
  const SysParams& P = a.sys[a.sysid];
  const int np = a.L.np, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nsub = a.n / np;
  double* acc_c = reinterpret_cast<double*>(esm);  // [np]
  double* acc_n = acc_c + np;
  long long* own = reinterpret_cast<long long*>(acc_n + np);  // [3][np] this subunit's coordinates
  long long* oth = own + 3 * np;                              // [3][np] the candidate's
  const int i = blockIdx.x;  // system-local subunit
  const int gi0 = a.n0 + i * np;
  if (threadIdx.x < 64) s_tab[threadIdx.x] = kExp2Tab[threadIdx.x];
  for (int l = threadIdx.x; l < np; l += blockDim.x) {
    acc_c[l] = acc_n[l] = 0.0;
    own[l] = a.px[gi0 + l];
    own[np + l] = a.py[gi0 + l];
    own[2 * np + l] = a.pz[gi0 + l];
  }
  const float unit = P.unit32;
  const double rmax = fmax(fmax(a.ecut, a.ecut_el), 1.12246205 * a.sigma_max);
  const float rmaxf = (float)rmax * 1.001f + 1e-3f;
  const float rmax2 = (float)(rmax * rmax) * 1.001f + 1e-3f;
  const PairCut pc(a, P);
  const int* species = a.tpl_i + a.L.o_species;
  const int4 si = a.sph[i];
  const float ri = __int_as_float(si.w);
  const int words = a.L.words;
  const int r0 = np * (int)blockIdx.y / (int)gridDim.y, r1 = np * ((int)blockIdx.y + 1) / (int)gridDim.y;
  const int items = (r1 - r0) * words;
  int nc = 0;  // candidates held (uniform over the CTA)

  auto run_candidates = [&]() {  // whole CTA: the nc candidates in s_cand
    __syncthreads();
    for (int c = 0; c < nc; c++) {
      const int gj0 = a.n0 + s_cand[c] * np;
      for (int l = threadIdx.x; l < np; l += blockDim.x) {
        oth[l] = a.px[gj0 + l];
        oth[np + l] = a.py[gj0 + l];
        oth[2 * np + l] = a.pz[gj0 + l];
      }
      __syncthreads();
      const int* oh = reinterpret_cast<const int*>(oth);  // high words at odd places
      for (int t0 = 0; t0 < items; t0 += 128) {
        const int t = t0 + threadIdx.x;
        const int q0 = t / words, row = r0 + q0, w0 = (t - q0 * words) * 32;
        unsigned int mask = 0;
        if (t < items) {
          const int x = (int)(own[row] >> 32), y = (int)(own[np + row] >> 32), z = (int)(own[2 * np + row] >> 32);
          const int w1 = min(np - w0, 32);
#pragma unroll 4
          for (int k = 0; k < w1; k++) {
            const int l = w0 + k;
            const float dx = hi_diff(x, oh[2 * l + 1], unit), dy = hi_diff(y, oh[2 * (np + l) + 1], unit),
                        dz = hi_diff(z, oh[2 * (2 * np + l) + 1], unit);
            if (!(dx * dx + dy * dy + dz * dz > rmax2)) mask |= 1u << k;
          }
        }
        const int cnt = __popc(mask);
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        if (lane == 31) s_wsum[wid] = incl;
        __syncthreads();
        int off = incl - cnt, total = 0;
        for (int q = 0; q < 4; q++) {
          if (q < wid) off += s_wsum[q];
          total += s_wsum[q];
        }
        s_item[threadIdx.x] = off;
        if (threadIdx.x == 0) s_item[128] = total;
        for (; mask; mask &= mask - 1)
          s_list[off++] = (unsigned short)(row | (w0 + __ffs(mask) - 1) << 8);
        __syncthreads();
        // rows of this pass, one thread each: items [first, last) of the pass
        const int q_t = t0 / words + threadIdx.x, row_t = r0 + q_t;
        const int first = max(q_t * words - t0, 0), last = min((q_t + 1) * words - t0, 128);
        const bool owner = row_t < r1 && first < last;
        const int lo = owner ? s_item[first] : 0, hi = owner ? s_item[last] : 0;
        double ac = 0.0, an = 0.0;
        for (int b = 0; b < total; b += 128) {
          int li = -1;
          double ce = 0.0, ne = 0.0;
          if (b + (int)threadIdx.x < total) {
            const int e = s_list[b + threadIdx.x], lj = e >> 8;
            li = e & 0xff;
            const long long d[3] = {own[li] - oth[lj], own[np + li] - oth[np + lj], own[2 * np + li] - oth[2 * np + lj]};
            const float f = pc.r2f(d);
            const double q = pc.r2(d), ir = inv_sqrt(q, f), r = f < 0.01f ? sqrt(q) : q * ir;
            const double wi = a.w[li], wj = a.w[lj];
            if (f <= pc.cut2_hi && wi != 0.0 && wj != 0.0) ce = wi * (wj * pc.term_r(r, ir, f, s_tab));
            const double shc = (a.sigma[li] + a.sigma[lj]) / 2;
            const bool att = (a.L.lj_att_bits[species[li]] >> species[lj]) & 1;
            if (att ? r < a.ecut : r < 1.12246205 * shc) {
              const double s3 = shc * shc * shc, ir3 = ir * ir * ir;
              const double q3 = s3 * ir3, q6 = q3 * q3;
              if (att) {
                const double e3 = s3 * a.inv_ecut3, e6 = e3 * e3;
                ne = 4 * a.elj_att * q6 * (q6 - 1) - 4 * a.elj_att * (e6 * (e6 - 1));
              } else {
                ne = 4 * q6 * (q6 - 1) + 1;
              }
            }
          }
          // sums over runs of equal rows inside the warp (a segmented scan: five dependent adds
          // instead of one per pair; a dependent FP64 add costs hundreds of cycles), the run's
          // sum at its first lane
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int r = __shfl_down_sync(0xffffffffu, li, o);
            const double c = __shfl_down_sync(0xffffffffu, ce, o), m = __shfl_down_sync(0xffffffffu, ne, o);
            if (lane + o < 32 && r == li) {
              ce += c;
              ne += m;
            }
          }
          s_val[0][threadIdx.x] = ce;
          s_val[1][threadIdx.x] = ne;
          __syncthreads();
          for (int k = max(lo, b); k < min(hi, b + 128); k = (k | 31) + 1) {  // the row's runs, a warp each
            ac += s_val[0][k - b];
            an += s_val[1][k - b];
          }
          __syncthreads();
        }
        if (hi > lo) {
          acc_c[row_t] += ac;
          acc_n[row_t] += an;
        }
      }
      __syncthreads();
    }
    nc = 0;
  };
  // appends the subunits j[k] that pass (k = 0 .. n - 1 per thread, ascending k then thread)
  auto gather = [&](const int* j, int n) {
    bool pass[kScanBatch];
    unsigned int below[kScanBatch];
#pragma unroll
    for (int k = 0; k < kScanBatch; k++) {
      if (k >= n) break;
      pass[k] = false;
      if (j[k] > i) {
        const int4 sj = a.sph[j[k]];
        const float x = hi_diff(si.x, sj.x, unit), y = hi_diff(si.y, sj.y, unit), z = hi_diff(si.z, sj.z, unit);
        const float lim = ri + __int_as_float(sj.w) + rmaxf;
        pass[k] = x * x + y * y + z * z < lim * lim;
      }
    }
#pragma unroll
    for (int k = 0; k < kScanBatch; k++) {
      if (k >= n) break;
      const unsigned int m = __ballot_sync(0xffffffffu, pass[k]);
      below[k] = __popc(m & ((1u << lane) - 1u));
      if (lane == 0) s_word[4 * k + wid] = m;
    }
    __syncthreads();
    if (wid == 0) {
      static_assert(4 * kScanBatch == 32, "one word per lane");
      const int c = lane < 4 * n ? __popc(s_word[lane]) : 0;
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      s_off[lane] = incl - c;
      if (lane == 31) s_off[32] = incl;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kScanBatch; k++) {
      if (k >= n) break;
      if (pass[k]) s_cand[nc + s_off[4 * k + wid] + below[k]] = j[k];
    }
    nc += s_off[32];
    if (nc > kEnergyCand - 128 * kScanBatch) run_candidates();
  };
  if (nsub <= kEnergyScan) {
    for (int base = i + 1; base < nsub; base += 128 * kScanBatch) {
      int j[kScanBatch];
#pragma unroll
      for (int k = 0; k < kScanBatch; k++) {
        const int q = base + 128 * k + threadIdx.x;
        j[k] = q < nsub ? q : -1;
      }
      gather(j, kScanBatch);
    }
  } else {
    const int n = P.ncell;
    const float edge = (float)(P.box / n) * 0.999f;
    const int range = (int)ceilf((rmaxf + 2.0f * __int_as_float(*a.rmax)) / edge);
    const int span = min(n, 2 * range + 1), ncells = span * span * span;
    const int c = gi0 + P.center_local;
    auto axis = [&](long long x) { return (int)__umul64hi((unsigned long long)x + 0x8000000000000000ull, (unsigned long long)n); };
    const int cx = axis(a.px[c]) - span / 2, cy = axis(a.py[c]) - span / 2, cz = axis(a.pz[c]) - span / 2;
    for (int base = 0; base < ncells; base += 128) {
      int cur = 0, end = 0;
      const int q = base + threadIdx.x;
      if (q < ncells) {
        const int gx = (cx + q / (span * span) + 2 * n) % n, gy = (cy + (q / span) % span + 2 * n) % n,
                  gz = (cz + q % span + 2 * n) % n;
        const int cell = P.cell0 + (gx * n + gy) * n + gz;
        cur = a.sub_cell_start[cell];
        end = cur + a.sub_cell_count[cell];
      }
      while (__syncthreads_or(cur < end)) {
        const int j = cur < end ? a.cell_subs[cur] - P.sub0 : -1;
        cur++;
        gather(&j, 1);
      }
    }
  }
  if (nc > 0) run_candidates();
  __syncthreads();
  for (int l = r0 + threadIdx.x; l < r1; l += blockDim.x) {
    a.ce[i * np + l] += acc_c[l];
    a.ne[i * np + l] += acc_n[l];
  }
}

// Per template bead pair (li, lj), the pair terms that do not depend on the distance, in the
// reference's expressions: the Yukawa size factor e^(kappa sbar) / ((1 + kappa s_i / 2)
// (1 + kappa s_j / 2)), sbar^6, the attractive LJ shift 4 eps ((sbar^6 / ecut^6)
// ((sbar^6 / ecut^6) - 1)), and whether (type_i, type_j) is a row of the directed LJ table.
__global__ void k_energy_tables(EnergyArgs a) {
  const int np = a.L.np;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= np * np) return;
  const int li = idx / np, lj = idx - li * np;
  const double kappa = a.kappa, ecut = a.ecut;
  const double ecut3 = ecut * ecut * ecut, ecut6 = ecut3 * ecut3;
  const double sgi = a.sigma[li], sgj = a.sigma[lj];
  const double shc = (sgi + sgj) / 2;
  const double s3 = shc * shc * shc, s6 = s3 * s3;
  a.pair_tab[idx] = exp(kappa * shc) / ((1 + kappa * sgi / 2) * (1 + kappa * sgj / 2));
  a.pair_tab[np * np + idx] = s6;
  a.pair_tab[2 * np * np + idx] = 4 * a.elj_att * ((s6 / ecut6) * ((s6 / ecut6) - 1));
  bool att = false;
  for (int m = 0; m < a.n_lj; m++)
    if (a.type[li] == a.lj_t[2 * m] && a.type[lj] == a.lj_t[2 * m + 1]) att = true;
  a.att_tab[idx] = att ? 1 : 0;
}

// The FP64 terms of one pair (i, j) within reach, credited to i (src/energies.cpp:40-89), with the
// distance-independent factors from k_energy_tables.  Out of line, so that none of its FP64
// work is scheduled into the pair loop's float test.
__device__ __noinline__ void pair_energy(const EnergyArgs& a, const SysParams& P, int gi, int gj, int lj_, int li,
                                         double qi, double sgi, bool elec, bool lj, double e_cut_el, double& ce,
                                         double& ne) {
  const double kappa = a.kappa, lb = a.lb, ecut = a.ecut, ecut_el = a.ecut_el;
  const int np = a.L.np, idx = li * np + lj_;
  const double qj = a.q[lj_];
  double x, y, z;
  ddiff(a, P.fx_to_len, gi, gj, x, y, z);
  const double r = sqrt(x * x + y * y + z * z);
  const double shc = (sgi + a.sigma[lj_]) / 2;
  const double ys = a.pair_tab[idx];
  if (elec && r < ecut_el && ecut_el != 0) {
    ce += ys * ((qi * qj * lb * exp(-kappa * r)) / r - ((qi * qj * lb * e_cut_el) / ecut_el));
  } else if (elec && ecut_el == 0) {
    ce += (qi * qj * lb * exp(-kappa * r) * ys) / r;
  }
  if (r >= ecut && r >= (1.12246205 * shc)) return;
  if (lj) {
    const double s6 = a.pair_tab[np * np + idx];
    const double r3 = r * r * r, r6 = r3 * r3;
    const double q6 = s6 / r6;
    const bool att = a.att_tab[idx] != 0;
    if (r < (1.12246205 * shc) && !att) {
      ne += (4 * q6 * (q6 - 1)) + 1;
    } else if (r < ecut && att) {
      ne += (4 * a.elj_att * q6 * (q6 - 1)) - a.pair_tab[2 * np * np + idx];
    }
  }
}

// One warp per bead i; lane L tests the partners j = i + 1 + L, i + 33 + L, ... of the whole
// system with integer and FP32 work only: the partner's template index is the .w of its position
// entry, "same subunit" is a range test on the index, "both charged" reads per-template flags in
// shared memory, then a float distance test with a conservative margin.  The few partners that
// pass go into a per-warp queue in shared memory (in lane order, by ballot), and the FP64 pair
// terms run 32 queued pairs at a time with every lane busy: GB300's FP64 unit is a small fraction
// of its FP32 rate, and with one call per passing lane most of it ran masked.  Each lane sums its
// queue slots in order; the warp then adds the lane sums in a fixed tree: deterministic.
constexpr int kEnergyWarps = 8;
__global__ void __launch_bounds__(32 * kEnergyWarps) k_energy_pairs(EnergyArgs a) {
  __shared__ unsigned char s_charged[kMaxNp];
  __shared__ int2 s_queue[kEnergyWarps][64];
  const SysParams& P = a.sys[a.sysid];
  const int np = a.L.np;
  for (int l = threadIdx.x; l < np; l += blockDim.x) s_charged[l] = a.q[l] != 0.0;  // np <= kMaxNp
  __syncthreads();
  const int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (t >= a.n) return;  // uniform over the warp
  int2* queue = s_queue[threadIdx.x >> 5];
  const int gi = a.n0 + t;
  const int li = gi % np, si = gi / np;
  const int sub_lo = si * np, sub_hi = sub_lo + np;  // global indices of i's subunit
  const int4 pi = a.pos32[gi];
  const double qi = a.q[li], sgi = a.sigma[li];
  const bool ci = qi != 0.0;
  const float unit = P.unit32;
  const double kappa = a.kappa, ecut = a.ecut, ecut_el = a.ecut_el;
  const double e_cut_el = exp(-kappa * ecut_el);  // the shift's exponential, the same for every pair
  const double rmax = fmax(fmax(ecut, ecut_el), 1.12246205 * a.sigma_max);
  const float rmax2 = (float)(rmax * rmax) * 1.001f + 1e-3f;
  // per-axis reach in high-word units (L / 2^32), rounded up with a margin: beyond it on any axis
  // the pair is out of reach without a conversion to floating point
  const int lim = (int)fmin(2147483647.0, ceil(rmax * 1.001 / (double)unit) + 4.0);
  const bool no_dh_cut = (ecut_el == 0.0);
  double ce = 0.0, ne = 0.0;
  int qn = 0;  // queued pairs (uniform over the warp)
  auto run_queue = [&](int count) {  // the first count queue slots, one per lane
    __syncwarp();
    if (lane < count) {
      const int2 e = queue[lane];
      pair_energy(a, P, gi, e.x, e.y & 0xffff, li, qi, sgi, (e.y >> 16) & 1, (e.y >> 17) & 1, e_cut_el, ce, ne);
    }
    __syncwarp();
  };
  const int n_iter = (a.n - (t + 1) + 31) / 32;  // uniform trip count
  for (int it = 0; it < n_iter; it++) {
    const int tj = t + 1 + it * 32 + lane;
    bool pass = false, lj = false, elec = false;
    int4 pj = make_int4(0, 0, 0, 0);
    if (tj < a.n) {
      const int gj = a.n0 + tj;
      pj = __ldg(&a.pos32[gj]);
      lj = gj < sub_lo || gj >= sub_hi;  // different subunits
      elec = ci && s_charged[pj.w];
      if (no_dh_cut && elec) {
        pass = true;
      } else if (elec || lj) {
        const int ix = (int)((unsigned int)pi.x - (unsigned int)pj.x), iy = (int)((unsigned int)pi.y - (unsigned int)pj.y),
                  iz = (int)((unsigned int)pi.z - (unsigned int)pj.z);
        // (abs of the most negative int stays negative and falls through to the float test)
        if (!(abs(ix) > lim || abs(iy) > lim || abs(iz) > lim)) {
          const float dx = (float)ix * unit, dy = (float)iy * unit, dz = (float)iz * unit;
          pass = !(dx * dx + dy * dy + dz * dz > rmax2);
        }
      }
    }
    const unsigned int m = __ballot_sync(0xffffffffu, pass);
    if (pass)
      queue[qn + __popc(m & ((1u << lane) - 1u))] =
          make_int2(a.n0 + tj, pj.w | (elec ? 1 << 16 : 0) | (lj ? 1 << 17 : 0));
    qn += __popc(m);
    if (qn >= 32) {
      run_queue(32);
      if (lane < qn - 32) queue[lane] = queue[32 + lane];
      qn -= 32;
    }
  }
  if (qn > 0) run_queue(qn);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ce += __shfl_xor_sync(0xffffffffu, ce, o);
    ne += __shfl_xor_sync(0xffffffffu, ne, o);
  }
  if (lane == 0) {
    a.ne[t] = ne;
    a.ce[t] = ce;
  }
}

// Encapsulation big beads (update_LJ_ES_energies_bigbeads, src/energies.cpp:96-137): per
// subunit bead, the unshifted screened Coulomb energy with each big bead inside the DH cut-off
// (none without one) and the shifted WCA energy (+1) inside delta + 2^(1/6) shc, added to the
// bead's ne / ce (the reference credits them to the subunit bead and to the big bead) and kept
// apart for the big-bead totals.  Exact fixed-point differences in double.
__global__ void __launch_bounds__(128) k_energy_bigbeads(EnergyArgs a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= a.n) return;
  const SysParams& P = a.sys[a.sysid];
  const int gi = a.n0 + t, li = gi % a.L.np;
  const double qj = a.q[li], sgj = a.sigma[li];
  const double kappa = a.kappa, lb = a.lb, ecut_el = a.ecut_el;
  const double shc = P.bb_shc_d, sigb = P.bb_sigma_d;
  const double sigavg = (sigb + sgj) / 2;
  const double delta = sigavg - shc;
  const double shc6 = pow(shc, 6);
  const double ys = exp(kappa * sigavg) / ((1 + kappa * sigb / 2) * (1 + kappa * sgj / 2));
  double ce = 0.0, ne = 0.0;
  for (int k = 0; k < P.nbb; k++) {
    const int b = P.bb0 + k;
    const double x = fixed_diff(a.bb_fx[b], a.px[gi], P.fx_to_len);
    const double y = fixed_diff(a.bb_fx[a.bb_total + b], a.py[gi], P.fx_to_len);
    const double z = fixed_diff(a.bb_fx[2 * a.bb_total + b], a.pz[gi], P.fx_to_len);
    const double r = sqrt(x * x + y * y + z * z);
    const double r6 = pow(r - delta, 6);
    if (qj != 0 && r < ecut_el) ce += (P.bb_q * qj * lb * exp(-kappa * r) * ys) / r;
    if (r < delta + 1.12246205 * shc) ne += (4 * (shc6 / r6) * ((shc6 / r6) - 1)) + 1;
  }
  a.ne[t] += ne;
  a.ce[t] += ce;
  a.ne_bb[t] = ne;
  a.ce_bb[t] = ce;
}

// Totals (kinetic, stretching, bending, lj, electrostatic, and the big-bead parts of the last
// two): each CTA sums a contiguous run of beads with a fixed tree, and the last one to finish sums
// the CTAs' partial sums the same way, so the result does not depend on scheduling.
__global__ void __launch_bounds__(kTotalThreads) k_energy_totals(EnergyArgs a, int count) {
  __shared__ double red[kTotalThreads / 32][7];
  __shared__ bool last;
  const double* src[7] = {a.ke, a.se, a.be, a.ne, a.ce, a.ne_bb, a.ce_bb};
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto reduce = [&](double (&s)[7]) {  // the CTA's sums, valid in thread 0
#pragma unroll
    for (int k = 0; k < 7; k++) {
      if (k >= count) break;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
      if (lane == 0) red[wid][k] = s[k];
    }
    __syncthreads();
    if ((int)threadIdx.x < count) {
      double t = 0.0;
      for (int w = 0; w < kTotalThreads / 32; w++) t += red[w][threadIdx.x];
      red[0][threadIdx.x] = t;
    }
    __syncthreads();
  };
  const int per = (a.n + gridDim.x - 1) / gridDim.x;
  const int beg = blockIdx.x * per, end = min(a.n, beg + per);
  double s[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int t = beg + threadIdx.x; t < end; t += blockDim.x)
#pragma unroll
    for (int k = 0; k < 7; k++)
      if (k < count) s[k] += src[k][t];
  reduce(s);
  if ((int)threadIdx.x < count) a.partials[blockIdx.x * 7 + threadIdx.x] = red[0][threadIdx.x];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < 7; k++) s[k] = 0.0;
  for (int t = threadIdx.x; t < (int)gridDim.x; t += blockDim.x)
#pragma unroll
    for (int k = 0; k < 7; k++)
      if (k < count) s[k] += __ldcg(a.partials + t * 7 + k);
  reduce(s);
  if ((int)threadIdx.x < count) a.totals[threadIdx.x] = red[0][threadIdx.x];
  if (threadIdx.x == 0) {  // ready for the next call
    *a.ticket = 0u;
    *a.rmax = 0;
  }
}

}  // namespace souffle

namespace souffle {
// Subunits per CTA of k_energy_sub (two threads per pair of rows, up to 128 threads), whether it keeps the
// faces' area vectors in shared memory, and its dynamic shared memory.  Templates with edges or faces
// by the thousand take fewer subunits, then form area vectors for each bending quad: a mesh without
// bending edges may have more faces than shared memory holds.
static size_t energy_sub_bytes(const TplLayout& L, int spc, bool faces) {
  return (size_t)spc * L.np * 24 +
         sizeof(double) * ((size_t)spc * (L.ne + L.nbend + (faces ? 4 * (size_t)L.nf : 0) + 2 * L.np) + L.np + 64);
}
EnergySubPlan energy_sub_plan(const TplLayout& L) {
  EnergySubPlan p{std::max(1, 128 / (2 * ((L.np + 1) / 2))), true, 0};
  while (p.spc > 1 && energy_sub_bytes(L, p.spc, true) > kMaxDynamicSmem) p.spc--;
  p.faces = energy_sub_bytes(L, p.spc, true) <= kMaxDynamicSmem;
  p.smem = energy_sub_bytes(L, p.spc, p.faces);
  return p;
}
cudaError_t set_energy_smem(const TplLayout& L) {
  return raise_smem_limit((const void*)k_energy_sub, energy_sub_plan(L).smem);
}
bool energy_needs_cells(int n_sub) { return n_sub > kEnergyScan; }
void launch_energies(const EnergyArgs& a, int n, cudaStream_t s) {
  const int np = a.L.np, nsub = n / np;
  const int per = 2 * ((np + 1) / 2);
  const int threads = std::max(64, (a.spc * per + 31) / 32 * 32);
  k_energy_sub<<<(nsub + a.spc - 1) / a.spc, threads, energy_sub_plan(a.L).smem, s>>>(a);
  if (a.ecut_el > 0) {
    k_energy_inter<<<dim3(nsub, std::min(2, (np + 15) / 16)), 128, energy_inter_bytes(np), s>>>(a);
  } else {  // no DH cut-off: every pair j > i
    k_energy_tables<<<(np * np + 127) / 128, 128, 0, s>>>(a);
    k_energy_pairs<<<(int)(((long long)n + kEnergyWarps - 1) / kEnergyWarps), 32 * kEnergyWarps, 0, s>>>(a);  // a warp per bead
  }
  const bool bb = a.ne_bb != nullptr;
  if (bb) k_energy_bigbeads<<<(n + 127) / 128, 128, 0, s>>>(a);
  k_energy_totals<<<std::min(kTotalCtas, (n + kTotalThreads - 1) / kTotalThreads), kTotalThreads, 0, s>>>(a, bb ? 7 : 5);
}
}  // namespace souffle
