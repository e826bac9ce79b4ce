// The phases of one force evaluation over a CTA's run of subunits (a work item), shared by the
// force kernel and the window kernel of forces.cu.
//
//   force_setup      template tables and per-item constants into shared memory
//   force_rel        a bead's packed coordinates relative to its subunit's centre bead
//   force_rows       the inter-subunit lists cut into pieces of like length
//   force_terms      everything that depends on positions alone, in chunks of 32 lanes that the
//                    warps take from a counter: intra-subunit Debye-Hueckel rows, bending quads,
//                    inter-subunit pairs, edges (the costliest chunks first)
//   force_gather     per bead: stretching and bending sums
// Every contribution ends as an exact 2^-32 fixed-point sum in the bead's limbs in shared memory,
// so the total does not depend on the CTA shape or on scheduling; the FP32 sums inside one
// contribution have a fixed order (a bead's edges, its bending roles, its even and its odd
// intra-subunit partners).
//
// What bounds them: instruction issue (a third of all instructions were the intra-subunit pairs),
// and for systems of a wave of CTAs or less the latency of one phase after the other.  So the
// intra-subunit row is walked densely, an even and an odd partner at a time in packed FP32 (f32x2)
// registers -- about 15 instructions per directed pair against 33 for extracting partners from the
// row's bitmask one by one; a pair off the list or beyond the cut-off is dropped by a select --
// and the independent kinds of work share one phase instead of taking one each.
#pragma once
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace souffle {

__device__ __forceinline__ float3 f3(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 dvec(int4 a, int4 b, float unit) {
  return f3(hi_diff(a.x, b.x, unit), hi_diff(a.y, b.y, unit), hi_diff(a.z, b.z, unit));
}

// ---- packed FP32: two values per 64-bit register, each operation rounded like its scalar form ----
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// t / d by a multiplication: magic = ceil(2^32 / d) (0 for d = 1), exact for t < 2^32 / d
__device__ __forceinline__ int fast_div(int t, unsigned int magic) { return magic ? (int)__umulhi((unsigned int)t, magic) : t; }

// A bead's force component in 2^-32 fixed point kept as three 21-bit limbs in 32-bit words
// (v = l2 2^42 + l1 2^21 + l0, l0 and l1 in [0, 2^21), l2 signed), so that pair forces can be
// added with native 32-bit shared-memory atomics: the limb sums stay exact for up to 2^11 adds.
__device__ __forceinline__ void limbs_add(unsigned int* L, long long v) {
  atomicAdd(L, (unsigned int)(v & 0x1FFFFF));
  atomicAdd(L + 1, (unsigned int)((v >> 21) & 0x1FFFFF));
  atomicAdd(L + 2, (unsigned int)(int)(v >> 42));
}
__device__ __forceinline__ long long limbs_value(const unsigned int* L) {
  const unsigned long long hi = (unsigned long long)(long long)(int)L[2] << 42;
  return (long long)(hi + ((unsigned long long)L[1] << 21) + (unsigned long long)L[0]);
}

// f32_to_fx32 of two values at once, |v| < 2^22, for sums: the floor by an addition that rounds down at
// 2^23 + 2^22, whose bits are that constant's plus the floor.  Those bits are added as they are: sum -=
// fx_bias(n) after n values.
__device__ __forceinline__ void fx_add2(unsigned long long& sum, f32x2 v) {
  f32x2 t;
  const f32x2 magic = pack2(12582912.0f, 12582912.0f);
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(t) : "l"(v), "l"(magic));
  const f32x2 hi = add2(t, pack2(-12582912.0f, -12582912.0f));
  float ha, hb;
  unpack2(hi, ha, hb);
  const f32x2 frac = mul2(add2(v, pack2(-ha, -hb)), pack2(4294967296.0f, 4294967296.0f));
  float fa, fb, ta, tb;
  unpack2(frac, fa, fb);
  unpack2(t, ta, tb);
  sum += (unsigned long long)__float_as_uint(ta) << 32 | __float2uint_rn(fa);
  sum += (unsigned long long)__float_as_uint(tb) << 32 | __float2uint_rn(fb);
}
__device__ __forceinline__ unsigned long long fx_bias(int n) { return (unsigned long long)(0x4B400000u * (unsigned int)n) << 32; }

// true for a non-finite component or one beyond 1e9 in magnitude
__device__ __forceinline__ bool force_bad(float x, float y, float z) {
  const float s = fabsf(x) + fabsf(y) + fabsf(z);  // NaN or infinite when a component is
  return !(s < 3.0e38f) || fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)) > 1.0e9f;
}

// Shared memory of a work item, carved from the CTA's dynamic allocation (16-byte aligned pieces
// first; force_smem_bytes is its size).
struct ForceSmem {
  float4* edge;        // [max_sub ne] length vector, stretching coefficient
  float4* bend;        // [max_sub nb 4] bending contributions
  int4* pos;           // [max_sub np] high words
  float* rel;          // [max_sub npp 8] packed partners: (x0, x1, y0, y1, z0, z1, w0, w1) per two beads
  long long* red;      // [4 warps]
  unsigned int* F;     // force limbs, 9 per bead
  int* rows;           // pieces of the beads' inter-subunit lists (force_rows)
  float* tpl_f;
  int* tpl_i;
  float* w;            // [np] DH weights
};
__device__ __forceinline__ ForceSmem force_smem(unsigned char* base, const ForceArgs& a, int warps) {
  const TplLayout& L = a.L;
  ForceSmem m;
  const int npp = (L.np + 1) >> 1;
  m.edge = reinterpret_cast<float4*>(base);
  m.bend = m.edge + a.max_sub * L.ne;
  m.pos = reinterpret_cast<int4*>(base + force_tile_bytes(a.max_sub, L.ne, L.nbend));
  m.rel = reinterpret_cast<float*>(m.pos + a.max_sub * L.np);
  m.red = reinterpret_cast<long long*>(m.rel + 8 * a.max_sub * npp);
  m.F = reinterpret_cast<unsigned int*>(m.red + 4 * warps);
  m.rows = reinterpret_cast<int*>(m.F + force_slot_len(a.max_sub * L.np));
  m.tpl_f = reinterpret_cast<float*>(m.rows + force_rows_len(a.max_sub * L.np));  // [n_float], n_float % 4 == 0
  m.tpl_i = reinterpret_cast<int*>(m.tpl_f + L.n_float);                          // [n_int], n_int % 4 == 0
  m.w = reinterpret_cast<float*>(m.tpl_i + L.n_int);
  return m;
}

// Template tables.
__device__ __forceinline__ void force_setup(const ForceArgs& a, const ForceSmem& m) {
  const TplLayout& L = a.L;
  const int4* gi = reinterpret_cast<const int4*>(a.tpl_i);
  int4* si = reinterpret_cast<int4*>(m.tpl_i);
  for (int t = threadIdx.x; t < (L.n_int >> 2); t += blockDim.x) si[t] = __ldg(gi + t);
  const float4* gf = reinterpret_cast<const float4*>(a.tpl_f);
  float4* sf = reinterpret_cast<float4*>(m.tpl_f);
  for (int t = threadIdx.x; t < (L.n_float >> 2); t += blockDim.x) sf[t] = __ldg(gf + t);
}

// The packed relative coordinates of bead t (subunit s, local index l) at high words p, centre
// bead at c, DH weight wt; an odd subunit's last slot is filled with the bead itself (its partner
// bit is never set).
__device__ __forceinline__ void force_rel(const ForceSmem& m, int np, int s, int l, int4 p, int4 c, float wt, float unit) {
  float* r = m.rel + 8 * (s * ((np + 1) >> 1) + (l >> 1)) + (l & 1);
  const float x = hi_diff(p.x, c.x, unit), y = hi_diff(p.y, c.y, unit), z = hi_diff(p.z, c.z, unit);
  r[0] = x;
  r[2] = y;
  r[4] = z;
  r[6] = wt;
  if (l == np - 1 && !(l & 1)) {
    r[1] = x;
    r[3] = y;
    r[5] = z;
    r[7] = 0.f;
  }
}

// Global index of an item's bead t, of its subunit s: a run of subunits, or subunits dealt to the CTAs
// (first[s]: the subunit's first bead less s np).
struct RunBeads {
  int bead0;
  __device__ __forceinline__ int operator()(int, int t) const { return bead0 + t; }
};
struct DealtBeads {
  const int* first;
  __device__ __forceinline__ int operator()(int s, int t) const { return first[s] + t; }
};

// What the warps of a CTA share: the position of the chunk queue and the numbers of pieces of the
// inter-subunit lists.  Zero before force_rows.
struct ForceQueue {
  int next, n_long, n_full, n_short;
};
constexpr int kPiece = 16;    // pairs of a piece: two for each of eight lanes
// Lists above this length are one piece, for a whole warp (m.rows has room for three pieces).
// From 32 or 16 pairs on instead: 64 subunits 1,390 -> 1,414 and 1,515 us per 100 steps, 2,000 of them
// 3,190 -> 3,337 and 3,391, 64 replicas 5,485 -> 5,910 and 6,420 per 20 steps.
constexpr int kLongRow = 48;

// The beads' inter-subunit lists in pieces into m.rows: whole lists above kLongRow pairs (at 0 ..),
// pieces of 9 to 16 pairs (at nbead ..) and of at most 8 (from 4 nbead down), each as
// bead | first pair / kPiece << 16 | pairs << 18.  Lists differ in length from bead to bead, and lanes
// that share a chunk wait for its longest piece.  (Order does not matter: every sum is exact.)  The
// caller's next barrier makes them visible.  thread: this thread's place among the CTA's.
template <class Beads>
__device__ __forceinline__ void force_rows(const ForceArgs& a, const ForceSmem& m, const Beads& bead, int nbead, int thread,
                                           ForceQueue* q) {
  const int lane = threadIdx.x & 31;
  const unsigned int below = (1u << lane) - 1u;
  for (int base = thread - lane; base < nbead; base += blockDim.x) {
    const int t = base + lane;
    const int n = t < nbead ? __ldg(a.inter_count + bead(fast_div(t, a.div_np), t)) : 0;
    if (!__any_sync(0xffffffffu, n > 0)) continue;
    const int cut = n <= kLongRow ? n : 0, rest = cut & (kPiece - 1);
    const int full = (cut + 7) / kPiece;  // pieces of 9 to 16 pairs
    const bool sh = rest > 0 && rest <= 8;
    const unsigned int lg = __ballot_sync(0xffffffffu, n > kLongRow), sb = __ballot_sync(0xffffffffu, sh);
    const unsigned int f1 = __ballot_sync(0xffffffffu, full > 0), f2 = __ballot_sync(0xffffffffu, full > 1),
                       f3 = __ballot_sync(0xffffffffu, full > 2);
    int at = 0;
    if (lane == 0) at = atomicAdd(&q->n_long, __popc(lg));
    if (lane == 1) at = atomicAdd(&q->n_full, __popc(f1) + __popc(f2) + __popc(f3));
    if (lane == 2) at = atomicAdd(&q->n_short, __popc(sb));
    const int l0 = __shfl_sync(0xffffffffu, at, 0) + __popc(lg & below);
    const int s0 = __shfl_sync(0xffffffffu, at, 2) + __popc(sb & below);
    const int f0 = __shfl_sync(0xffffffffu, at, 1) + __popc(f1 & below) + __popc(f2 & below) + __popc(f3 & below);
    if (n > kLongRow) m.rows[l0] = t | n << 18;
    for (int k = 0; k < full; k++) m.rows[nbead + f0 + k] = t | k << 16 | min(kPiece, cut - k * kPiece) << 18;
    if (sh) m.rows[4 * nbead - 1 - s0] = t | full << 16 | rest << 18;
  }
}

// Edge t of the item: length vector and stretching coefficient (len0 - l) ks / l (BEAD::
// update_stretching_force, src/bead.cpp:17-23, EDGE::update_length, src/edge.cpp:35-49).
__device__ __forceinline__ void force_edge(const ForceArgs& a, const SysParams& P, const ForceSmem& m, int t) {
  const TplLayout& L = a.L;
  const int s = fast_div(t, a.div_ne), e = t - s * L.ne;
  const int pk = m.tpl_i[L.o_edge + e];
  const int4* sp = m.pos + s * L.np;
  const float3 lv = dvec(sp[pk & 0xffff], sp[pk >> 16], P.unit32);
  const float l = sqrtf(dot3(lv, lv));
  const float coef = (m.tpl_f[L.o_len0 + e] - l) * P.ks / l;
  m.edge[t] = make_float4(lv.x, lv.y, lv.z, coef);
}

// Rest-angle option (no reference counterpart): E = kb (1 - cos(beta - beta0)) with beta the signed
// bend angle of (across0, b0, b1, across1); -dE/dx = -kb sin(beta - beta0) dbeta/dx, dbeta/dx the
// dihedral gradient (Blondel and Karplus 1996).  Out of line: it runs only for templates with a
// rest shape.
__device__ __noinline__ void force_quad_rest(const SysParams& P, int4 Q0, int4 Q1, int4 Q2, int4 Q3, float beta0, float4* o) {
  const float unit = P.unit32;
  const float3 v1 = dvec(Q0, Q2, unit), v2 = dvec(Q1, Q0, unit), v3 = dvec(Q3, Q1, unit);
  const float3 m = cross3(v1, v2), n = cross3(v2, v3);
  const float l2 = dot3(v2, v2), nv2 = sqrtf(l2);
  const float beta = atan2f(-nv2 * dot3(v1, n), -dot3(m, n));
  const float c = -P.kb * sinf(beta - beta0);
  const float3 ga0 = m * (-nv2 / dot3(m, m)), ga1 = n * (nv2 / dot3(n, n));
  const float p = dot3(v1, v2) / l2, q = dot3(v3, v2) / l2;
  const float3 gb0 = ga0 * (-(1.0f + p)) + ga1 * q, gb1 = ga0 * p - ga1 * (1.0f + q);
  o[0] = make_float4(gb0.x * c, gb0.y * c, gb0.z * c, 0.f);
  o[1] = make_float4(gb1.x * c, gb1.y * c, gb1.z * c, 0.f);
  o[2] = make_float4(ga0.x * c, ga0.y * c, ga0.z * c, 0.f);
  o[3] = make_float4(ga1.x * c, ga1.y * c, ga1.z * c, 0.f);
}

// Bending quad t of the item: the four bead contributions of EDGE::update_bending_forces
// (src/edge.cpp:69-188).  The in-place normal flip (src/edge.cpp:78-81) makes S = 4 |A0 . A1|
// whatever the flip history.
__device__ __forceinline__ void force_quad(const ForceArgs& a, const SysParams& P, const ForceSmem& m, int t) {
  const TplLayout& L = a.L;
  const int s = fast_div(t, a.div_nb), k = t - s * L.nbend;
  const int4* sp = m.pos + s * L.np;
  const int4 bq = *reinterpret_cast<const int4*>(m.tpl_i + L.o_bend + 4 * k);
  const int4 P0 = sp[bq.x], P1 = sp[bq.y], P2 = sp[bq.z], P3 = sp[bq.w];
  float4* o = m.bend + (size_t)t * 4;
  const float beta0 = m.tpl_f[L.o_beta0 + k];
  if (beta0 != 0.f) {
    force_quad_rest(P, P0, P1, P2, P3, beta0, o);
    return;
  }
  const float unit = P.unit32;
  // the edge's two faces: area vector 1/2 (b1 - b0) x (b2 - b1) and its magnitude
  const int* f_b = m.tpl_i + L.o_face;
  const int2 bf = *reinterpret_cast<const int2*>(m.tpl_i + L.o_bendf + 2 * k);
  auto face = [&](int f) {
    const int4 p0 = sp[f_b[3 * f]], p1 = sp[f_b[3 * f + 1]], p2 = sp[f_b[3 * f + 2]];
    const float3 A = cross3(dvec(p1, p0, unit), dvec(p2, p1, unit)) * 0.5f;
    return make_float4(A.x, A.y, A.z, sqrtf(dot3(A, A)));
  };
  const float4 F0 = face(bf.x), F1 = face(bf.y);
  const float a0 = F0.w, a1 = F1.w;
  const float S = 4.0f * fabsf(F0.x * F1.x + F0.y * F1.y + F0.z * F1.z);
  const float3 d01 = dvec(P0, P1, unit), d02 = dvec(P0, P2, unit), d03 = dvec(P0, P3, unit);
  const float3 d12 = dvec(P1, P2, unit), d13 = dvec(P1, P3, unit);
  const float sa0 = S / a0, sa1 = S / a1, q0 = 0.25f / a0, q1 = 0.25f / a1;
  const float kk = P.kb / (a0 * a1 * 4.0f);
  {  // role itsB[0]
    float3 d23 = d13, d32 = d13 * -1.0f, d20 = d01 * -1.0f, d21 = d12;
    float3 c1 = cross3(d20, d21), c2 = cross3(d20, d32);
    float3 gs = f3(d23.y * c1.z - d21.y * c2.z + d32.z * c1.y + d21.z * c2.y,
                   d32.x * c1.z + d21.x * c2.z + d23.z * c1.x - d21.z * c2.x,
                   d23.x * c1.y - d21.x * c2.y + d32.y * c1.x + d21.y * c2.x);
    float3 g0 = cross3(d12, cross3(d02, d01)) * (-q0);
    float3 g1 = cross3(d13, cross3(d03, d01)) * (-q1);
    float3 r = (gs - (g0 * sa0 + g1 * sa1)) * kk;
    o[0] = make_float4(r.x, r.y, r.z, 0.f);
  }
  {  // role itsB[1]
    float3 d23 = d03, d32 = d03 * -1.0f, d20 = d01, d21 = d02;
    float3 c1 = cross3(d20, d21), c2 = cross3(d20, d32);
    float3 gs = f3(d23.y * c1.z - d21.y * c2.z + d32.z * c1.y + d21.z * c2.y,
                   d32.x * c1.z + d21.x * c2.z + d23.z * c1.x - d21.z * c2.x,
                   d23.x * c1.y - d21.x * c2.y + d32.y * c1.x + d21.y * c2.x);
    float3 g0 = cross3(d02, cross3(d12, d01)) * q0;
    float3 g1 = cross3(d03, cross3(d13, d01)) * q1;
    float3 r = (gs - (g0 * sa0 + g1 * sa1)) * kk;
    o[1] = make_float4(r.x, r.y, r.z, 0.f);
  }
  {  // role across face 0: r1x = -r13 (the bead of face 1 off the edge)
    float3 gs = cross3(d01, cross3(d01, d13 * -1.0f));
    float3 g0 = cross3(d01, cross3(d02, d01)) * (-q0);
    float3 r = (gs - g0 * sa0) * kk;
    o[2] = make_float4(r.x, r.y, r.z, 0.f);
  }
  {  // role across face 1: r1x = -r12
    float3 gs = cross3(d01, cross3(d01, d12 * -1.0f));
    float3 g1 = cross3(d01, cross3(d03, d01)) * (-q1);
    float3 r = (gs - g1 * sa1) * kk;
    o[3] = make_float4(r.x, r.y, r.z, 0.f);
  }
}

// Intra-subunit Debye-Hueckel row of bead t (same subunit: no LJ, src/forces.cpp:79-80): all
// partners in order, the even and the odd ones in the two lanes of packed FP32 sums; both sums go
// to the bead's limbs.
template <class Beads>
__device__ __forceinline__ void force_intra(const ForceArgs& a, const SysParams& P, const ForceSmem& m, const Beads& bead, int t) {
  const TplLayout& L = a.L;
  const int np = L.np, npp = (np + 1) >> 1, words = L.words;
  const int s = fast_div(t, a.div_np), l = t - s * np;
  const f32x2 nk2 = pack2(-P.kappa, -P.kappa), kap2 = pack2(P.kappa, P.kappa), le2 = pack2(1.44269504f, 1.44269504f);
  const float cut2 = P.ecut_el2;
  const float* rs = m.rel + 8 * s * npp;
  const float* ri = rs + 8 * (l >> 1) + (l & 1);
  const float nx = -ri[0], ny = -ri[2], nz = -ri[4], wi = ri[6];
  const f32x2 nx2 = pack2(nx, nx), ny2 = pack2(ny, ny), nz2 = pack2(nz, nz), wi2 = pack2(wi, wi);
  f32x2 fx = 0, fy = 0, fz = 0;
  const unsigned int* mrow = a.intra_mask + (size_t)bead(s, t) * words;
  const float4* q = reinterpret_cast<const float4*>(rs);
  unsigned int next = __ldg(mrow);
  for (int wd = 0; wd < words; wd++) {
    unsigned int bits = next;
    if (wd + 1 < words) next = __ldg(mrow + wd + 1);
    const int b1 = min(npp, (wd + 1) << 4);
#pragma unroll 2
    for (int p = wd << 4; p < b1; p++, q += 2, bits >>= 2) {
      const float4 xy = q[0], zw = q[1];
      // partner - bead (the sums' sign is turned at the end; every operation is symmetric in it)
      const f32x2 dx = add2(pack2(xy.x, xy.y), nx2), dy = add2(pack2(xy.z, xy.w), ny2), dz = add2(pack2(zw.x, zw.y), nz2);
      const f32x2 r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
      float r2a, r2b;
      unpack2(r2, r2a, r2b);
      const f32x2 ir = pack2(rsqrt_ftz(r2a), rsqrt_ftz(r2b));
      float ea, eb;  // e^(-kappa r) = 2^(-kappa r log2 e)
      unpack2(mul2(mul2(nk2, mul2(r2, ir)), le2), ea, eb);
      const f32x2 ex = pack2(ex2_ftz(ea), ex2_ftz(eb));
      const f32x2 c = mul2(mul2(mul2(mul2(wi2, pack2(zw.z, zw.w)), ex), mul2(ir, ir)), add2(kap2, ir));
      float ca, cb;
      unpack2(c, ca, cb);
      ca = (bits & 1u) && r2a < cut2 ? ca : 0.f;
      cb = (bits & 2u) && r2b < cut2 ? cb : 0.f;
      const f32x2 cc = pack2(ca, cb);
      fx = fma2(dx, cc, fx);
      fy = fma2(dy, cc, fy);
      fz = fma2(dz, cc, fz);
    }
  }
  float xe, xo, ye, yo, ze, zo;
  unpack2(fx, xe, xo);
  unpack2(fy, ye, yo);
  unpack2(fz, ze, zo);
  if (force_bad(xe, ye, ze) || force_bad(xo, yo, zo)) atomicOr(a.err, kErrNonFinite);
  limbs_add(m.F + 9 * t, f32_to_fx32(-xe) + f32_to_fx32(-xo));
  limbs_add(m.F + 9 * t + 3, f32_to_fx32(-ye) + f32_to_fx32(-yo));
  limbs_add(m.F + 9 * t + 6, f32_to_fx32(-ze) + f32_to_fx32(-zo));
}

// The sums of kLanes (4 or 8) lanes' force vectors, or (whole) the warp's, added to a bead's limbs: the
// nine limbs are halved among the lanes while they are summed, ten exchanges (8 lanes) and two
// atomics of distinct addresses; nine atomics of eight lanes on one address each cost 72
// shared-memory cycles.
template <int kLanes>
__device__ __forceinline__ void limbs_add_lanes(unsigned int* F, long long x, long long y, long long z, bool valid, bool whole) {
  const int lane = threadIdx.x & 31;
  const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
  const unsigned int v[9] = {(unsigned int)(x & 0x1FFFFF), (unsigned int)((x >> 21) & 0x1FFFFF), (unsigned int)(int)(x >> 42),
                             (unsigned int)(y & 0x1FFFFF), (unsigned int)((y >> 21) & 0x1FFFFF), (unsigned int)(int)(y >> 42),
                             (unsigned int)(z & 0x1FFFFF), (unsigned int)((z >> 21) & 0x1FFFFF), (unsigned int)(int)(z >> 42)};
  unsigned int w[5], u[3];
#pragma unroll
  for (int k = 0; k < 5; k++) {  // limbs 0-4 to the even lanes, 5-8 to the odd
    const unsigned int lo = v[k], hi = k < 4 ? v[5 + k] : 0u;
    w[k] = (b0 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b0 ? lo : hi, 1);
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const unsigned int lo = w[k], hi = k < 2 ? w[3 + k] : 0u;
    u[k] = (b1 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b1 ? lo : hi, 2);
  }
  F += (b0 ? 5 : 0) + (b1 ? 3 : 0);
  int n = b1 ? (b0 ? 1 : 2) : 3;  // how many of the values are limbs
  if (kLanes == 8) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned int lo = u[k], hi = k < 1 ? u[2] : 0u;
      u[k] = (b2 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b2 ? lo : hi, 4);
    }
    F += b2 ? 2 : 0;
    n = b2 ? max(0, n - 2) : min(n, 2);
  }
  if (whole) {
#pragma unroll
    for (int o = kLanes; o <= 16; o <<= 1)
#pragma unroll
      for (int k = 0; k < (kLanes == 8 ? 2 : 3); k++) u[k] += __shfl_xor_sync(0xffffffffu, u[k], o);
    valid = valid && lane < kLanes;
  }
#pragma unroll
  for (int k = 0; k < (kLanes == 8 ? 2 : 3); k++)
    if (valid && n > k) atomicAdd(F + k, u[k]);
}

// LJ or WCA term of a pair (src/forces.cpp:81-138) added to its force coefficient.
__device__ __forceinline__ float lj_add(float c, float r2, const float* pair, float elj_att) {
  const float eps = pair[2] < 0.f ? elj_att : pair[2];
  const float ir2 = 1.0f / r2;
  const float s6 = pair[1] * ir2 * ir2 * ir2;
  c += 48.0f * eps * s6 * (s6 - 0.5f) * ir2;
  return c;
}

// Inter-subunit pairs (DH + LJ/WCA, src/forces.cpp:81-138) of a chunk: 32 / kLanes pieces by kLanes
// lanes each, or one long list by the whole warp.  A lane evaluates two of its piece's pairs at a time
// in packed FP32, adds its pair forces exactly in 2^-32 fixed point in registers, and the lanes' sums
// go to the bead's limbs at the end (order-independent).  In small systems what bounds it is the chain
// of loads and arithmetic from one pair to the next, and of a few crowded subunits' CTAs, which
// everyone else waits for; in large ones the instructions.  So a list is spread over lanes:
// neighbouring lanes read neighbouring partners, no lane searches for its bead, and lanes finish
// together.  Eight lanes take a piece in one round (the chain); four in two, with half the work of
// adding up (the instructions): the run form of the force kernel.
// Against runs of eight consecutive pairs of the flat pair sequence per thread: 2,000 subunits, a
// tenth of them in contact, 3,900 -> 3,450 us per 100 steps; 64: 1,870 -> 1,490; a force evaluation of
// 64 dense replicas (17,286 subunits) 222 -> 203 us.
// kFresh: the partners' positions are rewritten by other CTAs while this kernel runs (read past L1).
// wait: called once the first partners are known, before their positions are read.
template <bool kFresh, int kLanes, class Beads, class Wait>
__device__ __forceinline__ void force_inter(const ForceArgs& a, const SysParams& P, const ForceSmem& m, int nbead, const Beads& bead,
                                            const ForceQueue& q, int chunk, Wait wait) {
  const TplLayout& L = a.L;
  const int lane = threadIdx.x & 31;
  const int* species = m.tpl_i + L.o_species;
  const float unit = P.unit32, ecut_el2 = P.ecut_el2;
  constexpr int kRows = 32 / kLanes;
  const bool whole = chunk < q.n_long;
  const int lanes = whole ? 32 : kLanes;
  int at = chunk;  // the piece's place in m.rows
  bool valid = true;
  if (!whole) {
    const int kf = (q.n_full + kRows - 1) / kRows, c = chunk - q.n_long;
    if (c < kf) {
      const int k = kRows * c + lane / kLanes;
      valid = k < q.n_full;
      at = nbead + k;
    } else {
      const int k = kRows * (c - kf) + lane / kLanes;
      valid = k < q.n_short;
      at = 4 * nbead - 1 - k;
    }
  }
  const int rec = valid ? m.rows[at] : 0;
  const int b = rec & 0xffff, n = rec >> 18;
  const int sub = fast_div(b, a.div_np), g = bead(sub, b);
  const int* ids = a.inter_ids + (long long)g * a.inter_cap + ((rec >> 16) & 3) * kPiece;
  const int4 pi = m.pos[b];
  const int l = b - sub * L.np;
  const int si = species[l] * L.nspecies;
  const float wi = m.w[l];
  const f32x2 nk2 = pack2(-P.kappa, -P.kappa), kap2 = pack2(P.kappa, P.kappa), le2 = pack2(1.44269504f, 1.44269504f),
              wi2 = pack2(wi, wi);
  // (past the row's end: the bead itself, dropped below)
  auto partner = [&](int i) { return i < n ? __ldg(ids + i) : g; };
  auto position = [&](int j) { return kFresh ? __ldcg(&a.pos32[j]) : __ldg(&a.pos32[j]); };
  int i = lane & (lanes - 1);
  int j0 = partner(i), j1 = partner(i + lanes);
  if (kFresh) {
    asm volatile("" ::"r"(j0), "r"(j1));  // (loaded before the wait)
    wait();
  }
  unsigned long long ax = 0, ay = 0, az = 0;
  int added = 0;  // values added by fx_add2
  while (i < n) {
    const int4 p0 = position(j0), p1 = position(j1);
    const bool two = i + lanes < n;
    i += 2 * lanes;
    j0 = partner(i);  // the next two pairs' partners, while these are evaluated
    j1 = partner(i + lanes);
    const f32x2 u2 = pack2(unit, unit);
    const f32x2 dx = mul2(pack2((float)(int)((unsigned)pi.x - (unsigned)p0.x), (float)(int)((unsigned)pi.x - (unsigned)p1.x)), u2);
    const f32x2 dy = mul2(pack2((float)(int)((unsigned)pi.y - (unsigned)p0.y), (float)(int)((unsigned)pi.y - (unsigned)p1.y)), u2);
    const f32x2 dz = mul2(pack2((float)(int)((unsigned)pi.z - (unsigned)p0.z), (float)(int)((unsigned)pi.z - (unsigned)p1.z)), u2);
    const f32x2 r2 = fma2(dz, dz, fma2(dx, dx, mul2(dy, dy)));
    float ra, rb;
    unpack2(r2, ra, rb);
    const f32x2 ww = mul2(wi2, pack2(m.w[p0.w], m.w[p1.w]));
    const f32x2 ir = pack2(rsqrt_ftz(ra), rsqrt_ftz(rb));
    float ea, eb;
    unpack2(mul2(mul2(nk2, mul2(r2, ir)), le2), ea, eb);
    const f32x2 c = mul2(mul2(mul2(ww, pack2(ex2_ftz(ea), ex2_ftz(eb))), mul2(ir, ir)), add2(kap2, ir));
    float wa, wb, ca, cb;
    unpack2(ww, wa, wb);
    unpack2(c, ca, cb);
    ca = wa != 0.f && ra < ecut_el2 ? ca : 0.f;
    cb = two && wb != 0.f && rb < ecut_el2 ? cb : 0.f;
    const float* qa = m.tpl_f + L.o_pair + 3 * (si + species[p0.w]);  // cut-off squared, sigma^6, epsilon
    const float* qb = m.tpl_f + L.o_pair + 3 * (si + species[p1.w]);
    const bool la = ra < qa[0], lb = two && rb < qb[0];
    if (la || lb) {
      const float ta = lj_add(ca, ra, qa, P.elj_att), tb = lj_add(cb, rb, qb, P.elj_att);
      ca = la ? ta : ca;
      cb = lb ? tb : cb;
    }
    const f32x2 c2 = pack2(ca, cb);
    const f32x2 fx = mul2(dx, c2), fy = mul2(dy, c2), fz = mul2(dz, c2);
    float xa, xb, ya, yb, za, zb;
    unpack2(fx, xa, xb);
    unpack2(fy, ya, yb);
    unpack2(fz, za, zb);
    // (a sum below a bound of one component: every component is)
    if (fabsf(xa) + fabsf(ya) + fabsf(za) + fabsf(xb) + fabsf(yb) + fabsf(zb) < 4.0e6f) {
      fx_add2(ax, fx);
      fx_add2(ay, fy);
      fx_add2(az, fz);
      added += 2;
    } else {  // large or not finite
      const bool bad_a = force_bad(xa, ya, za), bad_b = force_bad(xb, yb, zb);
      if (bad_a || bad_b) atomicOr(a.err, kErrNonFinite);
      if (bad_a) xa = ya = za = 0.f;
      if (bad_b) xb = yb = zb = 0.f;
      ax += (unsigned long long)(f32_to_fx32(xa) + f32_to_fx32(xb));
      ay += (unsigned long long)(f32_to_fx32(ya) + f32_to_fx32(yb));
      az += (unsigned long long)(f32_to_fx32(za) + f32_to_fx32(zb));
    }
  }
  const unsigned long long bias = fx_bias(added);
  ax -= bias;
  ay -= bias;
  az -= bias;
  __syncwarp();
  limbs_add_lanes<kLanes>(m.F + 9 * b, (long long)ax, (long long)ay, (long long)az, n > 0, whole);
}

// Everything that depends on positions alone, in chunks that the warps take from the queue: long
// inter-subunit lists, the intra-subunit rows of 32 beads (900 instructions), 32 bending quads (400),
// pieces of inter-subunit lists, 64 edges (100).  kFresh (the window kernel): the inter-subunit
// pairs come last, and a warp's first one only after wait() -- by then the other CTAs have
// published their new positions while this one worked on its own subunits.
template <bool kFresh, int kLanes, class Beads, class Wait>
__device__ __forceinline__ void force_terms(const ForceArgs& a, const SysParams& P, const ForceSmem& m, const WorkItem& w,
                                            int nbead, const Beads& bead, ForceQueue* q, Wait wait) {
  const TplLayout& L = a.L;
  const int lane = threadIdx.x & 31;
  const int nq = w.nsub * L.nbend, ne = w.nsub * L.ne;
  const int ki = (nbead + 31) >> 5, kq = (nq + 31) >> 5, ke = (ne + 63) >> 6;
  const ForceQueue rows{0, q->n_long, q->n_full, q->n_short};
  constexpr int kRows = 32 / kLanes;
  const int kl = rows.n_long, ks = (rows.n_full + kRows - 1) / kRows + (rows.n_short + kRows - 1) / kRows;
  // the order of the kinds of chunk
  const int first_intra = kFresh ? 0 : kl, first_quad = first_intra + ki;
  const int first_edge = first_quad + kq + (kFresh ? 0 : ks);
  const int total = kl + ki + kq + ks + ke;
  bool waited = false;
  for (;;) {
    int k = 0;
    if (lane == 0) k = atomicAdd(&q->next, 1);
    k = __shfl_sync(0xffffffffu, k, 0);
    if (k >= total) break;
    if (k >= first_intra && k < first_quad) {
      const int t = 32 * (k - first_intra) + lane;
      if (t < nbead) force_intra(a, P, m, bead, t);
    } else if (k >= first_quad && k < first_quad + kq) {
      const int t = 32 * (k - first_quad) + lane;
      if (t < nq) force_quad(a, P, m, t);
    } else if (k >= first_edge && k < first_edge + ke) {
      const int t = 64 * (k - first_edge) + lane;
      if (t < ne) force_edge(a, P, m, t);
      if (t + 32 < ne) force_edge(a, P, m, t + 32);
    } else {
      // the long lists are the first kl of these chunks
      force_inter<kFresh, kLanes>(a, P, m, nbead, bead, rows, kFresh ? k - first_edge - ke : k < kl ? k : k - ki - kq, [&] {
        if (!waited) wait();
        waited = true;
      });
    }
    __syncwarp();
  }
}

// Stretching and bending sums per bead, two threads per bead in different halves of the CTA, added
// to the bead's limbs.
// kAtOnce list entries are fetched together: four where few warps share an SM and each waits for one load
// after the other (20 small subunits 1,155 -> 1,124 us per 100 steps, 64 large ones 1,417 -> 1,380), one
// where instructions count (840,000 beads: 7,338 against 7,495 us per 40 steps).
template <int kAtOnce, class Beads>
__device__ __forceinline__ void force_gather(const ForceArgs& a, const ForceSmem& m, int nbead, const Beads& bead) {
  const TplLayout& L = a.L;
  const int half = blockDim.x >> 1;
  const int h = (int)threadIdx.x >= half ? 1 : 0;
  const int* bead_edges = m.tpl_i + L.o_bead_edges;
  const int* bead_roles = m.tpl_i + L.o_bead_roles;
  for (int t = (int)threadIdx.x - h * half; t < nbead; t += half) {
    const int s = fast_div(t, a.div_np), l = t - s * L.np, g = bead(s, t);
    float3 f = f3(0.f, 0.f, 0.f);
    if (h == 0) {  // stretching, in the bead's edge order
      for (int k = 0; k < L.maxdeg; k += kAtOnce) {
        int e[kAtOnce];
        float4 E[kAtOnce];
#pragma unroll
        for (int j = 0; j < kAtOnce; j++) e[j] = k + j < L.maxdeg ? bead_edges[l * L.maxdeg + k + j] : -1;
        if (e[0] < 0) break;
#pragma unroll
        for (int j = 0; j < kAtOnce; j++) E[j] = m.edge[s * L.ne + (max(e[j], 0) & 0xffff)];
#pragma unroll
        for (int j = 0; j < kAtOnce; j++) {
          const float c = __int_as_float(__float_as_int(E[j].w) ^ ((e[j] >> 16) << 31));  // minus for the edge's second bead
          if (e[j] >= 0) f = f + f3(E[j].x, E[j].y, E[j].z) * c;
        }
      }
      if (a.sfx) { a.sfx[g] = f.x; a.sfy[g] = f.y; a.sfz[g] = f.z; }
    } else {  // bending, in template edge order
      for (int k = 0; k < L.maxrole; k += kAtOnce) {
        int r[kAtOnce];
        float4 B[kAtOnce];
#pragma unroll
        for (int j = 0; j < kAtOnce; j++) r[j] = k + j < L.maxrole ? bead_roles[l * L.maxrole + k + j] : -1;
        if (r[0] < 0) break;
#pragma unroll
        for (int j = 0; j < kAtOnce; j++) B[j] = m.bend[s * L.nbend * 4 + max(r[j], 0)];
#pragma unroll
        for (int j = 0; j < kAtOnce; j++)
          if (r[j] >= 0) f = f + f3(B[j].x, B[j].y, B[j].z);
      }
      if (a.bfx) { a.bfx[g] = f.x; a.bfy[g] = f.y; a.bfz[g] = f.z; }
    }
    if (force_bad(f.x, f.y, f.z)) atomicOr(a.err, kErrNonFinite);
    long long X = f32_to_fx32(f.x), Y = f32_to_fx32(f.y), Z = f32_to_fx32(f.z);
    if (a.surr_f && h == 0) {  // far-field subunit pairs from the learned surrogate
      const float4 sv = a.surr_f[g];
      if (force_bad(sv.x, sv.y, sv.z)) atomicOr(a.err, kErrNonFinite);
      X += f32_to_fx32(sv.x);
      Y += f32_to_fx32(sv.y);
      Z += f32_to_fx32(sv.z);
    }
    limbs_add(m.F + 9 * t, X);
    limbs_add(m.F + 9 * t + 3, Y);
    limbs_add(m.F + 9 * t + 6, Z);
  }
}

}  // namespace souffle
