// Pair-list rebuild: counting-sort grid of subunit centres, candidate subunits, bead pairs.
//
// Reference: update_pairlist (src/functions.cpp:69-117), called per subunit from
// forceCalculation when step % B == 0 (src/forces.cpp:63-65, src/md.cpp:435-438).  The
// reference tests every subunit pair's centre beads against 1.5 x the list radius
// (|c_i - c_j|^2 < 2.25 r^2), then every bead pair of a passing subunit pair against r^2,
// appending neighbour ids in ascending order.  Here the O(S^2) centre scan becomes a
// counting-sort cell grid (cell edge >= 1.5 r, 27-cell stencil) that yields the same
// candidate set; candidates are sorted so lists come out in the reference's order.
//
// Decisions are exact: a float test on the rounded high words settles every pair farther than
// a safety margin from the cut-off, and the rest are decided in double from the exact 64-bit
// fixed-point differences, matching the reference up to long double vs double ties.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"
#include "launch.cuh"

namespace souffle {


__device__ __forceinline__ int cell_coord(long long x, int ncell) {
  unsigned long long u = (unsigned long long)x + 0x8000000000000000ull;  // [0, 2^64) over [-L/2, L/2)
  return (int)__umul64hi(u, (unsigned long long)ncell);
}

__global__ void k_cells_count(CellArgs a) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n_sub_total) return;
  const SysParams& p = a.sys[a.sub_sys[s]];
  int c = s * a.np + p.center_local;
  int n = p.ncell;
  int cx = cell_coord(a.px[c], n), cy = cell_coord(a.py[c], n), cz = cell_coord(a.pz[c], n);
  int cell = p.cell0 + (cx * n + cy) * n + cz;
  a.sub_cell[s] = cell;
  a.sub_rank[s] = atomicAdd(&a.cell_count[cell], 1);
}

// A segment of cell_subs for every cell: each CTA scans its cells' counts and reserves room for all of
// them with one atomic, so the segments' order depends on scheduling (the candidates are sorted
// at the end, and k_cells_sort orders the cells' subunits, so nothing else does).  One CTA per
// system scanning its cells in order took 57 us for the 79,507 cells of 20,000 subunits.
constexpr int kPlacePer = 4;
__global__ void __launch_bounds__(256) k_cells_place(CellArgs a) {
  __shared__ int warp_sums[8];
  __shared__ int s_base;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int i0 = (blockIdx.x * 256 + threadIdx.x) * kPlacePer;
  int v[kPlacePer], sum = 0;
#pragma unroll
  for (int k = 0; k < kPlacePer; k++) {
    v[k] = i0 + k < a.total_cells ? a.cell_count[i0 + k] : 0;
    sum += v[k];
  }
  int x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (threadIdx.x == 0) {
    int total = 0;
    for (int w = 0; w < 8; w++) {
      const int t = warp_sums[w];
      warp_sums[w] = total;
      total += t;
    }
    s_base = total > 0 ? atomicAdd(a.cell_count + a.total_cells, total) : 0;
  }
  __syncthreads();
  int off = s_base + warp_sums[wid] + x - sum;
#pragma unroll
  for (int k = 0; k < kPlacePer; k++) {
    if (i0 + k < a.total_cells) a.cell_start[i0 + k] = off;
    off += v[k];
  }
}

__global__ void k_cells_scatter(CellArgs a) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= a.n_sub_total) return;
  a.cell_subs[a.cell_start[a.sub_cell[s]] + a.sub_rank[s]] = s;
}

// Each cell's subunits in ascending order (the scatter leaves them in the order of its atomics),
// for callers that sum over them in cell order.  A few subunits per cell: insertion sort.
__global__ void k_cells_sort(CellArgs a) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.total_cells) return;
  int* b = a.cell_subs + a.cell_start[c];
  const int m = a.cell_count[c];
  for (int i = 1; i < m; i++) {
    const int v = b[i];
    int k = i - 1;
    for (; k >= 0 && b[k] > v; k--) b[k + 1] = b[k];
    b[k + 1] = v;
  }
}

// Margin (in length^2) within which the float test defers to the exact double test.
__device__ __forceinline__ float pair_margin(float nl2) { return 1e-4f * (1.0f + nl2); }

// One warp per subunit i: lane k scans stencil cell k (27 cells; with fewer than 3 cells per side
// every cell of the system is a neighbour and is scanned once), testing centre distances
// (src/functions.cpp:80-91): in float on the high words, and exactly in double from the 64-bit
// fixed-point differences when the float value lies within a safety margin of the cut-off.  Hits
// are compacted with a warp scan into shared memory and put in ascending order by rank.
// blockDim must be 128 (4 warps).
__global__ void __launch_bounds__(128) k_candidates(CandArgs a) {
  extern __shared__ int s_cand[];  // [4 warps][cap]
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= a.c.n_sub_total) return;  // uniform per warp
  int* buf = s_cand + wib * a.cap;
  const SysParams& p = a.c.sys[a.c.sub_sys[i]];
  const int np = a.c.np, cl = p.center_local;
  const int ci = i * np + cl;
  const long long xi = a.c.px[ci], yi = a.c.py[ci], zi = a.c.pz[ci];
  const int n = p.ncell;
  const int span = (n < 3) ? n : 3;
  const int ncells = span * span * span;
  int s0 = 0, s1 = 0;
  if (lane < ncells) {
    const int dx = lane / (span * span), dy = (lane / span) % span, dz = lane % span;
    const int cx = cell_coord(xi, n), cy = cell_coord(yi, n), cz = cell_coord(zi, n);
    const int gx = (n < 3) ? dx : (cx + dx - 1 + n) % n;
    const int gy = (n < 3) ? dy : (cy + dy - 1 + n) % n;
    const int gz = (n < 3) ? dz : (cz + dz - 1 + n) % n;
    const int cell = p.cell0 + (gx * n + gy) * n + gz;
    s0 = a.c.cell_start[cell];
    s1 = s0 + a.c.cell_count[cell];
  }
  const int4 pci = a.pos32[ci];
  const float pre2f = (float)p.pre2, marg = pair_margin(pre2f);
  auto take = [&](int j) {
    if (j == i) return true;  // r2 = 0 for i == j (src/functions.cpp:90)
    const int cj = j * np + cl;
    const int4 pcj = a.pos32[cj];
    const float fx = hi_diff(pci.x, pcj.x, p.unit32), fy = hi_diff(pci.y, pcj.y, p.unit32),
                fz = hi_diff(pci.z, pcj.z, p.unit32);
    const float r2f = fx * fx + fy * fy + fz * fz;
    if (fabsf(r2f - pre2f) > marg) return r2f < pre2f;
    const double ddx = fixed_diff(xi, a.c.px[cj], p.fx_to_len);
    const double ddy = fixed_diff(yi, a.c.py[cj], p.fx_to_len);
    const double ddz = fixed_diff(zi, a.c.pz[cj], p.fx_to_len);
    return (ddx * ddx + ddy * ddy + ddz * ddz) < p.pre2;
  };
  int nh = 0;  // pass 1: count this lane's hits
  for (int k = s0; k < s1; k++) nh += take(a.c.cell_subs[k]) ? 1 : 0;
  // warp exclusive scan of hit counts
  int x = nh;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const int total = __shfl_sync(0xffffffffu, x, 31);
  int off = x - nh;  // pass 2: write at the lane's offset
  for (int k = s0; k < s1 && off < a.cap; k++) {
    const int j = a.c.cell_subs[k];
    if (take(j)) buf[off++] = j;
  }
  __syncwarp();
  const int cnt = total < a.cap ? total : a.cap;
  if (lane == 0 && total > a.cap) atomicOr(a.err, kErrCandOverflow);
  // rank sort (ids are distinct)
  int* out = a.cand + (size_t)i * a.cap;
  for (int k = lane; k < cnt; k += 32) {
    const int v = buf[k];
    int r = 0;
    for (int m = 0; m < cnt; m++) r += (buf[m] < v);
    out[r] = v;
  }
  if (lane == 0) a.cand_count[i] = cnt;
}



// r2 < lim from the exact fixed-point differences of beads ga and gb (global indices); out of line:
// only separations within the FP32 test's margin come here.
__device__ __noinline__ bool pair_exact(const long long* px, const long long* py, const long long* pz, double fx, int ga,
                                        int gb, double lim) {
  const double x = fixed_diff(px[ga], px[gb], fx), y = fixed_diff(py[ga], py[gb], fx), z = fixed_diff(pz[ga], pz[gb], fx);
  return x * x + y * y + z * z < lim;
}

// The pair lists of subunit i, one CTA of 128 threads (64 when the candidates are given and a block
// has at most 96 items: launch_pairs).  Candidates are taken in ascending j, so each row's entries come
// out in ascending global id.
//   search   (kSearch: systems of at most kSearchSubs subunits) the candidates by testing every
//            subunit of the system, in order; otherwise they come from k_candidates
//   stage    a chunk of candidates that stay in the pair list (far ones skipped by a warp ballot),
//            their high words in shared memory, and each one's radius about its centre bead
//   masks    every (candidate, row, 32 partners) item at once: FP32 test with a margin, exact FP64
//            inside it; a row farther than R_j + r_list from a candidate's centre has no pair with
//            it (triangle inequality, padded far beyond the rounding)
//   stale    blocks with the system's subunit 0: the stale-distance entries of src/functions.cpp:97
//            replaced (below)
//   append   per row the offsets of the chunk's items, then every item writes its ids
// Subunit i's own block gives the intra bits instead (electrostatic pairs only, :94-96).
//
// Bound by the latency of its rounds of loads and barriers, not by the tests: per-row appending by
// one thread each, two threads' worth of rows per lane and a per-candidate FP64 path for every
// block of subunit 0 took 48 us at 2,688 beads and 47 us at 84,000 in one launch behind four others;
// now 14 us (its search included) and 23 us; a whole rebuild 43 -> 13 us, 64 -> 44 us, and 183 -> 135
// us at 840,000.
//
// The stale-r2 reuse: the reference's test compares a local index with a global id, so a distance is
// recomputed unless (i is subunit 0 and ii is its centre) or (j is subunit 0 and jj is its centre);
// otherwise the r2 of the most recently computed pair (row-major over the visited pairs of the
// block) is reused, starting from the centre-centre distance (or 0 when i == j).  So the centre
// row of subunit 0 takes one value for all its entries -- the last computed pair of the rows
// before it -- and every other row's entry in the centre column of subunit 0 takes the computed
// pair before it in the row, or, when there is none, that of the rows before.
constexpr int kSearchSubs = 1024;
template <bool kSearch>
__global__ void __launch_bounds__(128) k_pairs(PairArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int np = a.np, words = a.words, chunk = a.chunk;
  int4* s_own = reinterpret_cast<int4*>(smem_raw);                                        // [np]
  int4* c32 = s_own + np;                                                                 // [chunk np]
  unsigned int* cmask = reinterpret_cast<unsigned int*>(c32 + (size_t)chunk * np);        // [chunk np words]
  int* coff = reinterpret_cast<int*>(cmask + (size_t)chunk * np * words);                 // [chunk np]
  int* s_n = coff + chunk * np;                                                           // [np] inter entries so far
  int* s_cand = s_n + np;                                                                 // [cand_cap] (kSearch)
  __shared__ unsigned int s_chg[kMaxNp / 32];  // charged beads
  __shared__ int s_cj[kPairChunkMax], s_ctl[2], s_word[5];
  __shared__ float s_cR[kPairChunkMax];

  const int i = blockIdx.x;
  const SysParams& p = a.sys[a.sub_sys[i]];
  const int i_local = i - p.sub0;  // subunit index inside its system
  const int cl = p.center_local;
  const float unit = p.unit32, nl2f = p.nl2_f, margin = pair_margin(nl2f);
  const float r_list = sqrtf(nl2f), eps = 1e-3f * (1.0f + r_list);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned int* mask_rows = a.intra_mask + (size_t)i * np * words;
  for (int t = threadIdx.x; t < np; t += blockDim.x) {
    s_own[t] = a.pos32[(size_t)i * np + t];
    s_n[t] = 0;
  }
  for (int t = threadIdx.x; t < np * words; t += blockDim.x) mask_rows[t] = 0u;
  for (int w = wid; w < words; w += nw) {
    const int l = 32 * w + lane;
    const unsigned int m = __ballot_sync(0xffffffffu, l < np && a.q[l < np ? l : 0] != 0.0f);
    if (lane == 0) s_chg[w] = m;
  }
  int ncand = 0;
  if (kSearch) {
    // centre distances to every subunit of the system (src/functions.cpp:80-91)
    const int ci = i * np + cl;
    const int4 pci = a.pos32[ci];
    const float pre2f = (float)p.pre2, marg = pair_margin(pre2f);
    for (int base = 0; base < p.n_sub; base += 128) {
      const int j = p.sub0 + base + threadIdx.x;
      bool take = false;
      if (base + (int)threadIdx.x < p.n_sub) {
        const int cj = j * np + cl;
        const int4 pcj = a.pos32[cj];
        const float fx = hi_diff(pci.x, pcj.x, unit), fy = hi_diff(pci.y, pcj.y, unit), fz = hi_diff(pci.z, pcj.z, unit);
        const float r2f = fx * fx + fy * fy + fz * fz;
        take = j == i || (fabsf(r2f - pre2f) > marg ? r2f < pre2f : pair_exact(a.px, a.py, a.pz, p.fx_to_len, ci, cj, p.pre2));
      }
      const unsigned int m = __ballot_sync(0xffffffffu, take);
      if (lane == 0) s_word[wid] = __popc(m);
      __syncthreads();
      int off = ncand, total = 0;
      for (int q = 0; q < 4; q++) {
        if (q < wid) off += s_word[q];
        total += s_word[q];
      }
      off += __popc(m & ((1u << lane) - 1u));
      if (take && off < a.cand_cap) s_cand[off] = j;
      ncand += total;
      __syncthreads();
    }
    if (ncand > a.cand_cap) {
      if (threadIdx.x == 0) atomicOr(a.err, kErrCandOverflow);
      ncand = a.cand_cap;
    }
  } else {
    ncand = a.cand_count[i];
  }
  const int* cand = kSearch ? s_cand : a.cand + (size_t)i * a.cand_cap;
  const bool skip_far = !kSearch && a.cand_far && *a.far_ok;

  // partners of row ii of this subunit among 32 beads w0 .. of the staged subunit at b32 (global
  // subunit j): FP32 decisions, then the few within the margin exactly
  auto test_word = [&](int ii, const int4* b32, int j, int w0) {
    const int4 pi = s_own[ii];
    const int n = min(32, np - w0);
    unsigned int bits = 0, unsure = 0;
#pragma unroll 4
    for (int b = 0; b < n; b++) {
      const int4 pj = b32[w0 + b];
      const float dx = hi_diff(pi.x, pj.x, unit), dy = hi_diff(pi.y, pj.y, unit), dz = hi_diff(pi.z, pj.z, unit);
      const float r2f = dx * dx + dy * dy + dz * dz;
      bits |= (unsigned int)(r2f < nl2f) << b;
      unsure |= (unsigned int)!(fabsf(r2f - nl2f) > margin) << b;
    }
    for (; unsure; unsure &= unsure - 1) {
      const int b = __ffs(unsure) - 1;
      const bool in = pair_exact(a.px, a.py, a.pz, p.fx_to_len, i * np + ii, j * np + w0 + b, p.nl2);
      bits = (bits & ~(1u << b)) | (unsigned int)in << b;
    }
    return bits;
  };
  auto test_one = [&](int ii, const int4* b32, int j, int jj) {
    const int4 pi = s_own[ii], pj = b32[jj];
    const float dx = hi_diff(pi.x, pj.x, unit), dy = hi_diff(pi.y, pj.y, unit), dz = hi_diff(pi.z, pj.z, unit);
    const float r2f = dx * dx + dy * dy + dz * dz;
    if (fabsf(r2f - nl2f) > margin) return r2f < nl2f;
    return pair_exact(a.px, a.py, a.pz, p.fx_to_len, i * np + ii, j * np + jj, p.nl2);
  };

  int c = 0;
  while (c < ncand) {
    __syncthreads();  // the previous chunk's readers are done (and the search's list is complete)
    // Warp 0 looks at the next 32 candidates: far ones (left to the surrogate, or beyond every
    // cut-off) are skipped, up to `chunk` others are taken.
    if (wid == 0) {
      const int cc = c + lane;
      const bool valid = cc < ncand;
      const int j = valid ? cand[cc] : -1;
      const bool far = valid && skip_far && a.cand_far[(size_t)i * a.cand_cap + cc];
      const unsigned int take = __ballot_sync(0xffffffffu, valid && !far);
      const int rank = __popc(take & ((1u << lane) - 1u));
      const bool mine = ((take >> lane) & 1u) && rank < chunk;
      if (mine) s_cj[rank] = j;
      const unsigned int last = __ballot_sync(0xffffffffu, mine && rank == chunk - 1);
      if (lane == 0) {
        s_ctl[0] = __popc(take) > chunk ? __ffs(last) : min(32, ncand - c);  // candidates consumed
        s_ctl[1] = min(__popc(take), chunk);
      }
    }
    __syncthreads();
    const int nk = s_ctl[1];
    c += s_ctl[0];
    if (nk == 0) continue;  // only far candidates in this window
    for (int t = threadIdx.x; t < nk * np; t += blockDim.x) {
      const int k = t / np;
      c32[t] = a.pos32[(size_t)s_cj[k] * np + (t - k * np)];
    }
    __syncthreads();
    for (int k = wid; k < nk; k += nw) {  // each candidate's radius about its centre bead
      const int4 pc = c32[k * np + cl];
      float m = 0.0f;
      for (int t = lane; t < np; t += 32) {
        const int4 pt = c32[k * np + t];
        const float dx = hi_diff(pt.x, pc.x, unit), dy = hi_diff(pt.y, pc.y, unit), dz = hi_diff(pt.z, pc.z, unit);
        m = fmaxf(m, dx * dx + dy * dy + dz * dz);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) s_cR[k] = sqrtf(m);
    }
    __syncthreads();
    const int items = nk * np * words;
    const int rows = nk * np;  // items word by word: a warp's lanes have equally many partners to test
    for (int t = threadIdx.x; t < items; t += blockDim.x) {
      const int w = words == 1 ? 0 : t / rows, q = t - w * rows, k = q / np, ii = q - k * np;
      const int j = s_cj[k];
      const int4* b32 = c32 + k * np;
      const int4 pi = s_own[ii], pc = b32[cl];
      const float reach = s_cR[k] + r_list + eps;
      const float ex = hi_diff(pi.x, pc.x, unit), ey = hi_diff(pi.y, pc.y, unit), ez = hi_diff(pi.z, pc.z, unit);
      unsigned int bits = 0;
      if (!(ex * ex + ey * ey + ez * ez > reach * reach)) bits = test_word(ii, b32, j, 32 * w);
      if (j == i) {  // charged pairs of different beads
        bits &= s_chg[w];
        if ((ii >> 5) == w) bits &= ~(1u << (ii & 31));
        if (!((s_chg[ii >> 5] >> (ii & 31)) & 1u)) bits = 0;
      }
      cmask[q * words + w] = bits;
    }
    __syncthreads();
    if (p.quirks) {
      for (int k = 0; k < nk; k++) {
        const int j = s_cj[k];
        const bool i0 = i_local == 0, j0 = j == p.sub0, same = j == i;
        if (!i0 && !j0) continue;  // uniform
        const int4* b32 = c32 + k * np;
        auto visited = [&](int r, int w) {  // partners that the reference's loop looks at in row r
          const unsigned int all = np - 32 * w >= 32 ? 0xffffffffu : (1u << (np - 32 * w)) - 1u;
          if (!same) return all;
          if (!((s_chg[r >> 5] >> (r & 31)) & 1u)) return 0u;
          return s_chg[w] & ~((r >> 5) == w ? 1u << (r & 31) : 0u);
        };
        auto computed = [&](int r, int w) {  // ... and computes a distance for
          if (i0 && r == cl) return 0u;
          return visited(r, w) & ~(j0 && (cl >> 5) == w ? 1u << (cl & 31) : 0u);
        };
        for (int ii = threadIdx.x; ii < np; ii += blockDim.x) {
          unsigned int* mk = cmask + (size_t)(k * np + ii) * words;
          const bool row_stale = i0 && ii == cl;
          if (!row_stale && !(j0 && ((visited(ii, cl >> 5) >> (cl & 31)) & 1u))) continue;
          // the most recently computed pair (fr, fj): before the centre column in this row, else the
          // last one of the rows before
          int fr = -1, fj = -1;
          if (!row_stale) {
            for (int w = cl >> 5; w >= 0 && fj < 0; w--) {
              const unsigned int m = computed(ii, w) & (w == (cl >> 5) ? (1u << (cl & 31)) - 1u : 0xffffffffu);
              if (m) fj = 32 * w + 31 - __clz(m);
            }
            if (fj >= 0) fr = ii;
          }
          for (int r = ii - 1; r >= 0 && fj < 0; r--)
            for (int w = words - 1; w >= 0 && fj < 0; w--) {
              const unsigned int m = computed(r, w);
              if (m) {
                fj = 32 * w + 31 - __clz(m);
                fr = r;
              }
            }
          const bool in = fj >= 0 ? test_one(fr, b32, j, fj) : same || test_one(cl, b32, j, cl);
          if (row_stale) {
            for (int w = 0; w < words; w++) mk[w] = in ? visited(ii, w) : 0u;
          } else {
            const unsigned int b = 1u << (cl & 31);
            mk[cl >> 5] = in ? mk[cl >> 5] | b : mk[cl >> 5] & ~b;
          }
        }
      }
      __syncthreads();
    }
    // own block to the intra bits; the others' entries get their places in the rows
    for (int ii = threadIdx.x; ii < np; ii += blockDim.x) {
      int n = s_n[ii];
      for (int k = 0; k < nk; k++) {
        unsigned int* mk = cmask + (size_t)(k * np + ii) * words;
        coff[k * np + ii] = n;
        if (s_cj[k] == i) {
          for (int w = 0; w < words; w++) mask_rows[ii * words + w] = mk[w];
        } else {
          for (int w = 0; w < words; w++) n += __popc(mk[w]);
        }
      }
      s_n[ii] = n;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < items; t += blockDim.x) {
      const int w = words == 1 ? 0 : t / rows, q = t - w * rows, k = q / np, ii = q - k * np;
      unsigned int bits = cmask[q * words + w];
      const int j = s_cj[k];
      if (!bits || j == i) continue;
      int n = coff[q];
      for (int v = 0; v < w; v++) n += __popc(cmask[q * words + v]);
      int* row = a.inter_ids + (size_t)(i * np + ii) * a.inter_cap;
      const int base = j * np + 32 * w;
      for (; bits && n < a.inter_cap; bits &= bits - 1) row[n++] = base + __ffs(bits) - 1;
    }
  }
  __syncthreads();
  for (int ii = threadIdx.x; ii < np; ii += blockDim.x) {
    const int gi = i * np + ii, n_inter = s_n[ii];
    if (n_inter > a.inter_cap) atomicOr(a.err, kErrInterOverflow);
    a.inter_count[gi] = min(n_inter, a.inter_cap);
    int n_intra = 0;
    for (int w = 0; w < words; w++) n_intra += __popc(mask_rows[ii * words + w]);
    a.ref_len[gi] = n_intra + n_inter;
  }
}

}  // namespace souffle

namespace souffle {
void launch_cells_count(const CellArgs& a, int grid, int block, cudaStream_t s) {
  k_cells_count<<<grid, block, 0, s>>>(a);
}
void launch_cells_place(const CellArgs& a, cudaStream_t s) {
  k_cells_place<<<(a.total_cells + 256 * kPlacePer - 1) / (256 * kPlacePer), 256, 0, s>>>(a);
}
void launch_cells_scatter(const CellArgs& a, int grid, int block, cudaStream_t s) {
  k_cells_scatter<<<grid, block, 0, s>>>(a);
}
void launch_cells_sort(const CellArgs& a, cudaStream_t s) { k_cells_sort<<<(a.total_cells + 127) / 128, 128, 0, s>>>(a); }
void launch_candidates(const CandArgs& a, cudaStream_t s) {
  const int warps_per_block = 4;
  const int g = (a.c.n_sub_total + warps_per_block - 1) / warps_per_block;
  k_candidates<<<g, 32 * warps_per_block, sizeof(int) * warps_per_block * a.cap, s>>>(a);
}
// About 10 KB of staging per CTA (8 candidates of 42 beads), so that a one-wave grid of CTAs still
// fits the shared memory of an SM.
int pair_chunk(int np, int words) {
  const int per = np * (int)(sizeof(int4) + sizeof(unsigned int) * words + sizeof(int));
  return std::max(1, std::min(kPairChunkMax, 10240 / per));
}
static size_t pair_smem_base(int np, int words, int chunk) {
  return sizeof(int4) * (size_t)np * (1 + chunk) + sizeof(unsigned int) * (size_t)chunk * np * words +
         sizeof(int) * (size_t)np * (chunk + 1);
}
// Every subunit of a system is tested by every CTA up to kSearchSubs subunits per system (16 bytes
// per test: 32 MB of L2 reads at 1024, less than 5 us), which replaces four launches (9 to 12 us);
// beyond, and for the surrogate, which classifies the candidates first, they come from the cell grid.
bool pairs_search(int max_sub, int cand_cap) { return max_sub <= kSearchSubs && cand_cap <= 4096; }
size_t pair_smem_bytes(int np, int words, int chunk) { return pair_smem_base(np, words, chunk) + sizeof(int) * 4096; }
// Candidates are given to systems of more than kSearchSubs subunits.  A block with few (row, word) items
// leaves most of 128 threads idle in the search for pairs, and with many subunits the SMs are better
// filled by more CTAs: a whole rebuild with 64 threads against 128, at 42 beads 136 and 147 us (20,000
// subunits), at 10 beads 39 and 42 (3,000), 83 and 102 (20,000), 251 and 337 (80,000); 128 are ahead
// below some 2,500 subunits (42 beads: 46 and 43 us at 2,000, 44 and 38 at 1,100).  With 60 to 100
// beads (128 items and more) the two are alike.
void launch_pairs(const PairArgs& a, int n_sub, bool search, cudaStream_t s) {
  const size_t smem = pair_smem_base(a.np, a.words, a.chunk);
  if (search) k_pairs<true><<<n_sub, 128, smem + sizeof(int) * a.cand_cap, s>>>(a);
  else k_pairs<false><<<n_sub, a.np * a.words <= 96 ? 64 : 128, smem, s>>>(a);
}
cudaError_t set_pairs_smem(size_t smem) {
  const cudaError_t e = raise_smem_limit((const void*)k_pairs<true>, smem);
  return e != cudaSuccess ? e : raise_smem_limit((const void*)k_pairs<false>, smem);
}
}  // namespace souffle
