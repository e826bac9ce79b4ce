// Host side of the C ABI in include/souffle_gpu.h: template derivation, device buffers, launch
// sequences and CUDA-graph windows for the MD loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <numeric>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "souffle_dev.cuh"
#include "souffle_gpu.h"

#include "devbuf.cuh"
#include "kernels.cuh"
#include "surrogate.cuh"
#include "system.cuh"
#include "thermostat.cuh"

using namespace souffle;

namespace {

thread_local std::string g_last_error;

souffle_status fail(souffle_status s, const std::string& msg) {
  g_last_error = msg;
  return s;
}

}  // namespace

namespace souffle {
// Lets entry points defined in other files report through souffle_gpu_last_error().
void record_error(const std::string& msg) { g_last_error = msg; }
}  // namespace souffle

namespace {


#define CUDA_TRY(x)                                                                         \
  do {                                                                                      \
    cudaError_t e_ = (x);                                                                   \
    if (e_ != cudaSuccess)                                                                  \
      return fail(SOUFFLE_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_));     \
  } while (0)

// Signed bend angle of the quad (a0, b0, b1, a1) in positions x [.][3]: the dihedral about b0 -> b1
// shifted so that a flat quad is 0, beta = atan2(-|v2| v1 . n, -m . n) with v1 = x_b0 - x_a0,
// v2 = x_b1 - x_b0, v3 = x_a1 - x_b1, m = v1 x v2, n = v2 x v3.
double bend_angle(const double* x, int b0, int b1, int a0, int a1) {
  double v1[3], v2[3], v3[3], m[3], n[3];
  for (int k = 0; k < 3; k++) {
    v1[k] = x[3 * b0 + k] - x[3 * a0 + k];
    v2[k] = x[3 * b1 + k] - x[3 * b0 + k];
    v3[k] = x[3 * a1 + k] - x[3 * b1 + k];
  }
  auto cross = [](const double* a, const double* b, double* c) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
  };
  cross(v1, v2, m);
  cross(v2, v3, n);
  const double l2 = std::sqrt(v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2]);
  const double y = l2 * (v1[0] * n[0] + v1[1] * n[1] + v1[2] * n[2]);
  const double xx = m[0] * n[0] + m[1] * n[1] + m[2] * n[2];
  const double b = std::atan2(-y, -xx);
  return std::fabs(b) < 1e-12 ? 0.0 : b;
}

souffle_status derive_template(const souffle_template* t, HostTemplate& h) {
  if (!t || t->np <= 0 || t->np > kMaxNp || t->ne < 0 || t->nf < 0 || t->n_lj < 0)
    return fail(SOUFFLE_ERR_BAD_INPUT, "template sizes out of range (np must be 1..256)");
  h.np = t->np;
  h.ne = t->ne;
  h.nf = t->nf;
  h.n_lj = t->n_lj;
  h.type.assign(t->bead_type, t->bead_type + h.np);
  h.q.assign(t->bead_charge, t->bead_charge + h.np);
  h.sigma.assign(t->bead_sigma, t->bead_sigma + h.np);
  h.mass.assign(t->bead_mass, t->bead_mass + h.np);
  h.edge.assign(t->edge_beads, t->edge_beads + 2 * h.ne);
  h.edge_type.assign(t->edge_type, t->edge_type + h.ne);
  h.len0.assign(t->edge_len0, t->edge_len0 + h.ne);
  h.face.assign(t->face_beads, t->face_beads + 3 * h.nf);
  h.lj.assign(t->lj_types, t->lj_types + 2 * h.n_lj);
  if (h.ne > 0xffff) return fail(SOUFFLE_ERR_BAD_INPUT, "more than 65535 edges");
  for (int v : h.edge)
    if (v < 0 || v >= h.np) return fail(SOUFFLE_ERR_BAD_INPUT, "edge bead index out of range");
  for (int v : h.face)
    if (v < 0 || v >= h.np) return fail(SOUFFLE_ERR_BAD_INPUT, "face bead index out of range");
  for (double m : h.mass)
    if (!(m > 0)) return fail(SOUFFLE_ERR_BAD_INPUT, "bead masses must be positive");
  // face <-> edge matching: a face joins an edge's face list (in face order) when any of its
  // three sides is the edge, in either orientation (src/initialize.cpp:370-401)
  h.edge_f0.assign(h.ne, -1);
  h.edge_f1.assign(h.ne, -1);
  std::vector<int> nfe(h.ne, 0);
  for (int f = 0; f < h.nf; f++) {
    int a = h.face[3 * f], b = h.face[3 * f + 1], c = h.face[3 * f + 2];
    for (int e = 0; e < h.ne; e++) {
      int e0 = h.edge[2 * e], e1 = h.edge[2 * e + 1];
      int hits = 0;
      if (a == e0 && b == e1) hits++;
      else if (a == e1 && b == e0) hits++;
      if (a == e0 && c == e1) hits++;
      else if (a == e1 && c == e0) hits++;
      if (b == e1 && c == e0) hits++;
      else if (b == e0 && c == e1) hits++;
      for (int k = 0; k < hits; k++) {
        if (nfe[e] == 0) h.edge_f0[e] = f;
        else if (nfe[e] == 1) h.edge_f1[e] = f;
        nfe[e]++;
      }
    }
  }
  // bending quads: itsB[0], itsB[1], FACE::across of each face (src/face.cpp:27-34)
  auto across = [&](int f, int b0, int b1) {
    for (int k = 0; k < 3; k++) {
      int b = h.face[3 * f + k];
      if (b != b0 && b != b1) return b;
    }
    return -1;
  };
  for (int e = 0; e < h.ne; e++) {
    if (h.edge_type[e] == 0) continue;
    if (nfe[e] < 2)
      return fail(SOUFFLE_ERR_BAD_INPUT,
                  "bending edge " + std::to_string(e) + " does not have two faces");
    int b0 = h.edge[2 * e], b1 = h.edge[2 * e + 1];
    int r2 = across(h.edge_f0[e], b0, b1), r3 = across(h.edge_f1[e], b0, b1);
    if (r2 < 0 || r3 < 0 || r2 == r3)
      return fail(SOUFFLE_ERR_BAD_INPUT, "degenerate bending quad at edge " + std::to_string(e));
    h.bend_edge.push_back(e);
    h.bend.insert(h.bend.end(), {b0, b1, r2, r3});
    h.bendf.insert(h.bendf.end(), {h.edge_f0[e], h.edge_f1[e]});
    h.beta0.push_back(t->bend_rest_pos ? bend_angle(t->bend_rest_pos, b0, b1, r2, r3) : 0.0);
  }
  // BEAD::itsE order = template edge order (src/initialize.cpp:328-329)
  std::vector<std::vector<int>> be(h.np), br(h.np);
  for (int e = 0; e < h.ne; e++) {
    be[h.edge[2 * e]].push_back(e);
    be[h.edge[2 * e + 1]].push_back(e);
  }
  const int nb = (int)h.bend_edge.size();
  for (int k = 0; k < nb; k++)
    for (int r = 0; r < 4; r++) br[h.bend[4 * k + r]].push_back(4 * k + r);
  for (int i = 0; i < h.np; i++) {
    h.maxdeg = std::max<int>(h.maxdeg, (int)be[i].size() + 1);
    h.maxrole = std::max<int>(h.maxrole, (int)br[i].size() + 1);
  }
  h.bead_edges.assign(h.np * h.maxdeg, -1);
  h.bead_roles.assign(h.np * h.maxrole, -1);
  for (int i = 0; i < h.np; i++) {
    for (size_t k = 0; k < be[i].size(); k++)  // the edge, and whether the bead is its second one
      h.bead_edges[i * h.maxdeg + k] = be[i][k] | (h.edge[2 * be[i][k]] == i ? 0 : 1 << 16);
    for (size_t k = 0; k < br[i].size(); k++) h.bead_roles[i * h.maxrole + k] = br[i][k];
  }
  // species: distinct (type, sigma) pairs
  h.species.assign(h.np, 0);
  for (int i = 0; i < h.np; i++) {
    int s = -1;
    for (int k = 0; k < h.nspecies; k++)
      if (h.sp_type[k] == h.type[i] && h.sp_sigma[k] == h.sigma[i]) s = k;
    if (s < 0) {
      if (h.nspecies == kMaxSpecies)
        return fail(SOUFFLE_ERR_BAD_INPUT, "more than 16 distinct (type, diameter) bead species");
      s = h.nspecies++;
      h.sp_type.push_back(h.type[i]);
      h.sp_sigma.push_back(h.sigma[i]);
    }
    h.species[i] = s;
  }
  return SOUFFLE_OK;
}

}  // namespace

namespace {

souffle_status upload(souffle_gpu_system* h) {
  HostTemplate& T = h->tpl;
  TplLayout& L = h->L;
  std::vector<int> ti;
  std::vector<float> tf;
  L.np = T.np;
  L.ne = T.ne;
  L.nf = T.nf;
  L.nbend = (int)T.bend_edge.size();
  L.words = (T.np + 31) / 32;
  L.maxdeg = T.maxdeg;
  L.maxrole = T.maxrole;
  // the bending quads on a 16-byte boundary, their faces on an 8-byte one
  L.o_bend = (int)ti.size();
  ti.insert(ti.end(), T.bend.begin(), T.bend.end());
  L.o_bendf = (int)ti.size();
  ti.insert(ti.end(), T.bendf.begin(), T.bendf.end());
  L.o_face = (int)ti.size();
  ti.insert(ti.end(), T.face.begin(), T.face.end());
  L.o_edge = (int)ti.size();
  for (int e = 0; e < T.ne; e++) ti.push_back(T.edge[2 * e] | (T.edge[2 * e + 1] << 16));
  L.o_bead_edges = (int)ti.size();
  ti.insert(ti.end(), T.bead_edges.begin(), T.bead_edges.end());
  L.o_bead_roles = (int)ti.size();
  ti.insert(ti.end(), T.bead_roles.begin(), T.bead_roles.end());
  L.o_species = (int)ti.size();
  ti.insert(ti.end(), T.species.begin(), T.species.end());
  while (ti.size() % 4) ti.push_back(0);
  L.n_int = (int)ti.size();
  L.nspecies = T.nspecies;
  // directed attraction (src/forces.cpp:119-125) and the type-7 epsilon (src/forces.cpp:127)
  L.type7_bits = 0;
  for (int a = 0; a < T.nspecies; a++) {
    L.lj_att_bits[a] = 0;
    if (T.sp_type[a] == 7) L.type7_bits |= 1 << a;
    for (int b = 0; b < T.nspecies; b++)
      for (int k = 0; k < T.n_lj; k++)
        if (T.sp_type[a] == T.lj[2 * k] && T.sp_type[b] == T.lj[2 * k + 1]) L.lj_att_bits[a] |= 1 << b;
  }
  // pair-species tables (ecut is common to all systems: it depends only on sigma in nm)
  PairTable pt{};
  const double replj2 = 1.12246205 * 1.12246205;
  const double ecut = h->prm[0].ecut;
  for (int a = 0; a < T.nspecies; a++)
    for (int b = 0; b < T.nspecies; b++) {
      const int idx = a * kMaxSpecies + b;
      const double s1 = T.sp_sigma[a], s2 = T.sp_sigma[b], shc = (s1 + s2) / 2;
      const bool att = (L.lj_att_bits[a] >> b) & 1;
      pt.sig6[idx] = (float)(att ? std::pow(s1, 6) : std::pow(shc, 6));
      pt.cut2[idx] = (float)(att ? ecut * ecut : replj2 * shc * shc);
    }
  L.o_len0 = (int)tf.size();
  for (double v : T.len0) tf.push_back((float)v);
  L.o_sigma = (int)tf.size();
  for (double v : T.sigma) tf.push_back((float)v);
  L.o_mass = (int)tf.size();
  for (double v : T.mass) tf.push_back((float)v);
  L.o_beta0 = (int)tf.size();
  for (double v : T.beta0) tf.push_back((float)v);
  L.o_pair = (int)tf.size();
  for (int a = 0; a < T.nspecies; a++)
    for (int b = 0; b < T.nspecies; b++) {
      const bool att = (L.lj_att_bits[a] >> b) & 1;
      tf.push_back(pt.cut2[a * kMaxSpecies + b]);
      tf.push_back(pt.sig6[a * kMaxSpecies + b]);
      tf.push_back(!att ? 1.0f : (L.type7_bits >> b) & 1 ? 50.0f : -1.0f);  // src/forces.cpp:119-130
    }
  while (tf.size() % 4) tf.push_back(0.f);
  L.n_float = (int)tf.size();
  L.o_q = (int)tf.size();
  for (double v : T.q) tf.push_back((float)v);
  CUDA_TRY(h->tpl_i.alloc(ti.size()));
  CUDA_TRY(h->tpl_f.alloc(tf.size()));
  CUDA_TRY(cudaMemcpy(h->tpl_i.p, ti.data(), ti.size() * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(h->tpl_f.p, tf.data(), tf.size() * sizeof(float), cudaMemcpyHostToDevice));

  CUDA_TRY(h->pt.alloc(1));
  CUDA_TRY(cudaMemcpy(h->pt.p, &pt, sizeof(pt), cudaMemcpyHostToDevice));

  // per-system DH weights w = q exp(kappa s/2) / (1 + kappa s/2) sqrt(lb): w_i w_j reproduces
  // q_i q_j lb exp(kappa shc) / ((1 + kappa s_i/2)(1 + kappa s_j/2)) of src/forces.cpp:98-103
  std::vector<float> w(h->n_sys * T.np);
  std::vector<double> wd(h->n_sys * T.np);
  for (int s = 0; s < h->n_sys; s++) {
    const double k = h->prm[s].kappa, lb = h->prm[s].lb;
    for (int i = 0; i < T.np; i++) {
      wd[s * T.np + i] = T.q[i] * std::exp(k * T.sigma[i] / 2) / (1 + k * T.sigma[i] / 2) * std::sqrt(lb);
      w[s * T.np + i] = (float)wd[s * T.np + i];
    }
  }
  CUDA_TRY(h->dh_wd.alloc(wd.size()));
  CUDA_TRY(cudaMemcpy(h->dh_wd.p, wd.data(), wd.size() * sizeof(double), cudaMemcpyHostToDevice));
  CUDA_TRY(h->dh_w.alloc(w.size()));
  CUDA_TRY(cudaMemcpy(h->dh_w.p, w.data(), w.size() * sizeof(float), cudaMemcpyHostToDevice));

  std::vector<dfloat> im(T.np);
  for (int i = 0; i < T.np; i++) im[i] = df_from(1.0 / T.mass[i]);
  CUDA_TRY(h->inv_mass.alloc(T.np));
  CUDA_TRY(cudaMemcpy(h->inv_mass.p, im.data(), T.np * sizeof(dfloat), cudaMemcpyHostToDevice));
  CUDA_TRY(h->mass_d.alloc(T.np));
  CUDA_TRY(cudaMemcpy(h->mass_d.p, T.mass.data(), T.np * sizeof(double), cudaMemcpyHostToDevice));
  CUDA_TRY(h->q_d.alloc(T.np));
  CUDA_TRY(cudaMemcpy(h->q_d.p, T.q.data(), T.np * sizeof(double), cudaMemcpyHostToDevice));
  CUDA_TRY(h->sigma_d.alloc(T.np));
  CUDA_TRY(cudaMemcpy(h->sigma_d.p, T.sigma.data(), T.np * sizeof(double), cudaMemcpyHostToDevice));
  CUDA_TRY(h->len0_d.alloc(std::max(1, T.ne)));
  if (T.ne) CUDA_TRY(cudaMemcpy(h->len0_d.p, T.len0.data(), T.ne * sizeof(double), cudaMemcpyHostToDevice));
  CUDA_TRY(h->type_d.alloc(T.np));
  CUDA_TRY(cudaMemcpy(h->type_d.p, T.type.data(), T.np * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(h->lj_d.alloc(std::max(2, 2 * T.n_lj)));
  if (T.n_lj) CUDA_TRY(cudaMemcpy(h->lj_d.p, T.lj.data(), 2 * T.n_lj * sizeof(int), cudaMemcpyHostToDevice));
  return SOUFFLE_OK;
}

souffle_status check_err(souffle_gpu_system* h) {
  CUDA_TRY(cudaMemcpyAsync(h->err_host, h->err.p, sizeof(unsigned int), cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  const unsigned int e = *h->err_host;
  if (e) {
    CUDA_TRY(cudaMemsetAsync(h->err.p, 0, sizeof(unsigned int), h->stream));
    if (e & kErrWindow) {
      // the counters stand where the launch gave up, and the state is between two steps: part of the
      // positions have moved, velocities and thermostat are those before the window
      h->began = h->have_state = false;
      CUDA_TRY(cudaMemsetAsync(h->win_count.p, 0, sizeof(unsigned int) * h->win_count.n, h->stream));
      CUDA_TRY(cudaMemsetAsync(h->win_acc.p, 0, sizeof(unsigned long long) * h->win_acc.n, h->stream));
      return fail(SOUFFLE_ERR_CUDA, "window kernel: a bounded wait ran out; set the state again");
    }
    if (e & kErrNonFinite) return fail(SOUFFLE_ERR_NONFINITE, "non-finite force or kinetic energy");
    if (e & kErrInterOverflow)
      return fail(SOUFFLE_ERR_NL_OVERFLOW, "inter-subunit pair list exceeded inter_capacity");
    if (e & kErrCandOverflow)
      return fail(SOUFFLE_ERR_NL_OVERFLOW, "candidate subunit list exceeded cand_capacity");
    if (e & kErrSurrogate) return fail(SOUFFLE_ERR_CUDA, "surrogate network: a bounded wait ran out");
  }
  return SOUFFLE_OK;
}

// |mean velocity| removed at the last step (src/md.cpp:505-514, 623)
double vcom_magnitude(const SysState& S) {
  const double x = (double)S.vsum[0] * S.inv_n, y = (double)S.vsum[1] * S.inv_n, z = (double)S.vsum[2] * S.inv_n;
  return std::sqrt(std::fma(z, z, std::fma(x, x, y * y))) * (1.0 / kVelScale);
}

CellArgs cell_args(souffle_gpu_system* h) {
  CellArgs a{};
  a.px = h->pos_fx.p;
  a.py = h->pos_fx.p + h->N;
  a.pz = h->pos_fx.p + 2 * h->N;
  a.sys = h->d_sys.p;
  a.sub_sys = h->d_sub_sys.p;
  a.np = h->tpl.np;

  a.n_sub_total = h->S;
  a.cell_count = h->cell_count.p;
  a.cell_start = h->cell_start.p;
  a.sub_rank = h->sub_rank.p;
  a.sub_cell = h->sub_cell.p;
  a.cell_subs = h->cell_subs.p;
  a.total_cells = h->total_cells;
  a.n_sys = h->n_sys;
  return a;
}

// the grid of subunit centres at the current positions
void launch_subunit_cells(souffle_gpu_system* h) {
  cudaStream_t st = h->stream;
  CellArgs c = cell_args(h);
  cudaMemsetAsync(h->cell_count.p, 0, sizeof(int) * (h->total_cells + 1), st);
  const int tb = 128, gb = (h->S + tb - 1) / tb;
  launch_cells_count(c, gb, tb, st);
  launch_cells_place(c, st);
  launch_cells_scatter(c, gb, tb, st);
}

void launch_candidates_all(souffle_gpu_system* h) {
  cudaStream_t st = h->stream;
  CellArgs c = cell_args(h);
  launch_subunit_cells(h);
  CandArgs ca{};
  ca.c = c;
  ca.pos32 = h->pos32.p;
  ca.cap = h->cand_cap;
  ca.cand = h->cand.p;
  ca.cand_count = h->cand_count.p;
  ca.err = h->err.p;
  launch_candidates(ca, st);
}

void launch_rebuild(souffle_gpu_system* h) {
  cudaStream_t st = h->stream;
  CellArgs c = cell_args(h);
  const bool search = !surrogate_enabled(h) && pairs_search(h->max_sub, h->cand_cap);
  if (!search) launch_candidates_all(h);
  PairArgs pa{};
  pa.px = c.px;
  pa.py = c.py;
  pa.pz = c.pz;
  pa.pos32 = h->pos32.p;
  pa.sys = h->d_sys.p;
  pa.sub_sys = h->d_sub_sys.p;
  pa.q = h->tpl_f.p + h->L.o_q;
  pa.np = h->tpl.np;
  pa.words = h->L.words;

  pa.cand = h->cand.p;
  pa.cand_count = h->cand_count.p;
  pa.cand_cap = h->cand_cap;
  pa.intra_mask = h->intra_mask.p;
  pa.inter_ids = h->inter_ids.p;
  pa.inter_count = h->inter_count.p;
  pa.ref_len = h->ref_len.p;
  pa.inter_cap = h->inter_cap;
  pa.chunk = h->pair_chunk;
  pa.err = h->err.p;
  if (surrogate_enabled(h)) surrogate_classify(h, pa);
  launch_pairs(pa, h->S, search, st);
  if (surrogate_enabled(h)) surrogate_compact(h);
}

// multiplier of fast_div: ceil(2^32 / d), 0 for d <= 1
unsigned int div_magic(int d) { return d > 1 ? (unsigned int)((4294967296ull + d - 1) / d) : 0u; }

ForceArgs force_args(souffle_gpu_system* h, int mode, bool want_parts) {
  ForceArgs a{};
  a.L = h->L;
  a.tpl_i = h->tpl_i.p;
  a.tpl_f = h->tpl_f.p;
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  a.work = h->d_work.p;
  a.sys_slots = h->d_slots.p;
  a.pos32 = h->pos32.p;
  a.intra_mask = h->intra_mask.p;
  a.inter_ids = h->inter_ids.p;
  a.inter_count = h->inter_count.p;
  a.inter_cap = h->inter_cap;
  a.dh_w = h->dh_w.p;
  a.inv_mass = h->inv_mass.p;
  a.kick_c = h->kick_c.p;
  const int64_t N = h->N;
  a.fx = h->force.p;
  a.fy = h->force.p + N;
  a.fz = h->force.p + 2 * N;
  a.vx = h->vel.p;
  a.vy = h->vel.p + N;
  a.vz = h->vel.p + 2 * N;
  if (want_parts) {
    a.sfx = h->sbforce.p;
    a.sfy = h->sbforce.p + N;
    a.sfz = h->sbforce.p + 2 * N;
    a.bfx = h->sbforce.p + 3 * N;
    a.bfy = h->sbforce.p + 4 * N;
    a.bfz = h->sbforce.p + 5 * N;
  }
  a.partial = h->partial.p;
  a.err = h->err.p;
  a.n_beads_total = (int)N;
  a.fdrag = h->bd_fdrag.p;
  a.fran = h->bd_fran.p;
  a.bb_pos32 = h->bb_pos32.p;
  a.chain64 = h->opt.chain_fp64 ? h->chain64.p : nullptr;
  a.max_sub = h->subs_per_cta;
  a.n_items = (int)h->work.size();
  a.ticket = h->force_ticket.p;
  a.div_np = div_magic(h->tpl.np);
  a.div_ne = div_magic(h->L.ne);
  a.div_nb = div_magic(h->L.nbend);
  a.mode = mode;
  return a;
}

DriftArgs drift_args(souffle_gpu_system* h) {
  DriftArgs a{};
  const int64_t N = h->N;
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  a.work = h->d_work.p;
  a.kick_c = h->kick_c.p;
  a.np = h->tpl.np;
  a.fx = h->force.p;
  a.fy = h->force.p + N;
  a.fz = h->force.p + 2 * N;
  a.vx = h->vel.p;
  a.vy = h->vel.p + N;
  a.vz = h->vel.p + 2 * N;
  a.px = h->pos_fx.p;
  a.py = h->pos_fx.p + N;
  a.pz = h->pos_fx.p + 2 * N;
  a.pos32 = h->pos32.p;
  // The idle half of each drift CTA brings the force kernel's pair rows into L2 only when the
  // step's working set (state, forces and about 64 list entries per bead) fits three quarters of
  // the 129 MB L2; in larger runs the rows would be evicted before the force kernel reads them
  // and the prefetch only adds DRAM traffic to the drift.
  const double step_bytes = (double)N * (200.0 + 4.0 * std::min(h->inter_cap, 64));
  a.inter_ids = step_bytes <= 96.0 * 1024 * 1024 ? h->inter_ids.p : nullptr;
  a.inter_count = h->inter_count.p;
  a.inter_cap = h->inter_cap;
  a.intra_mask = h->intra_mask.p;
  a.words = h->L.words;
  a.bd_drag = h->bd_drag.p;
  a.bd_noise = h->bd_noise.p;
  a.lcg_table = h->lcg_table.p;
  a.fdrag = h->bd_fdrag.p;
  a.fran = h->bd_fran.p;
  a.n_total = N;
  return a;
}

// k_drift: a thread per bead; twice as many where the upper half prefetches
void launch_drift_all(souffle_gpu_system* h) {
  const DriftArgs a = drift_args(h);
  const int threads = a.inter_ids ? h->threads : std::min(h->threads, (h->subs_per_cta * h->tpl.np + 31) / 32 * 32);
  launch_drift(a, h->force_grid < (int)h->work.size(), (int)h->work.size(), threads, h->stream);
}

// k_forces, preceded by the surrogate's far-field forces when it is on
void launch_forces_all(souffle_gpu_system* h, int mode, bool want_parts, bool judge = false) {
  ForceArgs fa = force_args(h, mode, want_parts);
  if (surrogate_enabled(h)) {
    surrogate_forces(h, fa);
    if (judge) surrogate_judge(h);
  }
  launch_forces(fa, h->n_sys, h->force_grid, h->threads, h->force_smem, h->stream);
}

void launch_step(souffle_gpu_system* h, bool rebuild, bool judge) {
  launch_drift_all(h);
  if (rebuild) launch_rebuild(h);
  launch_forces_all(h, 1, false, judge);
}


// Steps through the window kernel: MD or Brownian steps with the double-float chain whose forces
// come from the pair lists alone (no network, no big beads), every work item resident at once.
bool window_usable(const souffle_gpu_system* h) {
  if (!h->window_ok || h->opt.chain_fp64 || surrogate_enabled(h)) return false;
  for (const SysParams& P : h->sp)
    if (P.nbb > 0) return false;
  return true;
}
// whole rebuild periods up to this length are one graph
constexpr int kMaxPeriod = 64;

size_t force_smem_for(const souffle_gpu_system* h, int subs, int threads) {
  const TplLayout& L = h->L;
  const int np = h->tpl.np;
  return force_tile_bytes(subs, L.ne, L.nbend) + sizeof(int4) * subs * np + 8 * sizeof(float) * subs * ((np + 1) / 2) +
         sizeof(long long) * 4 * (threads / 32) + sizeof(unsigned int) * force_slot_len(subs * np) +
         sizeof(int) * force_rows_len(subs * np) + sizeof(float) * (np + L.n_float) + sizeof(int) * L.n_int;
}

// Bytes that decide whether a CTA shape is accepted: bonded tile, 72 bytes per bead, reductions and the
// template's tables.  (The kernels' own scratch on top is not counted: plan_work finds room for it.)
bool force_shape_ok(const souffle_gpu_system* h, int subs, int threads) {
  const TplLayout& L = h->L;
  const int np = h->tpl.np;
  auto up4 = [](int n) { return (n + 3) & ~3; };
  const size_t bytes = force_tile_bytes(subs, L.ne, L.nbend) + 32 * (size_t)(subs * np) + 32 * (size_t)(threads / 32) +
                       sizeof(unsigned int) * force_slot_len(subs * np) + sizeof(int) * up4(subs * np + 1) +
                       sizeof(float) * (np + up4(L.ne + 3 * np + L.nbend)) +
                       sizeof(int) * up4(L.ne + 3 * L.nf + 6 * L.nbend + np * (L.maxdeg + L.maxrole + 2));
  return bytes <= 200 * 1024;
}

DealArgs deal_args(souffle_gpu_system* h) {
  return DealArgs{h->inter_count.p, h->S, h->tpl.np, (int)h->work.size(), h->deal_key.p, h->deal_ticket.p, h->deal.p};
}

// `len` steps in one launch; forces_first: the drift of the first one has been launched already
cudaError_t launch_window_steps(souffle_gpu_system* h, int len, bool forces_first) {
  WindowArgs q{};
  q.steps = len;
  q.polls = h->window_polls;
  q.wide = h->window_wide ? 1 : 0;
  q.forces_first = forces_first ? 1 : 0;
  q.n_sys = h->n_sys;
  q.count = h->win_count.p;
  q.acc = h->win_acc.p;
  q.acc_stride = 16 * (size_t)h->n_sys;
  q.deal = h->deal_ok ? h->deal.p : nullptr;
  q.force_bytes = (force_smem_for(h, h->subs_per_cta, h->window_threads) + 15) & ~(size_t)15;
  return launch_window(force_args(h, 1, false), drift_args(h), q, (int)h->work.size(), h->window_threads, h->window_smem, h->stream);
}

// A graph of `len` steps: one window where the handle takes them, else the steps' kernels.  judge_mask: the
// steps after which the surrogate is judged.
cudaError_t capture_steps(souffle_gpu_system* h, int len, bool rebuild_first, unsigned long long judge_mask, cudaGraphExec_t* out) {
  cudaError_t e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  cudaError_t launched = cudaSuccess;
  if (len > 1 && window_usable(h)) {
    if (rebuild_first) {
      launch_drift_all(h);
      launch_rebuild(h);
      if (h->deal_ok) launch_deal(deal_args(h), h->stream);
    }
    launched = launch_window_steps(h, len, rebuild_first);
  } else {
    for (int k = 0; k < len; k++) launch_step(h, k == 0 && rebuild_first, (judge_mask >> k) & 1ull);
  }
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(h->stream, &g);
  if (launched != cudaSuccess) e = launched;
  if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
  if (g) cudaGraphDestroy(g);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

// Work items of up to `subs` subunits of one system each (one force-kernel CTA per item, in
// system order), their partial-sum slots, the force kernel's shared memory, and `threads` threads
// per CTA.  Cached graphs are dropped (their launch shapes change).  Items of more subunits than the
// force kernel's shared memory holds are cut smaller (the results do not depend on the shape).
//
// A single system whose items leave part of one wave of CTAs empty is cut into exactly as many
// items as the wave holds (or one per subunit), of floor or ceil(S / items) subunits with the
// larger ones first.  The block scheduler deals a one-wave grid out round-robin over the SMs, so
// every SM then holds the same number of larger items within one, and the per-SM work is even;
// equal items of `subs` subunits would leave some SMs with one CTA more than others (2000
// subunits in 3-subunit items: 667 CTAs on 152 SMs, 4 or 5 per SM).
souffle_status plan_work(souffle_gpu_system* h, int subs, int threads) {
  if (!force_shape_ok(h, subs, threads)) return fail(SOUFFLE_ERR_BAD_INPUT, "template too large for shared memory");
  while (subs > 1 && force_smem_for(h, subs, threads) > kMaxDynamicSmem) subs--;
  const size_t smem = force_smem_for(h, subs, threads);
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  CUDA_TRY(set_kernel_smem(smem, threads, h->pair_smem));
  int wave = 0, run_wave = 0, win_wave = 0;
  CUDA_TRY(force_wave_ctas(false, threads, smem, &wave));
  CUDA_TRY(force_wave_ctas(true, threads, smem, &run_wave));
  size_t win_smem = window_smem_bytes(smem, subs, h->tpl.np);
  if (win_smem <= kMaxDynamicSmem) CUDA_TRY(window_wave_ctas(false, threads, win_smem, &win_wave));
  std::vector<WorkItem> work;
  std::vector<int2> slots;
  bool even_items = false;  // of floor or ceil(S / items) subunits, the longer ones first
  int sub0 = 0;
  for (int k = 0; k < h->n_sys; k++) {
    const int n = h->prm[k].n_subunits;
    const int first = (int)work.size();
    const int w0 = (n + subs - 1) / subs;
    if (h->n_sys == 1 && wave > w0) {
      even_items = true;
      const int items = std::min(wave, n), q = n / items, r = n % items;
      for (int i = 0, b = 0; i < items; i++) {
        const int len = q + (i < r ? 1 : 0);
        work.push_back(WorkItem{k, sub0 + b, len, (int)work.size()});
        b += len;
      }
    } else {
      for (int b = 0; b < n; b += subs) work.push_back(WorkItem{k, sub0 + b, std::min(subs, n - b), (int)work.size()});
    }
    slots.push_back(make_int2(first, (int)work.size() - first));
    sub0 += n;
  }
  if (h->n_sys > 1) {
    // Systems of a batch differ in pair density, so their items differ in cost: costliest items
    // first (longest-processing-time order), so that the cheap ones fill the SMs at the end of
    // the grid instead of a few long ones running alone.  Estimated cost of a subunit: its
    // beads' intra-subunit pairs plus the inter-subunit pairs inside the list radius at the
    // system's bead density.  Results do not depend on the order (exact integer sums).
    const int np = h->tpl.np;
    std::vector<double> cost(h->n_sys);
    for (int k = 0; k < h->n_sys; k++) {
      const souffle_params& q = h->prm[k];
      const double rho = (double)q.n_subunits * np / (q.box * q.box * q.box);
      const double r = q.nlist_cutoff;
      cost[k] = np + rho * 4.18879 * r * r * r;  // 4/3 pi r^3
    }
    std::stable_sort(work.begin(), work.end(), [&](const WorkItem& x, const WorkItem& y) {
      return cost[x.sys] * x.nsub > cost[y.sys] * y.nsub;
    });
  }
  CUDA_TRY(h->d_work.alloc(work.size()));
  CUDA_TRY(cudaMemcpy(h->d_work.p, work.data(), sizeof(WorkItem) * work.size(), cudaMemcpyHostToDevice));
  CUDA_TRY(h->d_slots.alloc(slots.size()));
  CUDA_TRY(cudaMemcpy(h->d_slots.p, slots.data(), sizeof(int2) * slots.size(), cudaMemcpyHostToDevice));
  CUDA_TRY(h->partial.alloc(4 * work.size()));  // the force kernel's per-system running sums
  CUDA_TRY(cudaMemset(h->partial.p, 0, sizeof(long long) * h->partial.n));
  if (h->force_ticket.n == 0) {
    CUDA_TRY(h->force_ticket.alloc(1));
    CUDA_TRY(cudaMemset(h->force_ticket.p, 0, sizeof(unsigned int)));
  }
  h->work.swap(work);
  h->slots.swap(slots);
  h->subs_per_cta = subs;
  h->threads = threads;
  h->force_smem = smem;
  // more items than one wave of CTAs: the form whose CTAs draw items
  h->force_grid = (int)h->work.size() <= std::max(wave, run_wave) ? (int)h->work.size() : run_wave;
  h->window_ok = (int)h->work.size() <= std::min(win_wave, kWindowMaxCtas);
  h->window_wide = false;
  h->window_threads = threads;
  // Few enough items for CTAs of 64 registers (and no CTA shape asked for): the window kernel takes a warp
  // per chunk of a subunit's work (rows, quads, edges and four beads' lists each), up to 512 threads and
  // down to 256 as the items fit the GPU, so that a crowded subunit, which all others wait for, is done
  // sooner: 64 subunits 1,765 -> 1,645 us per 100 steps, 20 small ones 1,310 -> 1,240 (no spilled
  // registers), 333 Brownian ones 1,053 -> 970 per 50.
  if (h->window_ok && !h->opt.threads_per_cta) {
    const int np = h->tpl.np;
    int ns = 1;
    for (const WorkItem& w : h->work) ns = std::max(ns, w.nsub);
    const int chunks = (ns * np + 31) / 32 + (ns * h->L.nbend + 31) / 32 + (ns * h->L.ne + 31) / 32 + (ns * np + 3) / 4;
    const int most = std::min(512, std::max(128, 32 * chunks));
    for (int wide = most; wide >= std::min(most, 256) && !h->window_wide; wide -= 32) {
      const size_t bytes = window_smem_bytes(force_smem_for(h, subs, wide), subs, np);
      int wide_wave = 0;
      if (bytes <= kMaxDynamicSmem) CUDA_TRY(window_wave_ctas(true, wide, bytes, &wide_wave));
      if ((int)h->work.size() > wide_wave) continue;
      h->window_wide = true;
      h->window_threads = wide;
      win_smem = bytes;
    }
  }
  h->window_smem = win_smem;
  if (h->window_ok && h->win_count.n == 0) {
    CUDA_TRY(h->win_count.alloc(1 + (size_t)h->n_sys));
    CUDA_TRY(h->win_acc.alloc(48 * (size_t)h->n_sys));
    CUDA_TRY(cudaMemset(h->win_count.p, 0, sizeof(unsigned int) * h->win_count.n));
    CUDA_TRY(cudaMemset(h->win_acc.p, 0, sizeof(unsigned long long) * h->win_acc.n));
  }
  // one system cut into items of like length, some of them of several subunits: the window kernel takes
  // the subunits in an order by cost (in order until the first rebuild)
  h->deal_ok = h->window_ok && !h->window_wide && even_items && h->S > (int)h->work.size();
  if (h->deal_ok) {
    std::vector<int> order(h->S);
    std::iota(order.begin(), order.end(), 0);
    if (h->deal.n == 0) {
      CUDA_TRY(h->deal.alloc(h->S));
      CUDA_TRY(h->deal_key.alloc(h->S));
      CUDA_TRY(h->deal_ticket.alloc(1));
      CUDA_TRY(cudaMemset(h->deal_ticket.p, 0, sizeof(unsigned int)));
    }
    CUDA_TRY(cudaMemcpy(h->deal.p, order.data(), sizeof(int) * h->S, cudaMemcpyHostToDevice));
  }
  for (auto& g : h->graphs) cudaGraphExecDestroy(g.second);
  h->graphs.clear();
  return SOUFFLE_OK;
}

}  // namespace

namespace souffle {
souffle_status check_status(souffle_gpu_system* h) { return check_err(h); }
souffle_status rebuild_candidates(souffle_gpu_system* h) {
  launch_candidates_all(h);
  CUDA_TRY(cudaGetLastError());
  return SOUFFLE_OK;
}
}  // namespace souffle

extern "C" {

const char* souffle_gpu_last_error(void) { return g_last_error.c_str(); }

souffle_status souffle_gpu_create(const souffle_template* tpl, const souffle_params* params,
                                  int32_t n_systems, const souffle_options* opts,
                                  souffle_gpu_system** out) {
  if (!out) return fail(SOUFFLE_ERR_BAD_INPUT, "out is NULL");
  *out = nullptr;
  if (!params || n_systems <= 0) return fail(SOUFFLE_ERR_BAD_INPUT, "need at least one system");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return fail(SOUFFLE_ERR_NO_DEVICE, "no CUDA device available");
  std::unique_ptr<souffle_gpu_system> h(new souffle_gpu_system());
  if (opts) h->opt = *opts;
  if (h->opt.device < 0 || h->opt.device >= ndev) return fail(SOUFFLE_ERR_BAD_INPUT, "bad device ordinal");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  souffle_status s = derive_template(tpl, h->tpl);
  if (s != SOUFFLE_OK) return s;
  const int np = h->tpl.np;
  h->n_sys = n_systems;
  h->prm.assign(params, params + n_systems);
  for (int k = 0; k < n_systems; k++) {
    const souffle_params& p = params[k];
    if (p.n_subunits <= 0 || !(p.box > 0) || p.center_local < 0 || p.center_local >= np ||
        p.chain_length < 1 || p.chain_length >= kMaxChain || p.build_freq <= 0 || !(p.dt > 0))
      return fail(SOUFFLE_ERR_BAD_INPUT, "system " + std::to_string(k) + ": parameter out of range");
    if (p.ecut != params[0].ecut)
      return fail(SOUFFLE_ERR_BAD_INPUT, "all systems must share ecut (the bead size in nm)");
    if ((int64_t)h->S + p.n_subunits > (int64_t)1 << 30)
      return fail(SOUFFLE_ERR_BAD_INPUT, "too many subunits");
    h->S += p.n_subunits;
  }
  h->N = (int64_t)h->S * np;
  if (h->N > ((int64_t)1 << 31) - 1) return fail(SOUFFLE_ERR_BAD_INPUT, "too many beads");
  // default inter-subunit capacity: the reference's whole-list capacity (src/md.cpp:231-232),
  // which bounds the inter part of any list the reference can hold
  int ref_cap = 64;
  for (int k = 0; k < n_systems; k++) ref_cap = std::max<int>(ref_cap, params[k].nlist_capacity);
  // (at most kMaxInterPerBead: the force kernel's exact per-bead limb sums hold 2^11 pair forces,
  // and no bead can have more neighbours within a list radius at close packing)
  h->inter_cap = std::min(kMaxInterPerBead, h->opt.inter_capacity > 0 ? h->opt.inter_capacity : ref_cap);
  h->cand_cap = h->opt.cand_capacity > 0 ? h->opt.cand_capacity : 128;
  if (h->opt.threads_per_cta != 0 &&
      (h->opt.threads_per_cta < 64 || h->opt.threads_per_cta > 256 || h->opt.threads_per_cta % 32))
    return fail(SOUFFLE_ERR_BAD_INPUT, "threads_per_cta must be 64..256 in steps of 32");
  if (h->opt.subunits_per_cta < 0 || h->opt.subunits_per_cta > 16)
    return fail(SOUFFLE_ERR_BAD_INPUT, "subunits_per_cta must be 0..16");
  h->threads = h->opt.threads_per_cta ? h->opt.threads_per_cta : 256;  // two threads per bead
  h->subs_per_cta = h->opt.subunits_per_cta ? h->opt.subunits_per_cta : std::max(1, 128 / np);

  // per-system constants, cell grids, work items
  int sub0 = 0, cell0 = 0;
  std::vector<int> sub_sys(h->S), bead_sys(h->N);
  for (int k = 0; k < n_systems; k++) {
    const souffle_params& p = params[k];
    SysParams q{};
    q.box = p.box;
    q.fx_to_len = p.box / (kTwo32 * kTwo32);
    q.len_to_fx = (kTwo32 * kTwo32) / p.box;
    q.unit32 = (float)(p.box / kTwo32);
    q.ks = (float)p.ks;
    q.kb = (float)p.kb;
    q.ks_d = p.ks;
    q.kb_d = p.kb;
    q.kappa = (float)p.kappa;
    q.ecut2 = (float)(p.ecut * p.ecut);
    q.ecut_el2 = p.ecut_el != 0 ? (float)(p.ecut_el * p.ecut_el) : INFINITY;
    q.elj_att = (float)p.elj_att;
    q.nl2 = p.nlist_cutoff * p.nlist_cutoff;
    q.nl2_f = (float)q.nl2;
    q.pre2 = q.nl2 * 2.25;
    q.bead0 = sub0 * np;
    q.sub0 = sub0;
    q.n_sub = p.n_subunits;
    // cell edge >= sqrt(pre2) = 1.5 r (src/functions.cpp:91); at most 256 cells per side
    int nc = (int)std::floor(p.box / std::sqrt(q.pre2));
    nc = std::max(1, std::min(nc, 256));
    q.ncell = nc;
    q.cell0 = cell0;
    q.quirks = (h->opt.compat_quirks >= 0) ? 1 : 0;
    q.center_local = p.center_local;
    q.dt = p.dt;
    // x_fixed advances by v dt 2^64 / L = v_fixed dt 2^24 / L (v_fixed in 2^-40 units): the
    // multiplier, itself in 2^-40 units
    const double dx = p.dt * 16777216.0 / p.box;
    if (!(dx < 8388608.0))
      return fail(SOUFFLE_ERR_BAD_INPUT, "time step too large for the box (dt 2^24 / L >= 2^23)");
    q.drift_fx = (long long)std::llrint(dx * 1099511627776.0);
    q.brownian = p.brownian ? 1 : 0;
    if (p.brownian && !(p.damp > 0)) return fail(SOUFFLE_ERR_BAD_INPUT, "Brownian dynamics needs damp > 0");
    for (int i = 0; i < np; i++)
      if (!(0.5 * p.dt * 1.5 / tpl->bead_mass[i] < 0.45))  // kick coefficient below 0.49 * 2^64
        return fail(SOUFFLE_ERR_BAD_INPUT, "dt / (2 m) too large for the fixed-point kick");
    h->sp.push_back(q);
    for (int i = 0; i < p.n_subunits; i++) sub_sys[sub0 + i] = k;
    for (int i = 0; i < p.n_subunits * np; i++) bead_sys[(int64_t)sub0 * np + i] = k;
    sub0 += p.n_subunits;
    cell0 += nc * nc * nc;
  }
  h->total_cells = cell0;
  CUDA_TRY(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
  s = upload(h.get());
  if (s != SOUFFLE_OK) return s;

  const int64_t N = h->N;
  const TplLayout& L = h->L;
  CUDA_TRY(h->d_sys.alloc(n_systems));
  CUDA_TRY(cudaMemcpy(h->d_sys.p, h->sp.data(), sizeof(SysParams) * n_systems, cudaMemcpyHostToDevice));
  CUDA_TRY(h->d_state.alloc(n_systems));
  CUDA_TRY(cudaMemset(h->d_state.p, 0, sizeof(SysState) * n_systems));
  CUDA_TRY(h->d_sub_sys.alloc(h->S));
  CUDA_TRY(cudaMemcpy(h->d_sub_sys.p, sub_sys.data(), sizeof(int) * h->S, cudaMemcpyHostToDevice));
  CUDA_TRY(h->d_bead_sys.alloc(N));
  CUDA_TRY(cudaMemcpy(h->d_bead_sys.p, bead_sys.data(), sizeof(int) * N, cudaMemcpyHostToDevice));
  CUDA_TRY(h->pos_fx.alloc(3 * N));
  CUDA_TRY(h->pos32.alloc(N));
  CUDA_TRY(h->vel.alloc(3 * N));
  CUDA_TRY(h->force.alloc(3 * N));
  CUDA_TRY(h->sbforce.alloc(6 * N));
  CUDA_TRY(h->staging.alloc(9 * N));
  CUDA_TRY(h->kick_c.alloc((size_t)n_systems * np));
  CUDA_TRY(cudaMemset(h->kick_c.p, 0, sizeof(long long) * n_systems * np));
  CUDA_TRY(h->intra_mask.alloc((size_t)h->S * np * L.words));
  CUDA_TRY(h->inter_ids.alloc((size_t)h->inter_cap * N));
  CUDA_TRY(h->inter_count.alloc(N));
  CUDA_TRY(h->ref_len.alloc(N));
  CUDA_TRY(h->cand.alloc((size_t)h->cand_cap * h->S));
  CUDA_TRY(h->cand_count.alloc(h->S));
  CUDA_TRY(h->cell_count.alloc(h->total_cells + 1));
  CUDA_TRY(h->cell_start.alloc(h->total_cells));
  CUDA_TRY(h->sub_rank.alloc(h->S));
  CUDA_TRY(h->sub_cell.alloc(h->S));
  CUDA_TRY(h->cell_subs.alloc(h->S));
  CUDA_TRY(h->err.alloc(1));
  CUDA_TRY(cudaMemset(h->err.p, 0, sizeof(unsigned int)));
  CUDA_TRY(cudaMallocHost(&h->err_host, sizeof(unsigned int)));
  // Brownian systems (src/md.cpp:415-431, 461-501): drag m / damp and noise scale
  // sqrt(24 m / (damp dt)) per template bead, and minstd_rand0 skip-ahead multipliers
  for (int k = 0; k < n_systems; k++) h->any_brownian = h->any_brownian || params[k].brownian;
  if (h->any_brownian) {
    std::vector<long long> drag((size_t)n_systems * np, 0);
    std::vector<double> noise((size_t)n_systems * np, 0.0);
    int max_n = 0;
    for (int k = 0; k < n_systems; k++) {
      const souffle_params& p = params[k];
      max_n = std::max(max_n, p.n_subunits * np);
      if (!p.brownian) continue;
      for (int l = 0; l < np; l++) {
        const double m = tpl->bead_mass[l];
        drag[(size_t)k * np + l] = std::llrint(m / p.damp * 1099511627776.0);  // 2^40
        noise[(size_t)k * np + l] = std::sqrt((m * 24.0) / (p.damp * p.dt));
      }
    }
    // table[k] = 16807^(6k) mod (2^31 - 1); one step of a system of n beads advances by table[n]
    std::vector<unsigned int> table(max_n + 1);
    unsigned int m6 = 1;
    for (int k = 0; k < 6; k++) m6 = lcg_mul(m6, 16807u);
    table[0] = 1;
    for (int k = 1; k <= max_n; k++) table[k] = lcg_mul(table[k - 1], m6);
    for (int k = 0; k < n_systems; k++) h->sp[k].lcg_step = table[params[k].n_subunits * np];
    CUDA_TRY(cudaMemcpy(h->d_sys.p, h->sp.data(), sizeof(SysParams) * n_systems, cudaMemcpyHostToDevice));
    CUDA_TRY(h->bd_drag.alloc(drag.size()));
    CUDA_TRY(cudaMemcpy(h->bd_drag.p, drag.data(), drag.size() * sizeof(long long), cudaMemcpyHostToDevice));
    CUDA_TRY(h->bd_noise.alloc(noise.size()));
    CUDA_TRY(cudaMemcpy(h->bd_noise.p, noise.data(), noise.size() * sizeof(double), cudaMemcpyHostToDevice));
    CUDA_TRY(h->lcg_table.alloc(table.size()));
    CUDA_TRY(cudaMemcpy(h->lcg_table.p, table.data(), table.size() * sizeof(unsigned int), cudaMemcpyHostToDevice));
    CUDA_TRY(h->bd_fdrag.alloc(3 * N));
    CUDA_TRY(h->bd_fran.alloc(3 * N));
    CUDA_TRY(cudaMemset(h->bd_fdrag.p, 0, sizeof(long long) * 3 * N));
    CUDA_TRY(cudaMemset(h->bd_fran.p, 0, sizeof(long long) * 3 * N));
  }
  CUDA_TRY(h->e_tot.alloc(8));
  for (int k = 0; k < n_systems; k++) h->max_sub = std::max(h->max_sub, params[k].n_subunits);
  CUDA_TRY(h->e_sph.alloc(h->max_sub));
  CUDA_TRY(h->e_part.alloc(7 * kTotalCtas));
  CUDA_TRY(h->e_scr.alloc(2));
  CUDA_TRY(cudaMemset(h->e_scr.p, 0, 2 * sizeof(int)));
  CUDA_TRY(set_energy_smem(L));
  CUDA_TRY(cudaMemset(h->intra_mask.p, 0, sizeof(unsigned int) * (size_t)h->S * np * L.words));
  CUDA_TRY(cudaMemset(h->inter_count.p, 0, sizeof(int) * N));
  CUDA_TRY(cudaMemset(h->force.p, 0, sizeof(long long) * 3 * N));

  h->pair_chunk = pair_chunk(np, L.words);
  h->pair_smem = pair_smem_bytes(np, L.words, h->pair_chunk);
  s = plan_work(h.get(), h->subs_per_cta, h->threads);
  if (s != SOUFFLE_OK) return s;
  *out = h.release();
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_destroy(souffle_gpu_system* h) {
  delete h;
  return SOUFFLE_OK;
}

int64_t souffle_gpu_num_beads(const souffle_gpu_system* h) { return h ? h->N : 0; }

souffle_status souffle_gpu_set_big_beads(souffle_gpu_system* h, int32_t system, int32_t n, const double* pos,
                                         double sigma, double charge, double shc) {
  constexpr int kMaxBigBeads = 4096;  // per system: each subunit bead loops over them every step
  if (!h || system < 0 || system >= h->n_sys || n < 0 || (n > 0 && !pos))
    return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (n > kMaxBigBeads) return fail(SOUFFLE_ERR_BAD_INPUT, "at most 4096 big beads per system");
  if (n > 0 && !(sigma > 0 && shc > 0 && std::isfinite(charge) && std::isfinite(sigma) && std::isfinite(shc)))
    return fail(SOUFFLE_ERR_BAD_INPUT, "big-bead diameter and hard-core distance must be positive");
  for (int i = 0; i < 3 * n; i++)
    if (!std::isfinite(pos[i]) || std::fabs(pos[i]) > 0.75 * h->prm[system].box)
      return fail(SOUFFLE_ERR_BAD_INPUT, "big-bead position outside the box");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  if ((int)h->bb_pos.size() != h->n_sys) h->bb_pos.resize(h->n_sys);
  h->bb_pos[system].assign(pos, pos + 3 * (size_t)n);
  const souffle_params& q = h->prm[system];
  SysParams& P = h->sp[system];
  P.bb_q = charge;
  P.bb_sigma_d = sigma;
  P.bb_shc_d = shc;
  // the Yukawa size factor exp(kappa (s1 + s2)/2) / ((1 + kappa s1/2)(1 + kappa s2/2)) splits
  // into one weight per bead, as for the subunit beads' dh_w
  P.bb_w = (float)(charge * std::exp(q.kappa * sigma / 2) / (1 + q.kappa * sigma / 2) * std::sqrt(q.lb));
  P.bb_sigma = (float)sigma;
  P.bb_shc = (float)shc;
  P.bb_dh_cut2 = q.ecut_el > 0 ? (float)(q.ecut_el * q.ecut_el) : 0.0f;
  {
    const double smax = *std::max_element(h->tpl.sigma.begin(), h->tpl.sigma.end());
    const double reach = std::max(q.ecut_el > 0 ? q.ecut_el : 0.0, 0.5 * (sigma + smax) - shc + 1.12246205 * shc);
    P.bb_reach2 = (float)(1.01 * reach * 1.01 * reach);
  }
  if (q.brownian) {
    // one step draws six numbers per subunit bead, then six per big bead (src/md.cpp:482-487)
    unsigned int m6 = 1, r = 1;
    for (int k = 0; k < 6; k++) m6 = lcg_mul(m6, 16807u);
    for (long long e = (long long)q.n_subunits * h->tpl.np + n; e > 0; e >>= 1) {
      if (e & 1) r = lcg_mul(r, m6);
      m6 = lcg_mul(m6, m6);
    }
    P.lcg_step = r;
  }
  // all systems' big beads, in system order, as fixed point in each system's box
  int total = 0;
  for (int k = 0; k < h->n_sys; k++) total += (int)(h->bb_pos[k].size() / 3);
  std::vector<int4> p32(std::max(total, 1), make_int4(0, 0, 0, 0));
  std::vector<long long> fx(3 * (size_t)std::max(total, 1), 0);
  for (int k = 0, b = 0; k < h->n_sys; k++) {
    SysParams& Q = h->sp[k];
    const int nk = (int)(h->bb_pos[k].size() / 3);
    Q.bb0 = b;
    Q.nbb = nk;
    const double invL = 1.0 / Q.box;
    for (int i = 0; i < nk; i++, b++) {
      const long long X = fixed_from_fraction(h->bb_pos[k][3 * i] * invL);
      const long long Y = fixed_from_fraction(h->bb_pos[k][3 * i + 1] * invL);
      const long long Z = fixed_from_fraction(h->bb_pos[k][3 * i + 2] * invL);
      fx[b] = X;
      fx[(size_t)std::max(total, 1) + b] = Y;
      fx[2 * (size_t)std::max(total, 1) + b] = Z;
      p32[b] = make_int4(hi_word(X), hi_word(Y), hi_word(Z), k);
    }
  }
  CUDA_TRY(h->bb_pos32.alloc(p32.size()));
  CUDA_TRY(cudaMemcpy(h->bb_pos32.p, p32.data(), p32.size() * sizeof(int4), cudaMemcpyHostToDevice));
  CUDA_TRY(h->bb_fx.alloc(fx.size()));
  CUDA_TRY(cudaMemcpy(h->bb_fx.p, fx.data(), fx.size() * sizeof(long long), cudaMemcpyHostToDevice));
  CUDA_TRY(cudaMemcpy(h->d_sys.p, h->sp.data(), sizeof(SysParams) * h->n_sys, cudaMemcpyHostToDevice));
  for (auto& g : h->graphs) cudaGraphExecDestroy(g.second);  // captured arguments changed
  h->graphs.clear();
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_set_state(souffle_gpu_system* h, const double* pos, const double* vel) {
  if (!h || !pos) return fail(SOUFFLE_ERR_BAD_INPUT, "null argument");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const int64_t N = h->N;
  CUDA_TRY(cudaMemcpyAsync(h->staging.p, pos, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, h->stream));
  if (vel)
    CUDA_TRY(cudaMemcpyAsync(h->staging.p + 3 * N, vel, sizeof(double) * 3 * N, cudaMemcpyHostToDevice, h->stream));
  StateArgs a{};
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  a.bead_sys = h->d_bead_sys.p;
  a.np = h->tpl.np;
  a.n = (int)N;
  a.pos_in = h->staging.p;
  a.vel_in = vel ? h->staging.p + 3 * N : nullptr;
  a.px = h->pos_fx.p;
  a.py = h->pos_fx.p + N;
  a.pz = h->pos_fx.p + 2 * N;
  a.pos32 = h->pos32.p;
  a.vx = h->vel.p;
  a.vy = h->vel.p + N;
  a.vz = h->vel.p + 2 * N;
  // reset thermostat/COM bookkeeping
  CUDA_TRY(cudaMemsetAsync(h->d_state.p, 0, sizeof(SysState) * h->n_sys, h->stream));
  launch_state_in(a, (int)((N + 255) / 256), 256, h->stream);
  CUDA_TRY(cudaGetLastError());
  h->have_state = true;
  h->began = false;
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_get_state(souffle_gpu_system* h, double* pos, double* vel) {
  if (!h) return fail(SOUFFLE_ERR_BAD_INPUT, "null handle");
  if (!h->have_state) return fail(SOUFFLE_ERR_STATE, "no state set");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const int64_t N = h->N;
  StateArgs a{};
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  a.bead_sys = h->d_bead_sys.p;
  a.np = h->tpl.np;
  a.n = (int)N;
  a.px = h->pos_fx.p;
  a.py = h->pos_fx.p + N;
  a.pz = h->pos_fx.p + 2 * N;
  a.vx = h->vel.p;
  a.vy = h->vel.p + N;
  a.vz = h->vel.p + 2 * N;
  a.pos_out = pos ? h->staging.p : nullptr;
  a.vel_out = vel ? h->staging.p + 3 * N : nullptr;
  launch_state_out(a, (int)((N + 255) / 256), 256, h->stream);
  CUDA_TRY(cudaGetLastError());
  if (pos) CUDA_TRY(cudaMemcpyAsync(pos, h->staging.p, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, h->stream));
  if (vel)
    CUDA_TRY(cudaMemcpyAsync(vel, h->staging.p + 3 * N, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_snapshot_enqueue(souffle_gpu_system* h, int32_t slot, double* pos, double* vel) {
  if (!h || slot < 0 || slot > 1) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (!h->have_state) return fail(SOUFFLE_ERR_STATE, "no state set");
  if (h->snap_pending[slot]) return fail(SOUFFLE_ERR_STATE, "snapshot slot still pending: wait for it first");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const int64_t N = h->N;
  if (!h->snap[slot].p) CUDA_TRY(h->snap[slot].alloc(6 * N));
  if (!h->snap_err) {
    CUDA_TRY(cudaMallocHost(&h->snap_err, 2 * sizeof(unsigned int)));
    h->snap_err[0] = h->snap_err[1] = 0;
  }
  if (!h->snap_ev[slot]) CUDA_TRY(cudaEventCreateWithFlags(&h->snap_ev[slot], cudaEventDisableTiming));
  StateArgs a{};
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  a.bead_sys = h->d_bead_sys.p;
  a.np = h->tpl.np;
  a.n = (int)N;
  a.px = h->pos_fx.p;
  a.py = h->pos_fx.p + N;
  a.pz = h->pos_fx.p + 2 * N;
  a.vx = h->vel.p;
  a.vy = h->vel.p + N;
  a.vz = h->vel.p + 2 * N;
  a.pos_out = pos ? h->snap[slot].p : nullptr;
  a.vel_out = vel ? h->snap[slot].p + 3 * N : nullptr;
  launch_state_out(a, (int)((N + 255) / 256), 256, h->stream);
  CUDA_TRY(cudaGetLastError());
  if (pos) CUDA_TRY(cudaMemcpyAsync(pos, h->snap[slot].p, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, h->stream));
  if (vel)
    CUDA_TRY(cudaMemcpyAsync(vel, h->snap[slot].p + 3 * N, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost,
                             h->stream));
  CUDA_TRY(cudaMemcpyAsync(h->snap_err + slot, h->err.p, sizeof(unsigned int), cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaEventRecord(h->snap_ev[slot], h->stream));
  h->snap_pending[slot] = true;
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_snapshot_wait(souffle_gpu_system* h, int32_t slot) {
  if (!h || slot < 0 || slot > 1) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (!h->snap_pending[slot]) return fail(SOUFFLE_ERR_STATE, "no snapshot queued in this slot");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  h->snap_pending[slot] = false;
  CUDA_TRY(cudaEventSynchronize(h->snap_ev[slot]));
  // errors of the work queued before the snapshot: the full check (it also clears the flag)
  if (h->snap_err[slot]) return check_err(h);
  return SOUFFLE_OK;
}

void* souffle_gpu_host_alloc(int64_t bytes) {
  void* p = nullptr;
  if (bytes <= 0 || cudaMallocHost(&p, (size_t)bytes) != cudaSuccess) return nullptr;
  return p;
}

void souffle_gpu_host_free(void* p) {
  if (p) cudaFreeHost(p);
}

// Total (int64, 2^-32 units), stretching and bending forces (FP32) as doubles, xyz interleaved, in the
// staging buffer: stretching at 0, bending at 3 N, total at 6 N.
static void launch_force_out(souffle_gpu_system* h, bool total, bool stretch, bool bend) {
  const int64_t N = h->N;
  StateArgs a{};
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  a.bead_sys = h->d_bead_sys.p;
  a.np = h->tpl.np;
  a.n = (int)N;
  if (total) a.force_out = h->staging.p + 6 * N;
  a.fx_in = h->force.p;
  a.fy_in = h->force.p + N;
  a.fz_in = h->force.p + 2 * N;
  if (stretch) a.sforce_out = h->staging.p;
  if (bend) a.bforce_out = h->staging.p + 3 * N;
  a.sb_in = h->sbforce.p;
  launch_state_out(a, (int)((N + 255) / 256), 256, h->stream);
}

souffle_status souffle_gpu_forces(souffle_gpu_system* h, int32_t rebuild, double* tforce, double* sforce,
                                  double* bforce) {
  if (!h) return fail(SOUFFLE_ERR_BAD_INPUT, "null handle");
  if (!h->have_state) return fail(SOUFFLE_ERR_STATE, "no state set");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const bool parts = sforce || bforce;
  souffle_status s = SOUFFLE_OK;
  for (int attempt = 0; attempt < 4; attempt++) {
    if (rebuild) launch_rebuild(h);
    launch_forces_all(h, 0, parts);
    launch_force_out(h, tforce != nullptr, sforce != nullptr, bforce != nullptr);
    CUDA_TRY(cudaGetLastError());
    s = check_err(h);
    // a forces-only call changes no state, so an overflowing list is rebuilt with twice the room
    if (s != SOUFFLE_ERR_NL_OVERFLOW || !rebuild) break;
    if (g_last_error.find("candidate") != std::string::npos) {
      h->cand_cap *= 2;
      CUDA_TRY(h->cand.alloc((size_t)h->cand_cap * h->S));
    } else {
      if (h->inter_cap >= kMaxInterPerBead) break;
      h->inter_cap = std::min(kMaxInterPerBead, 2 * h->inter_cap);
      CUDA_TRY(h->inter_ids.alloc((size_t)h->inter_cap * h->N));
    }
    for (auto& g : h->graphs) cudaGraphExecDestroy(g.second);
    h->graphs.clear();
  }
  if (s != SOUFFLE_OK) return s;
  const int64_t N = h->N;
  double* const out[3] = {sforce, bforce, tforce};
  for (int k = 0; k < 3; k++)
    if (out[k])
      CUDA_TRY(cudaMemcpyAsync(out[k], h->staging.p + 3 * k * N, sizeof(double) * 3 * N, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_get_pairlist(souffle_gpu_system* h, int32_t cap, int32_t* counts, int32_t* ids) {
  if (!h || cap < 0) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const int np = h->tpl.np, words = h->L.words;
  const int64_t N = h->N;
  std::vector<unsigned int> mask((size_t)h->S * np * words);
  std::vector<int> icnt(N), iids((size_t)h->inter_cap * N);
  CUDA_TRY(cudaMemcpyAsync(mask.data(), h->intra_mask.p, mask.size() * 4, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaMemcpyAsync(icnt.data(), h->inter_count.p, N * 4, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaMemcpyAsync(iids.data(), h->inter_ids.p, iids.size() * 4, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  // merge the intra-subunit block into the ascending inter list: the reference order
  for (int64_t g = 0; g < N; g++) {
    const int sub = (int)(g / np), l = (int)(g % np);
    const int lo = sub * np, hi = lo + np;
    std::vector<int> out;
    int k = 0;
    const int n_in = icnt[g];
    const int* row = iids.data() + (size_t)g * h->inter_cap;  // row-major [N][cap]
    while (k < n_in && row[k] < lo) out.push_back(row[k++]);
    for (int jj = 0; jj < np; jj++)
      if (mask[((size_t)sub * np + l) * words + (jj >> 5)] >> (jj & 31) & 1u) out.push_back(lo + jj);
    while (k < n_in) {
      int v = row[k++];
      (void)hi;
      out.push_back(v);
    }
    if (counts) counts[g] = (int)out.size();
    if (ids) {
      for (int c = 0; c < cap; c++) ids[(size_t)g * cap + c] = c < (int)out.size() ? out[c] : -1;
    }
  }
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_pairlist_stats(souffle_gpu_system* h, int32_t system, souffle_pairlist_stats* out) {
  if (!h || !out || system < 0 || system >= h->n_sys) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const SysParams& P = h->sp[system];
  const int n = P.n_sub * h->tpl.np;
  std::vector<int> len(n), icnt(n);
  CUDA_TRY(cudaMemcpyAsync(len.data(), h->ref_len.p + P.bead0, n * 4, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaMemcpyAsync(icnt.data(), h->inter_count.p + P.bead0, n * 4, cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  double sum = 0;
  int mx = 0, mi = 0, over = 0;
  for (int i = 0; i < n; i++) {
    sum += len[i];
    mx = std::max(mx, len[i]);
    mi = std::max(mi, icnt[i]);
    if (len[i] > h->prm[system].nlist_capacity) over++;
  }
  out->mean_length = sum / n;
  out->max_length = mx;
  out->max_inter = mi;
  out->over_reference_capacity = over;
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_energies(souffle_gpu_system* h, int32_t system, souffle_energies* out, double* se,
                                    double* be, double* ne, double* ce, double* ke) {
  if (!h || system < 0 || system >= h->n_sys) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (!h->have_state) return fail(SOUFFLE_ERR_STATE, "no state set");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const SysParams& P = h->sp[system];
  const souffle_params& p = h->prm[system];
  const int n = P.n_sub * h->tpl.np;
  if (h->e_bead.n < (size_t)7 * n) CUDA_TRY(h->e_bead.alloc((size_t)7 * n));
  EnergyArgs a{};
  a.L = h->L;
  a.tpl_i = h->tpl_i.p;
  a.tpl_f = h->tpl_f.p;
  a.sys = h->d_sys.p;
  a.state = h->d_state.p;
  const int64_t N = h->N;
  a.px = h->pos_fx.p;
  a.py = h->pos_fx.p + N;
  a.pz = h->pos_fx.p + 2 * N;
  a.pos32 = h->pos32.p;
  a.vx = h->vel.p;
  a.vy = h->vel.p + N;
  a.vz = h->vel.p + 2 * N;
  a.len0 = h->len0_d.p;
  a.mass = h->mass_d.p;
  a.q = h->q_d.p;
  a.sigma = h->sigma_d.p;
  a.type = h->type_d.p;
  a.lj_t = h->lj_d.p;
  a.n_lj = h->tpl.n_lj;
  a.ecut = p.ecut;
  a.elj_att = p.elj_att;
  a.lb = p.lb;
  a.kappa = p.kappa;
  a.ecut_el = p.ecut_el;
  a.sigma_max = *std::max_element(h->tpl.sigma.begin(), h->tpl.sigma.end());
  a.sysid = system;
  a.n0 = P.bead0;
  a.n = n;
  a.se = h->e_bead.p;
  a.be = h->e_bead.p + n;
  a.ne = h->e_bead.p + 2 * (size_t)n;
  a.ce = h->e_bead.p + 3 * (size_t)n;
  a.ke = h->e_bead.p + 4 * (size_t)n;
  a.totals = h->e_tot.p;
  if (P.nbb > 0) {  // encapsulation big beads
    a.bb_fx = h->bb_fx.p;
    a.bb_total = (int)(h->bb_fx.n / 3);
    a.ne_bb = h->e_bead.p + 5 * (size_t)n;
    a.ce_bb = h->e_bead.p + 6 * (size_t)n;
  }
  {
    const size_t np2 = (size_t)h->tpl.np * h->tpl.np;
    if (h->e_pair_tab.n != 3 * np2) CUDA_TRY(h->e_pair_tab.alloc(3 * np2));
    if (h->e_att_tab.n != np2) CUDA_TRY(h->e_att_tab.alloc(np2));
    a.pair_tab = h->e_pair_tab.p;
    a.att_tab = h->e_att_tab.p;
  }
  a.w = h->dh_wd.p + (size_t)system * h->tpl.np;
  a.el_shift = p.ecut_el > 0 ? std::exp(-p.kappa * p.ecut_el) / p.ecut_el : 0.0;
  a.exp_scale = -p.kappa * (64.0 / 0.69314718055994530942);
  a.inv_ecut3 = 1.0 / (p.ecut * p.ecut * p.ecut);
  const EnergySubPlan sub_plan = energy_sub_plan(h->L);
  a.spc = sub_plan.spc;
  a.faces = sub_plan.faces;
  a.sph = h->e_sph.p;
  a.rmax = h->e_scr.p;
  a.ticket = reinterpret_cast<unsigned int*>(h->e_scr.p + 1);
  a.partials = h->e_part.p;
  if (p.ecut_el > 0 && energy_needs_cells(P.n_sub)) {
    launch_subunit_cells(h);
    launch_cells_sort(cell_args(h), h->stream);  // the sums do not depend on scheduling
    a.sub_cell_start = h->cell_start.p;
    a.sub_cell_count = h->cell_count.p;
    a.cell_subs = h->cell_subs.p;
  }
  launch_energies(a, n, h->stream);
  CUDA_TRY(cudaGetLastError());
  double tot[8];
  SysState S;
  tot[5] = tot[6] = 0.0;
  CUDA_TRY(cudaMemcpyAsync(tot, h->e_tot.p, sizeof(double) * (P.nbb > 0 ? 7 : 5), cudaMemcpyDeviceToHost,
                           h->stream));
  CUDA_TRY(cudaMemcpyAsync(&S, h->d_state.p + system, sizeof(SysState), cudaMemcpyDeviceToHost, h->stream));
  double* outs[5] = {se, be, ne, ce, ke};
  const int order[5] = {0, 1, 2, 3, 4};
  for (int k = 0; k < 5; k++)
    if (outs[k])
      CUDA_TRY(cudaMemcpyAsync(outs[k], h->e_bead.p + (size_t)order[k] * n, sizeof(double) * n,
                               cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  if (out) {
    out->kinetic = tot[0];
    out->stretching = tot[1];
    out->bending = tot[2];
    out->lj = tot[3];
    out->electrostatic = tot[4];
    // THERMOSTAT::potential_energy / kinetic_energy (src/thermostat.h:43-52), kB = 1
    double tpe = 0, tke = 0;
    for (int j = 0; j < S.m; j++) {
      const double eta = df_to(S.eta[j]), xi = df_to(S.xi[j]);
      tpe += S.dof[j] * 1.0 * S.t[j] * eta;
      tke += 0.5 * S.q[j] * xi * xi;
    }
    out->thermo_pe = tpe;
    out->thermo_ke = tke;
    out->temperature = tot[0] * 2 / (3.0 * n);
    out->vcom_magnitude = vcom_magnitude(S);
    out->bigbead_lj = tot[5];
    out->bigbead_electrostatic = tot[6];
  }
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_kinetic_energy(souffle_gpu_system* h, int32_t system, double* ke) {
  souffle_energies e;
  if (!ke) return fail(SOUFFLE_ERR_BAD_INPUT, "null output");
  souffle_status s = souffle_gpu_energies(h, system, &e, nullptr, nullptr, nullptr, nullptr, nullptr);
  if (s == SOUFFLE_OK) *ke = e.kinetic;
  return s;
}

souffle_status souffle_gpu_md_begin(souffle_gpu_system* h) {
  if (!h) return fail(SOUFFLE_ERR_BAD_INPUT, "null handle");
  if (!h->have_state) return fail(SOUFFLE_ERR_STATE, "no state set");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  // thermostat chain (src/md.cpp:187-196): [Q, T, 3N], (1, T, 1)..., dummy (0, T, 3N)
  std::vector<SysState> st(h->n_sys);
  for (int k = 0; k < h->n_sys; k++) {
    const souffle_params& p = h->prm[k];
    SysState& S = st[k];
    std::memset(&S, 0, sizeof(S));
    const double n3 = 3.0 * p.n_subunits * h->tpl.np;
    S.n_beads = p.n_subunits * h->tpl.np;
    if (p.chain_length == 1) {
      S.m = 1;
      S.q[0] = 0;
      S.t[0] = p.temperature;
      S.dof[0] = n3;
    } else {
      int m = 0;
      S.q[m] = p.nhc_mass;
      S.t[m] = p.temperature;
      S.dof[m++] = n3;
      while (m != p.chain_length - 1) {
        S.q[m] = 1;
        S.t[m] = p.temperature;
        S.dof[m++] = 1;
      }
      S.q[m] = 0;
      S.t[m] = p.temperature;
      S.dof[m++] = n3;
      S.m = m;
    }
    if (p.brownian) {  // no thermostat (src/md.cpp:187 sets one up for -D m only); the noise
      S.m = 0;         // generator restarts from its seed every run (src/md.cpp:382-385)
      S.lcg = kLcgSeed;
    }
    nhc_set_constants(S, p.dt);
    S.inv_n = 1.0 / S.n_beads;
  }
  CUDA_TRY(cudaMemcpyAsync(h->d_state.p, st.data(), sizeof(SysState) * h->n_sys, cudaMemcpyHostToDevice, h->stream));
  if (h->opt.chain_fp64) {
    std::vector<Chain64> c64(h->n_sys);
    for (int k = 0; k < h->n_sys; k++) {
      Chain64& c = c64[k];
      std::memset(&c, 0, sizeof(c));
      c.m = st[k].m;
      c.dt = h->prm[k].dt;
      for (int j = 0; j < c.m; j++) {
        c.q[j] = st[k].q[j];
        c.t[j] = st[k].t[j];
        c.dof[j] = st[k].dof[j];
      }
    }
    if (h->chain64.n != (size_t)h->n_sys) CUDA_TRY(h->chain64.alloc(h->n_sys));  // kept: graphs hold the pointer
    CUDA_TRY(cudaMemcpyAsync(h->chain64.p, c64.data(), sizeof(Chain64) * h->n_sys, cudaMemcpyHostToDevice,
                             h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
  }
  // initial forces with a rebuild (src/md.cpp:241) and particle_ke (src/md.cpp:258); the last
  // CTA then applies the backward half of the first step
  launch_rebuild(h);
  launch_forces_all(h, 2, false);
  CUDA_TRY(cudaGetLastError());
  souffle_status s = check_err(h);
  if (s != SOUFFLE_OK) return s;
  h->began = true;
  return SOUFFLE_OK;
}

souffle_status souffle_gpu_md_steps(souffle_gpu_system* h, int64_t first_step, int32_t n_steps) {
  const souffle_status s = souffle_gpu_md_enqueue(h, first_step, n_steps);
  if (s != SOUFFLE_OK) return s;
  return check_err(h);
}

souffle_status souffle_gpu_md_enqueue(souffle_gpu_system* h, int64_t first_step, int32_t n_steps) {
  if (!h || n_steps < 0 || first_step < 0) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (!h->began) return fail(SOUFFLE_ERR_STATE, "md_begin has not been called");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  // All systems share the rebuild period of system 0 (a batch is rebuilt together).
  const int B = h->prm[0].build_freq;
  int64_t a = first_step;
  const int64_t end = first_step + n_steps;
  // graphs: key 2*len + rebuild-first; a whole rebuild window is one graph of B steps, any other
  // step is a one-step graph with or without the rebuild
  auto run_graph = [&](int len, bool rebuild_first) -> souffle_status {
    unsigned long long judge_mask = 0;
    for (int k = 0; k < len && k < 64; k++)
      if (surrogate_judge_due(h, a + k)) judge_mask |= 1ull << k;
    const std::pair<int, unsigned long long> key(2 * len + (rebuild_first ? 1 : 0), judge_mask);
    auto it = h->graphs.find(key);
    if (it == h->graphs.end()) {
      cudaGraphExec_t ge = nullptr;
      CUDA_TRY(capture_steps(h, len, rebuild_first, judge_mask, &ge));
      it = h->graphs.emplace(key, ge).first;
    }
    CUDA_TRY(cudaGraphLaunch(it->second, h->stream));
    return SOUFFLE_OK;
  };
  while (a < end) {
    souffle_status s;
    if (a % B == 0 && end - a >= B && B <= kMaxPeriod) {
      s = run_graph(B, true);
      a += B;
    } else {
      s = run_graph(1, a % B == 0);
      a += 1;
    }
    if (s != SOUFFLE_OK) return s;
  }
  CUDA_TRY(cudaGetLastError());
  return SOUFFLE_OK;
}

void* souffle_gpu_stream(souffle_gpu_system* h) { return h ? (void*)h->stream : nullptr; }

souffle_status souffle_gpu_md_profile(souffle_gpu_system* h, int64_t first_step, int32_t n_steps,
                                      souffle_kernel_times* out) {
  if (!h || !out || n_steps < 0 || first_step < 0) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (!h->began) return fail(SOUFFLE_ERR_STATE, "md_begin has not been called");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const int B = h->prm[0].build_freq;
  std::memset(out, 0, sizeof(*out));
  cudaEvent_t ev[4];
  for (auto& e : ev) CUDA_TRY(cudaEventCreate(&e));
  souffle_status st = SOUFFLE_OK;
  for (int64_t a = first_step; a < first_step + n_steps && st == SOUFFLE_OK; a++) {
    const bool rb = (a % B == 0);
    cudaEventRecord(ev[0], h->stream);
    launch_drift_all(h);
    cudaEventRecord(ev[1], h->stream);
    if (rb) launch_rebuild(h);
    cudaEventRecord(ev[2], h->stream);
    launch_forces_all(h, 1, false, surrogate_judge_due(h, a));
    cudaEventRecord(ev[3], h->stream);
    if (cudaEventSynchronize(ev[3]) != cudaSuccess) {
      st = fail(SOUFFLE_ERR_CUDA, "event synchronize failed");
      break;
    }
    float t0, t1, t2;
    cudaEventElapsedTime(&t0, ev[0], ev[1]);
    cudaEventElapsedTime(&t1, ev[1], ev[2]);
    cudaEventElapsedTime(&t2, ev[2], ev[3]);
    out->drift_ms += t0;
    out->forces_ms += t2;
    if (rb) {
      out->rebuild_ms += t1;
      out->rebuilds++;
    }
    out->steps++;
  }
  for (auto& e : ev) cudaEventDestroy(e);
  if (st != SOUFFLE_OK) return st;
  CUDA_TRY(cudaGetLastError());
  return check_err(h);
}

souffle_status souffle_gpu_md_scalars(souffle_gpu_system* h, int32_t system, double* ke, double* xi0,
                                      double* vcom) {
  if (!h || system < 0 || system >= h->n_sys) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  SysState S;
  CUDA_TRY(cudaMemcpyAsync(&S, h->d_state.p + system, sizeof(S), cudaMemcpyDeviceToHost, h->stream));
  CUDA_TRY(cudaStreamSynchronize(h->stream));
  if (ke) *ke = df_to(S.ke);
  if (xi0) *xi0 = df_to(S.xi[0]);
  if (vcom) *vcom = vcom_magnitude(S);
  return SOUFFLE_OK;
}

}  // extern "C"

namespace {
// Mean microseconds per step over at least n steps of graphs of one rebuild period, no rebuild in them.
souffle_status time_steps(souffle_gpu_system* h, int n, cudaEvent_t e0, cudaEvent_t e1, double* us) {
  const int len = h->prm[0].build_freq, runs = (n + len - 1) / len;
  if (h->deal_ok) launch_deal(deal_args(h), h->stream);
  cudaGraphExec_t g = nullptr;
  CUDA_TRY(capture_steps(h, len, false, 0, &g));
  cudaError_t e = cudaGraphLaunch(g, h->stream);  // warm-up
  if (e == cudaSuccess) e = cudaEventRecord(e0, h->stream);
  for (int k = 0; k < runs && e == cudaSuccess; k++) e = cudaGraphLaunch(g, h->stream);
  if (e == cudaSuccess) e = cudaEventRecord(e1, h->stream);
  if (e == cudaSuccess) e = cudaEventSynchronize(e1);
  cudaGraphExecDestroy(g);
  CUDA_TRY(e);
  float ms = 0;
  CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
  *us = 1e3 * ms / ((double)runs * len);
  return check_err(h);
}

// What timing at the current positions overwrites: the forces of the last step, which the next one starts
// from, and, where steps are timed, velocities, kicks and thermostat, all zero so that nothing moves.
// Velocities and forces go to the staging buffer.
struct SavedState {
  DevBuf<long long> kick;
  DevBuf<SysState> state;
  template <class T>
  static cudaError_t copy(T* to, const T* from, size_t n, cudaStream_t st) {
    return cudaMemcpyAsync(to, from, sizeof(T) * n, cudaMemcpyDeviceToDevice, st);
  }
  static long long* vel(souffle_gpu_system* h) { return reinterpret_cast<long long*>(h->staging.p); }
  static long long* force(souffle_gpu_system* h) { return vel(h) + h->vel.n; }
  souffle_status save(souffle_gpu_system* h, bool rest) {
    static_assert(sizeof(long long) == sizeof(double), "staged as doubles");
    CUDA_TRY(kick.alloc(h->kick_c.n));
    CUDA_TRY(state.alloc(h->d_state.n));
    CUDA_TRY(copy(vel(h), h->vel.p, h->vel.n, h->stream));
    CUDA_TRY(copy(force(h), h->force.p, h->force.n, h->stream));
    CUDA_TRY(copy(kick.p, h->kick_c.p, kick.n, h->stream));
    CUDA_TRY(copy(state.p, h->d_state.p, state.n, h->stream));
    if (!rest) return SOUFFLE_OK;
    CUDA_TRY(cudaMemsetAsync(h->vel.p, 0, sizeof(long long) * h->vel.n, h->stream));
    CUDA_TRY(cudaMemsetAsync(h->kick_c.p, 0, sizeof(long long) * kick.n, h->stream));
    CUDA_TRY(cudaMemsetAsync(h->d_state.p, 0, sizeof(SysState) * state.n, h->stream));
    return SOUFFLE_OK;
  }
  souffle_status put_back(souffle_gpu_system* h) {
    CUDA_TRY(copy(h->vel.p, vel(h), h->vel.n, h->stream));
    CUDA_TRY(copy(h->force.p, force(h), h->force.n, h->stream));
    CUDA_TRY(copy(h->kick_c.p, kick.p, kick.n, h->stream));
    CUDA_TRY(copy(h->d_state.p, state.p, state.n, h->stream));
    CUDA_TRY(cudaStreamSynchronize(h->stream));
    return SOUFFLE_OK;
  }
};
}  // namespace

extern "C" {

souffle_status souffle_gpu_autotune(souffle_gpu_system* h, int32_t trials, souffle_tuning* out) {
  if (!h || trials < 1 || trials > 1000) return fail(SOUFFLE_ERR_BAD_INPUT, "bad argument");
  if (!h->have_state) return fail(SOUFFLE_ERR_STATE, "no state set");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  const int np = h->tpl.np;
  const int def_subs = std::max(1, 128 / np), def_threads = 256;
  // candidate shapes: subunits per CTA x threads per CTA (force kernel: two threads per bead,
  // any bead count; at most 256 threads)
  std::vector<std::pair<int, int>> cand;
  for (int subs : {1, 2, 3, 4, 6, 8})
    for (int thr : {96, 128, 192, 256}) {
      if (!force_shape_ok(h, subs, thr)) continue;
      if (subs * np * 2 > 4 * thr) continue;  // more than two passes per thread pair
      if (subs * np * 2 < thr / 2) continue;   // most of the CTA idle
      cand.emplace_back(subs, thr);
    }
  if (std::find(cand.begin(), cand.end(), std::make_pair(def_subs, def_threads)) == cand.end())
    cand.emplace_back(def_subs, def_threads);
  // a rebuild at the current positions, so every shape sees the same lists
  launch_rebuild(h);
  souffle_status s = check_err(h);
  if (s != SOUFFLE_OK) return s;
  // Where the default shape's steps run in windows, whole periods of steps are timed (a shape with too many
  // items loses the window, by which 64 subunits take half the time), else the force kernel alone.
  if ((s = plan_work(h, def_subs, def_threads)) != SOUFFLE_OK) return s;
  const bool steps = window_usable(h) && h->prm[0].build_freq > 1 && h->prm[0].build_freq <= kMaxPeriod;
  cudaEvent_t e0, e1;
  CUDA_TRY(cudaEventCreate(&e0));
  CUDA_TRY(cudaEventCreate(&e1));
  SavedState saved;
  if ((s = saved.save(h, steps)) != SOUFFLE_OK) return s;
  double best = 1e30, def_us = 0;
  std::pair<int, int> best_shape = cand.front();
  for (auto& c : cand) {
    if ((s = plan_work(h, c.first, c.second)) != SOUFFLE_OK) break;
    double us = 0;
    if (steps) {
      if ((s = time_steps(h, trials, e0, e1, &us)) != SOUFFLE_OK) break;
    } else {
      for (int k = 0; k < 3; k++) launch_forces_all(h, 0, false);
      cudaEventRecord(e0, h->stream);
      for (int k = 0; k < trials; k++) launch_forces_all(h, 0, false);
      cudaEventRecord(e1, h->stream);
      if (cudaEventSynchronize(e1) != cudaSuccess) {
        s = fail(SOUFFLE_ERR_CUDA, "event synchronize failed");
        break;
      }
      if ((s = check_err(h)) != SOUFFLE_OK) break;
      float ms = 0;
      cudaEventElapsedTime(&ms, e0, e1);
      us = 1e3 * ms / trials;
    }
    if (c.first == def_subs && c.second == def_threads) def_us = us;
    if (us < best) {
      best = us;
      best_shape = c;
    }
  }
  const souffle_status back = saved.put_back(h);
  if (s == SOUFFLE_OK) s = back;
  // The default shape stays unless another is clearly faster: differences of a few percent are within
  // run-to-run noise.
  if (def_us > 0 && best > 0.97 * def_us) {
    best = def_us;
    best_shape = std::make_pair(def_subs, def_threads);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (s != SOUFFLE_OK) return s;
  if ((s = plan_work(h, best_shape.first, best_shape.second)) != SOUFFLE_OK) return s;
  if (out) {
    out->subunits_per_cta = best_shape.first;
    out->threads_per_cta = best_shape.second;
    out->forces_us = best;
    out->default_forces_us = def_us;
    out->candidates = (int)cand.size();
  }
  return SOUFFLE_OK;
}

// Not in the public header, for tests: sets how often a wait of the window kernel tries before it gives
// up, and returns the CTAs of the handle's windows (0: its steps do not take windows; -1: no handle).
int32_t souffle_gpu_window_polls(souffle_gpu_system* h, uint32_t polls) {
  if (!h || cudaSetDevice(h->opt.device) != cudaSuccess || cudaStreamSynchronize(h->stream) != cudaSuccess) return -1;
  h->window_polls = polls;
  for (auto& g : h->graphs) cudaGraphExecDestroy(g.second);  // captured arguments changed
  h->graphs.clear();
  return window_usable(h) ? (int32_t)h->work.size() : 0;
}

souffle_status souffle_gpu_synchronize(souffle_gpu_system* h) {
  if (!h) return fail(SOUFFLE_ERR_BAD_INPUT, "null handle");
  CUDA_TRY(cudaSetDevice(h->opt.device));
  return check_err(h);
}

}  // extern "C"
