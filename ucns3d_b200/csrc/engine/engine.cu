// C ABI of the engine (include/ucns3d_gpu.h): handle, uploads, stage
// driver.  The stage sequence mirrors CALL_FLUX_SUBROUTINES_3D
// (src/time_p.f90:2253-2497) and RUNGE_KUTTA3 (src/time_p.f90:885-1027).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <functional>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "engine_internal.h"
#include "kernels.cuh"

using namespace ucg;

namespace {

std::string g_create_err;

}  // namespace

namespace ucg_host {

int fail(ucg_engine* e, int code, const std::string& msg) {
  if (e) e->err = msg;
  return code;
}

int cuda_fail(ucg_engine* e, cudaError_t st, const char* where) {
  return fail(e, UCG_ECUDA, std::string(where) + ": " + cudaGetErrorString(st));
}

int alloc(ucg_engine* e, DevBuf& b, size_t bytes) {
  if (b.p && b.bytes >= bytes) return UCG_OK;
  if (b.p) {
    cudaFree(b.p);
    e->bytes -= (int64_t)b.bytes;
    b.p = nullptr;
    b.bytes = 0;
  }
  if (bytes == 0) return UCG_OK;
  cudaError_t st = cudaMalloc(&b.p, bytes);
  if (st != cudaSuccess) {
    cudaGetLastError();
    return fail(e, UCG_ENOMEM, "cudaMalloc of " + std::to_string(bytes) + " bytes failed: " + cudaGetErrorString(st));
  }
  b.bytes = bytes;
  e->bytes += (int64_t)bytes;
  return UCG_OK;
}

void release(DevBuf& b) {
  if (b.p) cudaFree(b.p);
  b.p = nullptr;
  b.bytes = 0;
}

size_t tsize(const ucg_engine* e) { return e->mixed ? sizeof(float) : sizeof(double); }

template <typename H>
int upload(ucg_engine* e, DevBuf& b, const std::vector<H>& h) {
  int rc = alloc(e, b, h.size() * sizeof(H));
  if (rc) return rc;
  if (!h.empty()) CK(cudaMemcpyAsync(b.p, h.data(), h.size() * sizeof(H), cudaMemcpyHostToDevice, e->stream));
  return UCG_OK;
}

Problem make_problem(ucg_engine* e) {
  Problem p;
  std::memset(&p, 0, sizeof(p));
  const ucg_config& c = e->cfg;
  p.n = e->n;
  p.nall = e->n;
  p.iorder = c.iorder;
  p.ideg = c.ideg;
  p.imax = c.imax;
  p.admis_max = c.admis_max;
  p.ideg2 = c.ideg2;
  p.imax2 = c.imax2;
  p.ees = c.ees;
  p.scheme = c.scheme;
  p.governing = c.governing;
  p.wenoz = c.wenoz;
  p.nq_quad = c.nq_quad;
  p.nq_tri = c.nq_tri;
  p.gamma = c.gamma;
  p.prandtl = c.prandtl;
  p.visc = c.visc;
  p.r_gas = c.r_gas;
  p.pres = c.pres;
  p.rres = c.rres;
  p.lwci = c.lwci;
  p.weno_eps = c.weno_eps;
  p.kappa_ven = c.kappa_ven;
  p.lamx = c.lamx;
  for (int q = 0; q < MQ; ++q) {
    p.quad_w[q] = c.quad_w[q];
    p.tri_w[q] = c.tri_w[q];
  }
  for (int v = 0; v < NV; ++v) p.bc_state[v] = c.bc_state[v];
  p.nfaces = (const int8_t*)e->nfaces.p;
  p.ftype = (const int8_t*)e->ftype.p;
  p.neigh = (const int32_t*)e->neigh.p;
  p.nface = (const int8_t*)e->nface.p;
  p.bc = (const int8_t*)e->bc.p;
  p.qperm = (const uint8_t*)e->qperm.p;
  p.rot = (const double*)e->rot.p;
  p.area = (const double*)e->area.p;
  p.dih = (const double*)e->dih.p;
  p.vol = (const double*)e->vol.p;
  p.minedge = (const double*)e->minedge.p;
  p.jinv = (const double*)e->jinv.p;
  p.admis = (const int8_t*)e->admis.p;
  p.full = (const int8_t*)e->full.p;
  p.qpts = e->qpts.p;
  p.bmean = e->bmean.p;
  p.sten = (const int32_t*)e->sten.p;
  p.invmat = e->invmat.p;
  p.ind = e->ind.p;
  p.tstride = e->layout.tstride;
  p.istride = e->layout.istride;
  p.i2off = e->layout.i2off;
  for (int k = 0; k < 8; ++k) {
    p.soff[k] = e->layout.soff[k];
  }
  p.ntile = e->ntile;
  p.together = e->tiles_together;
  p.tcell = (const int32_t*)e->tcell.p;
  p.tset = (const int32_t*)e->tset.p;
  p.tiled = e->all_tiled ? nullptr : (const int8_t*)e->tiled.p;
  p.setmat = e->setmat.p;
  p.sstride = e->sstride;
  for (int k = 0; k < 8; ++k) p.sso[k] = e->sso[k];
  p.setind = e->setind.p;
  p.gset = (const int32_t*)e->gset.p;
  p.ugrp = (const int32_t*)e->ugrp.p;
  p.nugrp = e->nugrp;
  p.gbuf = e->gbuf.p;
  p.qbuf = (double*)e->qbuf.p;
  p.isb = (double*)e->isb.p;
  p.wflag = (int8_t*)e->wflag.p;
  p.wface = e->wface;
  p.mprev = e->cfg.mood ? (int8_t*)e->mprev.p : nullptr;
  p.mood = (int8_t*)e->mflag.p;
  p.msel = nullptr;
  p.mmus = nullptr;
  p.mord = (int8_t*)e->mord.p;
  p.dul = e->dul.p;
  p.ulv = (double*)e->ulv.p;
  p.fgrad = (double*)e->fgrad.p;
  p.gv = e->gv.p;
  p.prim = (double*)e->prim.p;
  p.rhs = (double*)e->rhs.p;
  p.own = (const int32_t*)e->own.p;
  p.nown = e->nown;
  p.fflux = (double*)e->fflux.p;
  p.vflux = (double*)e->vflux.p;
  p.health = (unsigned*)e->health.p;
  p.dt_dev = nullptr;
  p.dt_next = nullptr;
  p.ccfl = 0.0;
  p.nsm = e->nsm;
  p.lsq_bulk = e->lsq_bulk;
  p.lsq_wait = e->lsq_bulk || e->lsq_limit ? e->lsq_wait : -1;
  p.wenwrt = c.wenwrt;
  p.riemann = c.riemann;
  p.limiter = c.limiter;
  p.boundtype = c.boundtype;
  return p;
}

bool ready(ucg_engine* e) { return e->have_geometry && e->recon_cells == e->n; }

// ------------------------------------------------------------ launching
template <typename T>
int launch_recon_t(ucg_engine* e, const Problem& p, const double* U) {
  const ucg_config& c = e->cfg;
  if (c.scheme == 2 && c.iorder == 1) {
    const unsigned blocks = (unsigned)((p.n + 31) / 32);
    const bool vk = c.limiter == 7;
    cudaError_t err;
    if (c.governing == 1) {
      constexpr int TH = 32 * muscl_warps<true>();
      if (vk) err = launch_pdl(k_muscl<T, true, true>, blocks, TH, e->stream, p, U);
      else err = launch_pdl(k_muscl<T, true, false>, blocks, TH, e->stream, p, U);
    } else {
      constexpr int TH = 32 * muscl_warps<false>();
      if (vk) err = launch_pdl(k_muscl<T, false, true>, blocks, TH, e->stream, p, U);
      else err = launch_pdl(k_muscl<T, false, false>, blocks, TH, e->stream, p, U);
    }
    e->launches++;
    CK(err);
    return UCG_OK;
  }
  if (c.iorder < 1 || c.iorder > 4) return fail(e, UCG_EINVAL, "iorder out of range");
  const bool ns = c.governing == 1;
  CK(sizeof(T) == 4 ? launch_weno_f32(c.iorder, p, U, ns, e->QS, e->stream, &e->launches, e->mark)
                    : launch_weno_f64(c.iorder, p, U, ns, e->QS, e->stream, &e->launches, e->mark));
  return UCG_OK;
}

// the reconstruction covers cells [0, n_recon) (all of them unless a
// partition's roles leave its outer halo out); the per-cell records that
// the viscous stencils gather (k_visc_prim) still cover every cell
int launch_recon(ucg_engine* e, const Problem& p, const double* U) {
  Problem pr = p;
  pr.n = e->n_recon;
  return e->mixed ? launch_recon_t<float>(e, pr, U) : launch_recon_t<double>(e, pr, U);
}

template <typename T, bool NS>
cudaError_t launch_faces_t(ucg_engine* e, const Problem& p, const double* Uc) {
  cudaError_t err;
  constexpr int FB = UCG_FACE_BLOCK;
  const unsigned fb = (unsigned)((e->nown + FB - 1) / FB);
  switch (e->cfg.riemann) {  // the Riemann solver is a template argument of the face kernel
    case 2: err = launch_pdl(k_face<T, NS, 2>, fb, FB, e->stream, p, Uc); break;
    case 3: err = launch_pdl(k_face<T, NS, 3>, fb, FB, e->stream, p, Uc); break;
    case 4: err = launch_pdl(k_face<T, NS, 4>, fb, FB, e->stream, p, Uc); break;
    case 5: err = launch_pdl(k_face<T, NS, 5>, fb, FB, e->stream, p, Uc); break;
    case 9: err = launch_pdl(k_face<T, NS, 9>, fb, FB, e->stream, p, Uc); break;
    default: err = launch_pdl(k_face<T, NS, 1>, fb, FB, e->stream, p, Uc); break;
  }
  e->launches += 1;
  return err;
}

int launch_faces(ucg_engine* e, const Problem& p, const double* Uc) {
  const bool ns = e->cfg.governing == 1;
  const cudaError_t err = e->mixed ? ns ? launch_faces_t<float, true>(e, p, Uc) : launch_faces_t<float, false>(e, p, Uc)
                                   : ns ? launch_faces_t<double, true>(e, p, Uc) : launch_faces_t<double, false>(e, p, Uc);
  CK(err);
  return UCG_OK;
}

// the residual and the update cover cells [0, n_update) (all of them unless
// a partition's roles step only its owned cells)
template <bool NS, bool CHK>
cudaError_t launch_update_t(ucg_engine* e, const Problem& p0, int mode, const double* Uc, const double* Un, double* Uo,
                     double dt) {
  Problem p = p0;
  p.n = e->n_update;
  const unsigned blocks = (unsigned)((p.n + UPD_CELLS - 1) / UPD_CELLS);
  constexpr int TH = UPD_CELLS * NV;
  cudaError_t err;
  switch (mode) {
    case 0: err = launch_pdl(k_update<NS, 0, CHK>, blocks, TH, e->stream, p, Uc, Un, Uo, dt); break;
    case 1: err = launch_pdl(k_update<NS, 1, CHK>, blocks, TH, e->stream, p, Uc, Un, Uo, dt); break;
    case 2: err = launch_pdl(k_update<NS, 2, CHK>, blocks, TH, e->stream, p, Uc, Un, Uo, dt); break;
    default: err = launch_pdl(k_update<NS, 3, CHK>, blocks, TH, e->stream, p, Uc, Un, Uo, dt); break;
  }
  e->launches += 1;
  return err;
}

// face fluxes, then the residual (mode 0) or RK stage `mode`; check = false
// leaves the new state's physical test to the caller (MOOD's candidate)
int launch_flux(ucg_engine* e, const Problem& p, int mode, const double* Uc, const double* Un, double* Uo, double dt,
                bool check) {
  int rc = launch_faces(e, p, Uc);
  if (rc) return rc;
  const bool ns = e->cfg.governing == 1;
  const cudaError_t err = ns ? check ? launch_update_t<true, true>(e, p, mode, Uc, Un, Uo, dt)
                                     : launch_update_t<true, false>(e, p, mode, Uc, Un, Uo, dt)
                             : check ? launch_update_t<false, true>(e, p, mode, Uc, Un, Uo, dt)
                                     : launch_update_t<false, false>(e, p, mode, Uc, Un, Uo, dt);
  CK(err);
  return UCG_OK;
}

// One RK stage under MOOD (RUNGE_KUTTA3_MOOD, time_p.f90:582-880): the
// candidate into Um from the stage input Uc (step base Un), then the two
// cascades of MOOD_OPERATOR_2 / MOOD_OPERATOR_1 (mood.f90:337-437): PAD_NAD,
// FIX_LIST, the selected cells' faces recomputed (first cascade after the
// MUSCL of the selected reduced cells, second with the flagged cells at
// first order) and their stage redone; the result into Uo.  The second
// cascade's selection stays in mprev (RECALC) for the next reconstruction.
int mood_stage(ucg_engine* e, const Problem& p, int mode, const double* Uc, const double* Un, double* Uo, double dt) {
  double* Um = (double*)e->Um.p;
  int8_t* sel1 = (int8_t*)e->msel.p;
  const ucg_config& c = e->cfg;
  const unsigned blocks = (unsigned)((e->n + 255) / 256);
  int rc;
  if ((rc = launch_recon(e, p, Uc))) return rc;
  if ((rc = launch_flux(e, p, mode, Uc, Un, Um, dt, false))) return rc;
  // first cascade (MOOD_VAR1/2): MUSCL where the reconstruction was reduced
  k_mood_detect<<<blocks, 256, 0, e->stream>>>(p, Uc, Um, c.mood_var[0], c.mood_var[1], c.mood_mode);
  k_mood_fix<<<blocks, 256, 0, e->stream>>>(p, sel1, (int8_t*)e->mmus.p);
  e->launches += 2;
  Problem p1 = p;
  p1.mmus = (int8_t*)e->mmus.p;
  if ((rc = launch_recon(e, p1, Uc))) return rc;
  Problem p2 = p;
  p2.msel = sel1;
  if ((rc = launch_faces(e, p2, Uc))) return rc;
  switch (mode) {
    case 1: k_mood_update<1, false><<<blocks, 256, 0, e->stream>>>(p2, Uc, Un, Um, Um, nullptr, dt); break;
    case 2: k_mood_update<2, false><<<blocks, 256, 0, e->stream>>>(p2, Uc, Un, Um, Um, nullptr, dt); break;
    default: k_mood_update<3, false><<<blocks, 256, 0, e->stream>>>(p2, Uc, Un, Um, Um, nullptr, dt); break;
  }
  // second cascade (MOOD_VAR3/4): first order on the flagged cells
  k_mood_detect<<<blocks, 256, 0, e->stream>>>(p, Uc, Um, c.mood_var[2], c.mood_var[3], c.mood_mode);
  k_mood_fix<<<blocks, 256, 0, e->stream>>>(p, (int8_t*)e->mprev.p, nullptr);
  const int64_t nd = e->n * MF * e->QS * NV;
  if (e->mixed) k_mood_first<float><<<(unsigned)((nd + 255) / 256), 256, 0, e->stream>>>(p);
  else k_mood_first<double><<<(unsigned)((nd + 255) / 256), 256, 0, e->stream>>>(p);
  e->launches += 4;
  Problem p3 = p;
  p3.msel = (int8_t*)e->mprev.p;
  if ((rc = launch_faces(e, p3, Uc))) return rc;
  switch (mode) {
    case 1: k_mood_update<1, true><<<blocks, 256, 0, e->stream>>>(p3, Uc, Un, Um, Uo, sel1, dt); break;
    case 2: k_mood_update<2, true><<<blocks, 256, 0, e->stream>>>(p3, Uc, Un, Um, Uo, sel1, dt); break;
    default: k_mood_update<3, true><<<blocks, 256, 0, e->stream>>>(p3, Uc, Un, Um, Uo, sel1, dt); break;
  }
  e->launches += 1;
  CK(cudaGetLastError());
  return UCG_OK;
}

// one RUNGE_KUTTA3 step; dt from the host value or, if dt_dev, from device
// memory; dt_next: see k_update
int rk3(ucg_engine* e, double dt, double* dt_dev, double* dt_next, double ccfl) {
  Problem p = make_problem(e);
  p.dt_dev = dt_dev;
  p.dt_next = dt_next;
  p.ccfl = ccfl;
  double* Un = (double*)e->Un.p;
  double* Ua = (double*)e->Ua.p;
  double* Ub = (double*)e->Ub.p;
  int rc;
  if (e->cfg.mood) {
    if ((rc = mood_stage(e, p, 1, Un, Un, Ua, dt))) return rc;
    if ((rc = mood_stage(e, p, 2, Ua, Un, Ub, dt))) return rc;
    return mood_stage(e, p, 3, Ub, Un, Un, dt);
  }
  if ((rc = launch_recon(e, p, Un))) return rc;
  if ((rc = launch_flux(e, p, 1, Un, Un, Ua, dt))) return rc;
  if ((rc = launch_recon(e, p, Ua))) return rc;
  if ((rc = launch_flux(e, p, 2, Ua, Un, Ub, dt))) return rc;
  if ((rc = launch_recon(e, p, Ub))) return rc;
  if ((rc = launch_flux(e, p, 3, Ub, Un, Un, dt))) return rc;
  return UCG_OK;
}

// Reverse Cuthill-McKee order of the face-neighbour graph: each connected
// component is numbered breadth first from a pseudo-peripheral cell (the
// far end of two breadth-first sweeps started at a cell of least degree),
// neighbours in order of increasing degree, then the whole order is
// reversed.  Ties are broken by the caller's index, so the order is
// deterministic.  n2o[c] = the caller's cell at position c.
void rcm_order(int64_t n, const int32_t* nfaces, const int32_t* neigh, std::vector<int32_t>& n2o) {
  std::vector<int32_t> deg(n, 0);
  auto nbr = [&](int64_t c, int f) -> int64_t {
    const int64_t y = neigh[c * MF + f];
    return (f < nfaces[c] && y >= 0 && y != c) ? y : -1;
  };
  for (int64_t c = 0; c < n; ++c)
    for (int f = 0; f < MF; ++f) deg[c] += nbr(c, f) >= 0;
  std::vector<int32_t> mark(n, -1), order, queue;
  order.reserve(n);
  queue.reserve(n);
  int32_t stamp = 0;
  // breadth-first sweep from `s` over the unnumbered cells; returns the last
  // level's cell of least degree; appends the visit order to `out` if given
  auto sweep = [&](int64_t s, std::vector<int32_t>* out) -> int64_t {
    const int32_t tag = stamp++;
    queue.clear();
    queue.push_back((int32_t)s);
    mark[s] = tag;
    size_t head = 0, level_start = 0;
    while (head < queue.size()) {
      const size_t level_end = queue.size();
      level_start = head;
      for (; head < level_end; ++head) {
        const int64_t u = queue[head];
        int32_t nb[MF];
        int k = 0;
        for (int f = 0; f < MF; ++f) {
          const int64_t y = nbr(u, f);
          if (y >= 0 && mark[y] != tag && mark[y] != -2) {
            mark[y] = tag;
            nb[k++] = (int32_t)y;
          }
        }
        std::sort(nb, nb + k, [&](int32_t a, int32_t b) { return deg[a] != deg[b] ? deg[a] < deg[b] : a < b; });
        for (int j = 0; j < k; ++j) queue.push_back(nb[j]);
      }
    }
    if (out) out->insert(out->end(), queue.begin(), queue.end());
    int64_t best = queue[level_start];
    for (size_t i = level_start; i < queue.size(); ++i)
      if (deg[queue[i]] < deg[best] || (deg[queue[i]] == deg[best] && queue[i] < best)) best = queue[i];
    return best;
  };
  std::vector<int32_t> comp;
  for (int64_t s0 = 0; s0 < n; ++s0) {
    if (mark[s0] == -2) continue;
    // least-degree cell of this component (found by a first sweep)
    comp.clear();
    sweep(s0, &comp);
    int64_t start = comp[0];
    for (int32_t c : comp)
      if (deg[c] < deg[start] || (deg[c] == deg[start] && c < start)) start = c;
    start = sweep(start, nullptr);
    start = sweep(start, nullptr);
    comp.clear();
    sweep(start, &comp);
    for (int32_t c : comp) mark[c] = -2;  // numbered
    order.insert(order.end(), comp.begin(), comp.end());
  }
  n2o.assign(order.rbegin(), order.rend());
}

// Gather cost of a cell order: over every group of 32 consecutive device
// cells (one warp of the lane-per-cell kernels) and face slot, the number of
// distinct 128-byte lines of the [n][5] FP64 state that the face neighbours
// of the group occupy, averaged.  n2o empty = the caller's order.
double gather_cost(int64_t n, const int32_t* nfaces, const int32_t* neigh, const std::vector<int32_t>& n2o) {
  std::vector<int32_t> o2n;
  if (!n2o.empty()) {
    o2n.assign(n, 0);
    for (int64_t c = 0; c < n; ++c) o2n[n2o[c]] = (int32_t)c;
  }
  double lines = 0.0;
  int64_t slots = 0;
  int64_t ids[32];
  for (int64_t g = 0; g < n; g += 32)
    for (int f = 0; f < MF; ++f) {
      int k = 0;
      for (int64_t c = g; c < g + 32 && c < n; ++c) {
        const int64_t o = n2o.empty() ? c : n2o[c];
        const int64_t y = f < nfaces[o] ? neigh[o * MF + f] : -1;
        if (y >= 0) ids[k++] = (n2o.empty() ? y : o2n[y]) * (NV * 8) / 128;
      }
      if (!k) continue;
      std::sort(ids, ids + k);
      lines += (double)(std::unique(ids, ids + k) - ids);
      ++slots;
    }
  return slots ? lines / (double)slots : 0.0;
}

int cells_in(ucg_engine* e, double* dev_dst, const double* host_src) {
  const size_t bytes = (size_t)e->n * NV * 8;
  if (e->n2o.empty()) {
    CK(cudaMemcpyAsync(dev_dst, host_src, bytes, cudaMemcpyHostToDevice, e->stream));
    return UCG_OK;
  }
  CK(cudaMemcpyAsync(e->permbuf.p, host_src, bytes, cudaMemcpyHostToDevice, e->stream));
  k_perm_rows<true><<<(unsigned)((e->n * NV + 255) / 256), 256, 0, e->stream>>>(
      (const int32_t*)e->d_n2o.p, (const double*)e->permbuf.p, dev_dst, e->n);
  e->launches++;
  CK(cudaGetLastError());
  return UCG_OK;
}

int cells_out(ucg_engine* e, double* host_dst, const double* dev_src) {
  const size_t bytes = (size_t)e->n * NV * 8;
  if (e->n2o.empty()) {
    CK(cudaMemcpyAsync(host_dst, dev_src, bytes, cudaMemcpyDeviceToHost, e->stream));
    return UCG_OK;
  }
  k_perm_rows<false><<<(unsigned)((e->n * NV + 255) / 256), 256, 0, e->stream>>>(
      (const int32_t*)e->d_n2o.p, dev_src, (double*)e->permbuf.p, e->n);
  e->launches++;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(host_dst, e->permbuf.p, bytes, cudaMemcpyDeviceToHost, e->stream));
  return UCG_OK;
}

int cfl_device(ucg_engine* e, double cfl) {
  Problem p = make_problem(e);
  e->dt_slot = 0;
  k_dt_init<<<1, 1, 0, e->stream>>>((double*)e->dt.p);
  k_cfl<<<(unsigned)((e->n + 255) / 256), 256, 0, e->stream>>>(p, (const double*)e->Un.p, cfl / 3.0, (double*)e->dt.p);
  e->launches += 2;
  CK(cudaGetLastError());
  return UCG_OK;
}

}  // namespace ucg_host

using namespace ucg_host;

// =================================================================== ABI
extern "C" {

const char* ucg_create_error(void) { return g_create_err.c_str(); }

int ucg_create(const ucg_config* cfg, int64_t ncells, int device, ucg_engine** out) {
  g_create_err.clear();
  if (!cfg || !out || ncells <= 0) {
    g_create_err = "null argument or ncells <= 0";
    return UCG_EINVAL;
  }
  *out = nullptr;
  const ucg_config& c = *cfg;
  bool okscheme = (c.scheme == 2 || c.scheme == 3) && c.iorder >= 1 && c.iorder <= 4 && (c.ees == 0 || c.ees == 5) &&
                  (c.governing == 1 || c.governing == 2) && (c.precision == UCG_FP64 || c.precision == UCG_MIXED);
  int ideg = (c.iorder + 1) * (c.iorder + 2) * (c.iorder + 3) / 6 - 1;
  if (!okscheme || c.ideg != ideg || c.imax < ideg || c.admis_max < 1 || c.admis_max > 7 || c.nq_quad < 1 ||
      c.nq_quad > UCG_MAX_QP || c.nq_tri < 1 || c.nq_tri > UCG_MAX_QP || (c.ees == 5 && ((c.ideg2 != 3 && c.ideg2 != 9) || c.imax2 < c.ideg2 || c.ideg2 > c.ideg || c.imax2 > c.imax)) ||
      c.gamma <= 1.0 || c.limiter < 1 || c.limiter > 9 || !((c.riemann >= 1 && c.riemann <= 5) || c.riemann == 9) ||
      !(c.wenwrt == 1 || (c.wenwrt == 2 && c.scheme == 3)) || (c.boundtype != 0 && c.boundtype != 1) ||
      (c.reorder != 0 && c.reorder != 1) || (c.mood != 0 && c.mood != 1) ||
      (c.mood && (c.scheme != 3 || c.governing != 2 || (c.mood_mode != 0 && c.mood_mode != 1) ||
                  !(c.mood_var[0] >= 0.0 && c.mood_var[1] >= 0.0 && c.mood_var[2] >= 0.0 && c.mood_var[3] >= 0.0 &&
                    std::isfinite(c.mood_var[0] + c.mood_var[1] + c.mood_var[2] + c.mood_var[3]))))) {
    g_create_err = "unsupported or inconsistent configuration (scheme 2|3, iorder 1..4, ees 0|5, HLLC/Rusanov/Roe/rotated Roe-HLL/t-Roe/HLL, limiter 1..9, "
                   "conserved or (WENO only) characteristic-variable WENO, CWENO lower-order degree 3 or 9, boundtype 0|1, reorder 0|1, "
                   "MOOD 0|1 with WENO, Euler, mode 0|1 and finite non-negative MOOD_VAR1-4)";
    return UCG_EINVAL;
  }
  if (c.scheme == 2 && c.admis_max != 1) {
    g_create_err = "MUSCL uses one stencil (admis_max 1)";
    return UCG_EINVAL;
  }
  int ndev = 0;
  cudaError_t st = cudaGetDeviceCount(&ndev);
  if (st != cudaSuccess || ndev <= device || device < 0) {
    g_create_err = std::string("no usable CUDA device: ") + (st != cudaSuccess ? cudaGetErrorString(st) : "index out of range");
    return UCG_ECUDA;
  }
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, device);
  if (prop.major < 10) {
    g_create_err = "the engine is built for sm_100a (B200); device is sm_" + std::to_string(prop.major * 10 + prop.minor);
    return UCG_ECUDA;
  }
  auto* e = new ucg_engine;
  e->cfg = c;
  e->n = ncells;
  e->device = device;
  e->mixed = c.precision == UCG_MIXED;
  e->QS = c.nq_quad > c.nq_tri ? c.nq_quad : c.nq_tri;
  {
    const char* bulk = std::getenv("UCG_LSQ_BULK");
    e->lsq_bulk = bulk && bulk[0] == '1';
    const char* limit = std::getenv("UCG_LSQ_WAIT");
    e->lsq_limit = limit && limit[0] == '1';
    e->nsm = prop.multiProcessorCount;
  }
  {
    // slices and smoothness blocks padded to 16 bytes (bulk-copy granularity)
    const int64_t ts = e->mixed ? 4 : 8, pad = 16 / ts;
    auto up = [&](int64_t x) { return (x + pad - 1) / pad * pad; };
    Layout& L = e->layout;
    int64_t off = 0;
    for (int ll = 0; ll < c.admis_max; ++ll) {
      bool low = c.ees == 5 && ll > 0;
      int64_t el = low ? (int64_t)c.imax2 * c.ideg2 : (int64_t)c.imax * c.ideg;
      L.soff[ll] = (int)off;
      off += up(el);  // 16-byte aligned slices
    }
    L.tstride = off;
    // smoothness matrices: packed upper triangles (S and the CWENO S2), each
    // row padded to whole 16-byte vectors
    auto tri = [&](int64_t m) {
      int64_t t = 0;
      for (int64_t d = 0; d < m; ++d) t += up(m - d);
      return t;
    };
    L.i2off = (int)tri(c.ideg);
    L.istride = L.i2off + (c.ees == 5 ? tri(c.ideg2) : 0);
  }
  cudaSetDevice(device);
  st = cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking);
  if (st != cudaSuccess) {
    g_create_err = std::string("cudaStreamCreate: ") + cudaGetErrorString(st);
    delete e;
    return UCG_ECUDA;
  }
  const int64_t n = ncells;
  int rc = UCG_OK;
  const size_t T = tsize(e);
  rc = rc ? rc : alloc(e, e->Un, n * NV * 8);
  rc = rc ? rc : alloc(e, e->Ua, n * NV * 8);
  rc = rc ? rc : alloc(e, e->Ub, n * NV * 8);
  rc = rc ? rc : alloc(e, e->rhs, n * NV * 8);
  rc = rc ? rc : alloc(e, e->fflux, (size_t)n * MF * NV * 8);
  if (c.governing == 1) rc = rc ? rc : alloc(e, e->vflux, (size_t)n * MF * NV * 8);
  rc = rc ? rc : alloc(e, e->dul, (size_t)n * MF * e->QS * NV * T);
  const int64_t ngrp = (n + 31) / 32;
  if (!(c.scheme == 2 && c.iorder == 1))
    rc = rc ? rc : alloc(e, e->gbuf, (size_t)ngrp * 32 * c.admis_max * c.ideg * NV * T);
  if (c.scheme == 3 && c.wenwrt == 1) {
    // IORDER 4: smoothness indicators of every stencil in their own kernel
    const char* wis = std::getenv("UCG_WENO_IS");
    const bool own = c.iorder == 4 && !(wis && wis[0] == '0');
    if (own) rc = rc ? rc : alloc(e, e->isb, (size_t)ngrp * 32 * c.admis_max * NV * 8);
    // face values one warp per variable (k_wface), unless UCG_WENO_FACE=0
    const char* wf = std::getenv("UCG_WENO_FACE");
    e->wface = (own || c.iorder < 4) && !(wf && wf[0] == '0');
    if (e->wface) rc = rc ? rc : alloc(e, e->wflag, (size_t)n);
  }
  if (c.mood) {  // RECALC (zero at the start, memory.f90:1002-1005), flags, MOOD_O, candidate
    rc = rc ? rc : alloc(e, e->wflag, (size_t)n);
    rc = rc ? rc : alloc(e, e->mprev, (size_t)n);
    rc = rc ? rc : alloc(e, e->mflag, (size_t)n);
    rc = rc ? rc : alloc(e, e->msel, (size_t)n);
    rc = rc ? rc : alloc(e, e->mmus, (size_t)n);
    rc = rc ? rc : alloc(e, e->mord, (size_t)n);
    rc = rc ? rc : alloc(e, e->Um, n * NV * 8);
    if (!rc && cudaMemset(e->mprev.p, 0, (size_t)n) != cudaSuccess) rc = fail(e, UCG_ECUDA, "cudaMemset failed");
    if (!rc && cudaMemset(e->mord.p, c.iorder + 1, (size_t)n) != cudaSuccess) rc = fail(e, UCG_ECUDA, "cudaMemset failed");
  }
  if (c.wenwrt == 2)  // characteristic WENO: G^T S G of every stencil (15 values)
    rc = rc ? rc : alloc(e, e->qbuf, (size_t)ngrp * 32 * c.admis_max * 15 * 8);
  if (c.wenwrt == 2) rc = rc ? rc : alloc(e, e->wflag, (size_t)n);
  if (c.governing == 1) {
    if (c.scheme == 2 && c.iorder == 1) {
      rc = rc ? rc : alloc(e, e->ulv, (size_t)n * e->QS * 12 * 8);
    } else {
      rc = rc ? rc : alloc(e, e->gv, (size_t)n * c.ideg * 4 * T);
      rc = rc ? rc : alloc(e, e->prim, (size_t)n * 4 * 8);
    }
  }
  rc = rc ? rc : alloc(e, e->health, 64);
  rc = rc ? rc : alloc(e, e->dt, 64);
  rc = rc ? rc : alloc(e, e->partial, ((n + 255) / 256 + 1) * 8);
  rc = rc ? rc : alloc(e, e->red, 64);
  if (rc) {
    g_create_err = e->err;
    ucg_destroy(e);
    return rc;
  }
  cudaMemsetAsync(e->health.p, 0, 64, e->stream);
  cudaMemsetAsync(e->dul.p, 0, e->dul.bytes, e->stream);
  if (e->ulv.p) cudaMemsetAsync(e->ulv.p, 0, e->ulv.bytes, e->stream);
  e->recon_done.assign(n, 0);
  *out = e;
  return UCG_OK;
}

void ucg_destroy(ucg_engine* e) {
  if (!e) return;
  cudaSetDevice(e->device);
  if (e->stream) cudaStreamSynchronize(e->stream);
  DevBuf* all[] = {&e->nfaces, &e->ftype, &e->neigh, &e->nface, &e->bc, &e->qperm, &e->rot, &e->area, &e->dih,
                   &e->vol, &e->minedge, &e->jinv, &e->admis, &e->full, &e->qpts, &e->bmean, &e->sten, &e->invmat,
                   &e->ind, &e->dul, &e->ulv, &e->gv, &e->prim, &e->rhs, &e->Un, &e->Ua, &e->Ub,
                   &e->health, &e->dt, &e->partial, &e->red, &e->staging, &e->own, &e->fflux, &e->vflux, &e->gbuf,
                   &e->qbuf, &e->d_n2o, &e->permbuf, &e->fgrad, &e->isb, &e->wflag, &e->mprev, &e->mflag,
                   &e->msel, &e->mmus, &e->mord, &e->Um, &e->imp_dtl, &e->imp_dinv, &e->imp_off, &e->imp_du,
                   &e->tcell, &e->tset, &e->tiled, &e->setmat, &e->setind,
                   &e->gset, &e->ugrp,
                   &e->dual_hist, &e->dual_part, &e->halo_send, &e->halo_recv, &e->wl_buf};
  for (DevBuf* b : all) release(*b);
  adjoint_release(e);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete e;
}

int ucg_upload_geometry(ucg_engine* e, const ucg_geometry* g) {
  if (!e || !g) return fail(e, UCG_EINVAL, "null argument");
  if (g->ncells != e->n) return fail(e, UCG_EINVAL, "geometry has " + std::to_string(g->ncells) + " cells, engine " + std::to_string(e->n));
  if (!g->nfaces || !g->face_type || !g->neigh || !g->neigh_face || !g->bc || !g->qperm || !g->face_angle ||
      !g->face_area || !g->dih || !g->qpoints || !g->volume || !g->minedge || !g->invccjac ||
      !g->admis || !g->full)
    return fail(e, UCG_EINVAL, "a geometry array is NULL");
  cudaSetDevice(e->device);
  const int64_t n = e->n;
  const int QS = e->QS, ideg = e->cfg.ideg;
  const bool ns = e->cfg.governing == 1;
  if (n >= (int64_t(1) << 28)) return fail(e, UCG_EINVAL, "too many cells (face codes are 32-bit)");
  // validate in the caller's order first (the renumbering follows the
  // neighbour lists, which must be in range)
  for (int64_t c = 0; c < n; ++c) {
    int nf = g->nfaces[c];
    if (nf < 4 || nf > MF) return fail(e, UCG_EINVAL, "cell " + std::to_string(c) + " has " + std::to_string(nf) + " faces");
    if (!(g->volume[c] > 0.0)) return fail(e, UCG_EINVAL, "non-positive cell volume at cell " + std::to_string(c));
    int adm = g->admis[c];
    if (adm < 1 || adm > e->cfg.admis_max) return fail(e, UCG_EINVAL, "ADMIS out of range at cell " + std::to_string(c));
    for (int f = 0; f < nf; ++f) {
      int64_t i = c * MF + f;
      int ft = g->face_type[i];
      if (ft != 5 && ft != 6) return fail(e, UCG_EINVAL, "face type must be 5 or 6");
      int64_t nb = g->neigh[i];
      if (nb >= n || nb < -1) return fail(e, UCG_EINVAL, "neighbour index out of range at cell " + std::to_string(c));
      if (nb >= 0 && (g->neigh_face[i] < 0 || g->neigh_face[i] >= MF))
        return fail(e, UCG_EINVAL, "neighbour face out of range at cell " + std::to_string(c));
      if (nb < 0) {
        int code = g->bc[i];
        if (code != 1 && code != 2 && code != 3 && code != 4 && code != 6)
          return fail(e, UCG_EINVAL, "unsupported boundary code " + std::to_string(code));
      }
      int nq = ft == 5 ? e->cfg.nq_quad : e->cfg.nq_tri;
      for (int q = 0; q < nq; ++q) {
        int qq = g->qperm[i * UCG_MAX_QP + q];
        if (qq < 0 || qq >= nq) return fail(e, UCG_EINVAL, "qperm out of range at cell " + std::to_string(c));
      }
    }
  }
  // device order: n2o[c] = the caller's cell stored at device cell c
  e->n2o.clear();
  e->o2n.clear();
  e->n_recon = e->n_update = n;
  if (!e->roles.empty()) {
    // a partition: stepped cells, then the other reconstructed cells, then
    // the rest, each in the caller's order
    e->n2o.reserve(n);
    for (int r = 0; r < 3; ++r) {
      for (int64_t o = 0; o < n; ++o)
        if (e->roles[o] == r) e->n2o.push_back((int32_t)o);
      if (r == 0) e->n_update = (int64_t)e->n2o.size();
      if (r == 1) e->n_recon = (int64_t)e->n2o.size();
    }
    e->o2n.assign(n, -1);
    for (int64_t c = 0; c < n; ++c) e->o2n[e->n2o[c]] = (int32_t)c;
  } else if (e->cfg.reorder == 1) {
    // reverse Cuthill-McKee, kept only where it gathers from fewer cache
    // lines than the caller's order (a structured or already local order,
    // such as a box numbered row by row, is better left as it is)
    std::vector<int32_t> rcm, none;
    rcm_order(n, g->nfaces, g->neigh, rcm);
    e->cost_caller = gather_cost(n, g->nfaces, g->neigh, none);
    e->cost_rcm = gather_cost(n, g->nfaces, g->neigh, rcm);
    if (e->cost_rcm < 0.95 * e->cost_caller) {
      e->n2o = std::move(rcm);
      e->o2n.assign(n, -1);
      for (int64_t c = 0; c < n; ++c) e->o2n[e->n2o[c]] = (int32_t)c;
    }
  }
  const bool perm = !e->n2o.empty();
  auto src = [&](int64_t c) -> int64_t { return perm ? e->n2o[c] : c; };
  auto dst = [&](int64_t o) -> int64_t { return perm ? e->o2n[o] : o; };
  std::vector<int8_t> nfaces(n), ftype(n * MF), nface(n * MF), bc(n * MF), admis(n), full(n);
  std::vector<int32_t> neigh(n * MF);
  std::vector<uint8_t> qperm((size_t)n * MF * QS);
  std::vector<double> rot((size_t)n * MF * 4), area(n * MF), dih(n * MF), vol(n), minedge(n), jinv(n * 9);
  for (int64_t c = 0; c < n; ++c) {
    const int64_t o = src(c);
    const int nf = g->nfaces[o];
    nfaces[c] = (int8_t)nf;
    admis[c] = (int8_t)g->admis[o];
    full[c] = (int8_t)(g->full[o] ? 1 : 0);
    vol[c] = g->volume[o];
    minedge[c] = g->minedge[o];
    for (int k = 0; k < 9; ++k) jinv[c * 9 + k] = g->invccjac[o * 9 + k];
    for (int f = 0; f < MF; ++f) {
      const int64_t i = c * MF + f, io = o * MF + f;
      ftype[i] = (int8_t)g->face_type[io];
      const int64_t nb = f < nf ? g->neigh[io] : -1;
      neigh[i] = (int32_t)(nb >= 0 ? dst(nb) : -1);
      nface[i] = (int8_t)(f < nf ? g->neigh_face[io] : -1);
      bc[i] = (int8_t)(f < nf ? g->bc[io] : 0);
      area[i] = g->face_area[io];
      dih[i] = g->dih[io];
      double a1 = g->face_angle[io * 2], a2 = g->face_angle[io * 2 + 1];
      rot[i * 4 + 0] = cos(a1);
      rot[i * 4 + 1] = sin(a1);
      rot[i * 4 + 2] = cos(a2);
      rot[i * 4 + 3] = sin(a2);
      if (f < nf) {
        int nq = ftype[i] == 5 ? e->cfg.nq_quad : e->cfg.nq_tri;
        for (int q = 0; q < QS; ++q) qperm[(size_t)i * QS + q] = (uint8_t)(q < nq ? g->qperm[io * UCG_MAX_QP + q] : 0);
      }
    }
  }
  // owned faces, grouped: interior faces, then mirror boundaries (symmetry,
  // slip wall), then the other boundaries (each group in device cell order),
  // so that kernels branching on the face kind see uniform warps.  An
  // interior face belongs to the side of the lower caller index, so the
  // renumbering leaves every face flux bit for bit as it was.  With
  // partition roles only the faces of stepped cells are kept (both their
  // sides are then reconstructed).
  std::vector<int32_t> own, own_mir, own_bnd;
  own.reserve(n * 3);
  for (int64_t c = 0; c < n; ++c)
    for (int f = 0; f < nfaces[c]; ++f) {
      const int64_t nb = neigh[c * MF + f];
      const int32_t code = (int32_t)(c * 8 + f);
      if (c >= e->n_update && (nb < 0 || nb >= e->n_update)) continue;
      if (nb >= 0) {
        const int64_t oc = src(c), onb = src(nb);
        if (oc < onb || (oc == onb && f < nface[c * MF + f])) own.push_back(code);
      } else if (bc[c * MF + f] == 3 || bc[c * MF + f] == 4) {
        own_mir.push_back(code);
      } else {
        own_bnd.push_back(code);
      }
    }
  own.insert(own.end(), own_mir.begin(), own_mir.end());
  e->nown_plain = (int64_t)own.size();
  own.insert(own.end(), own_bnd.begin(), own_bnd.end());
  int rc = UCG_OK;
  rc = rc ? rc : upload(e, e->own, own);
  e->nown = (int64_t)own.size();
  if (ns && !(e->cfg.scheme == 2 && e->cfg.iorder == 1))  // face-point gradients, one record per owned face point
    rc = rc ? rc : alloc(e, e->fgrad, (size_t)e->nown * QS * 12 * 8);
  rc = rc ? rc : upload(e, e->nfaces, nfaces);
  rc = rc ? rc : upload(e, e->ftype, ftype);
  rc = rc ? rc : upload(e, e->neigh, neigh);
  rc = rc ? rc : upload(e, e->nface, nface);
  rc = rc ? rc : upload(e, e->bc, bc);
  rc = rc ? rc : upload(e, e->qperm, qperm);
  rc = rc ? rc : upload(e, e->rot, rot);
  rc = rc ? rc : upload(e, e->area, area);
  rc = rc ? rc : upload(e, e->dih, dih);
  rc = rc ? rc : upload(e, e->vol, vol);
  rc = rc ? rc : upload(e, e->minedge, minedge);
  rc = rc ? rc : upload(e, e->jinv, jinv);
  rc = rc ? rc : upload(e, e->admis, admis);
  rc = rc ? rc : upload(e, e->full, full);
  if (perm) {
    rc = rc ? rc : upload(e, e->d_n2o, e->n2o);
    rc = rc ? rc : alloc(e, e->permbuf, (size_t)n * NV * 8);
  }
  if (rc) return rc;
  e->ntile = 0;  // the tiles follow the cell order; ucg_upload_recon makes them
  // reference-frame quadrature points and basis means, in table precision
  // interleaved over 32-cell groups: element j of cell c at ((c/32)*len + j)*32 + c%32
  const int64_t ngrp = (n + 31) / 32, lq = (int64_t)MF * QS * 3;
  std::vector<double> qp((size_t)ngrp * 32 * lq, 0.0), bm((size_t)ngrp * 32 * ideg, 0.0);
  for (int64_t c = 0; c < n; ++c) {
    const int64_t o = src(c);
    const int64_t gq = (c >> 5) * lq, gb = (c >> 5) * ideg, ln = c & 31;
    for (int f = 0; f < MF; ++f)
      for (int q = 0; q < QS; ++q)
        for (int k = 0; k < 3; ++k)
          qp[(size_t)((gq + (f * QS + q) * 3 + k) * 32 + ln)] = g->qpoints[((o * MF + f) * UCG_MAX_QP + q) * 3 + k];
    if (g->basis_mean)  // else formed by ucg_build_recon
      for (int d = 0; d < ideg; ++d) bm[(size_t)((gb + d) * 32 + ln)] = g->basis_mean[(size_t)o * ideg + d];
  }
  if (e->mixed) {
    std::vector<float> qf(qp.begin(), qp.end()), bf(bm.begin(), bm.end());
    rc = rc ? rc : upload(e, e->qpts, qf);
    rc = rc ? rc : upload(e, e->bmean, bf);
  } else {
    rc = rc ? rc : upload(e, e->qpts, qp);
    rc = rc ? rc : upload(e, e->bmean, bm);
  }
  if (rc) return rc;
  CK(cudaStreamSynchronize(e->stream));
  e->admis_h = std::move(admis);
  e->totvol = 0.0;
  for (int64_t c = 0; c < n; ++c) e->totvol += g->volume[c];
  e->neigh_h = neigh;
  for (int64_t c = 0; c < n; ++c)  // no neighbour past the cell's last face
    for (int f = nfaces[c]; f < MF; ++f) e->neigh_h[(size_t)c * MF + f] = -1;
  e->adj_ready = false;
  e->adjw_ready = false;
  e->have_geometry = true;
  return UCG_OK;
}

}  // extern "C"

// The stencils of cells [first, first + count) (caller order): checked,
// mapped to device numbering, interleaved on the device; the table buffers
// allocated.  rowbuf/d_rowmap (renumbered engines): the device cell that
// takes each row of this upload, for the table expansion; the caller
// releases rowbuf.
int ucg_host::upload_stencils(ucg_engine* e, int64_t first, int64_t count, const int32_t* stencil, DevBuf& rowbuf,
                              const int32_t** d_rowmap) {
  const ucg_config& c = e->cfg;
  const int64_t n = e->n;
  const int A = c.admis_max, W = c.imax + 1;
  const bool cw = c.ees == 5, weno = c.scheme == 3;
  *d_rowmap = nullptr;
  for (int64_t i = 0; i < count; ++i) {
    int64_t cell = first + i;
    for (int ll = 0; ll < A; ++ll)
      for (int k = 0; k < W; ++k) {
        int32_t y = stencil[(i * A + ll) * W + k];
        if (y >= n || y < -1) return fail(e, UCG_EINVAL, "stencil index out of range at cell " + std::to_string(cell));
        // rows 1..nk of the admissible stencils are read by the kernels
        const int nk = cw && ll > 0 ? c.imax2 : c.imax;
        if (y < 0 && ll < e->admis_h[e->o2n.empty() ? cell : e->o2n[cell]] && k >= 1 && k <= nk)
          return fail(e, UCG_EINVAL, "unused slot (-1) inside admissible stencil " + std::to_string(ll) + " of cell " +
                                         std::to_string(cell));
      }
    if (stencil[i * A * W] != cell) return fail(e, UCG_EINVAL, "stencil slot 0 must be the cell itself");
  }
  // stencil indices in device numbering, and which device cell takes each
  // row of this upload (renumbered engines only)
  const bool perm = !e->o2n.empty();
  std::vector<int32_t> sten_dev;
  const int32_t* sten = stencil;
  if (perm) {
    sten_dev.resize((size_t)count * A * W);
    for (size_t j = 0; j < sten_dev.size(); ++j) sten_dev[j] = stencil[j] >= 0 ? e->o2n[stencil[j]] : -1;
    sten = sten_dev.data();
    std::vector<int32_t> rowmap(n, -1);
    for (int64_t i = 0; i < count; ++i) rowmap[e->o2n[first + i]] = (int32_t)i;
    CK(cudaMalloc(&rowbuf.p, (size_t)n * 4));
    CK(cudaMemcpyAsync(rowbuf.p, rowmap.data(), (size_t)n * 4, cudaMemcpyHostToDevice, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    *d_rowmap = (const int32_t*)rowbuf.p;
  }
  auto dcell = [&](int64_t o) -> int64_t { return perm ? e->o2n[o] : o; };
  if (c.scheme == 2 && c.iorder == 1) {  // first stencil kept on the host for the adjoint's reverse map
    e->sten1_h.resize((size_t)n * W, -1);
    for (int64_t i = 0; i < count; ++i)
      for (int k = 0; k < W; ++k) e->sten1_h[(size_t)dcell(first + i) * W + k] = sten[(i * A) * W + k];
    e->adj_ready = false;
  }
  const Layout& Ly = e->layout;
  const size_t T = tsize(e);
  int rc = UCG_OK;
  const int64_t ngrp = (n + 31) / 32;
  rc = rc ? rc : alloc(e, e->sten, (size_t)ngrp * 32 * A * W * 4);
  rc = rc ? rc : alloc(e, e->invmat, (size_t)ngrp * 32 * Ly.tstride * T);
  if (weno) rc = rc ? rc : alloc(e, e->ind, (size_t)ngrp * 32 * Ly.istride * T);
  if (rc) return rc;
  // stencils: staged per cell, interleaved on the device
  rc = alloc(e, e->staging, (size_t)count * A * W * 4);
  if (rc) return rc;
  CK(cudaMemcpyAsync(e->staging.p, sten, (size_t)count * A * W * 4, cudaMemcpyHostToDevice, e->stream));
  int64_t total = (perm ? n : count) * A * W;
  unsigned blocks = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 64);
  k_expand_il<int32_t, int32_t, 1><<<blocks, 256, 0, e->stream>>>((int32_t*)e->sten.p, (const int32_t*)e->staging.p,
                                                              nullptr, first, count, (int64_t)A * W, 0, count,
                                                              *d_rowmap, n);
  e->launches++;
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(e->stream));
  return UCG_OK;
}

namespace {

// Which cells k_lsq_set reconstructs: the cells of a matrix set that at least
// SET_MIN cells share (a quarter of a tile: below that a tile costs more than
// the group of 32 that k_lsq_ring would read), cut into tiles of SET_TILE in
// device order.  set_of gets each table's set, -1 where its cells read their
// own tables.  None where the rows of a stencil do not fit in shared memory
// (k_lsq_set with its rings takes the most of it; IORDER 4 from 701 members in
// FP64, 1,465 in FP32): k_lsq_ring takes any number.  At IORDER 1, whose sets are
// smaller than what a block sets up for them, only where a tile's cells follow one
// another in memory, without CWENO and below 512 cells per SM (14,580 mixed cells,
// 5.4 groups a warp: 28 us tiled, 20 through the ring; hexahedra 13,824: 17, 19;
// 32,768: 26, k_lsq_lane 33; 110,592: 77, 71).  Kept only where it pays:
// a tile is taken to cost three fifths of what its 128 cells cost k_lsq_ring,
// which costs the same for a group of 32 cells whether one or all of them are
// left to it.  Measured, all cells tiled against all through the ring: WENO5
// 64^3 mixed 2.13 / 4.81 ms, 40^3 FP64 1.21 / 2.11, 12^3 FP64 0.058 / 0.090;
// WENO3 48^3 0.193 / 0.298 (mixed), 0.290 / 0.340 (FP64); CWENO4 271,872 cells
// mixed 0.438 / 0.482, 75,776 FP64 0.236 / 0.234.
constexpr int64_t SET_MIN = 32;
int plan_sets(ucg_engine* e, const int32_t* table_id, int64_t ntab, std::vector<int32_t>& set_of, int64_t* tiles) {
  const ucg_config& c = e->cfg;
  const int64_t n = e->n_recon;
  const bool perm = !e->n2o.empty();
  const int64_t vec = e->mixed ? 4 : 2, ts = (int64_t)tsize(e);
  auto row = [&](int nd) { return (nd + vec - 1) / vec * vec; };
  if ((c.iorder == 1 && (c.ees == 5 || n >= (int64_t)e->nsm * 512)) || (c.imax * row(c.ideg) + SET_RING) * ts > (int64_t)SET_SMEM ||
      (c.ees == 5 && c.admis_max > 1 && c.imax2 * row(c.ideg2) * ts > (int64_t)LOW_SMEM))
    return UCG_OK;
  auto table = [&](int64_t cell) { return table_id[perm ? e->n2o[cell] : cell]; };
  std::vector<int64_t> cells(ntab, 0);
  for (int64_t i = 0; i < n; ++i) cells[table(i)]++;
  set_of.assign(ntab, -1);
  std::vector<int64_t> at;  // first tile slot of each set
  int64_t nset = 0, ntile = 0;
  for (int64_t t = 0; t < ntab; ++t)
    if (cells[t] >= SET_MIN) {
      set_of[t] = (int32_t)nset++;
      at.push_back(ntile * SET_TILE);
      ntile += (cells[t] + SET_TILE - 1) / SET_TILE;
    }
  std::vector<int32_t> ugrp;  // groups with cells of their own tables
  for (int64_t g = 0; g < n; g += 32)
    for (int64_t i = g; i < n && i < g + 32; ++i)
      if (set_of[table(i)] < 0) {
        ugrp.push_back((int32_t)(g >> 5));
        break;
      }
  if (!ntile || ntile >= (1 << 30) || 5 * (int64_t)ugrp.size() * 32 + 3 * ntile * SET_TILE > 5 * n) {
    set_of.clear();
    return UCG_OK;
  }
  std::vector<int32_t> tcell((size_t)ntile * SET_TILE, -1), tset((size_t)ntile);
  std::vector<int8_t> tiled((size_t)e->n, 0);
  // 32-cell groups that the tiles' warps touch: one each where the cells of a
  // set follow one another
  std::vector<int64_t> grp((size_t)nset, -1);
  int64_t warps = 0, touched = 0;
  e->all_tiled = true;
  e->ntiled = 0;
  for (int64_t i = 0; i < n; ++i) {
    const int32_t s = set_of[table(i)];
    if (s < 0) {
      e->all_tiled = false;
      continue;
    }
    tset[(size_t)(at[s] / SET_TILE)] = s;
    if (at[s] % 32 == 0) ++warps, grp[(size_t)s] = -1;
    if (grp[(size_t)s] != i >> 5) ++touched, grp[(size_t)s] = i >> 5;
    tcell[(size_t)at[s]++] = (int32_t)i;
    tiled[(size_t)i] = 1;
    e->ntiled++;
  }
  e->tiles_together = touched <= 2 * warps;
  if (c.iorder == 1 && !e->tiles_together) {
    set_of.clear();
    return UCG_OK;
  }
  int64_t off = 0;
  for (int ll = 0; ll < c.admis_max; ++ll) {
    const bool low = c.ees == 5 && ll > 0;
    e->sso[ll] = (int)off;
    off += (int64_t)(low ? c.imax2 : c.imax) * row(low ? c.ideg2 : c.ideg);
  }
  e->sstride = off;
  e->nset = nset;
  int rc = UCG_OK;
  rc = rc ? rc : upload(e, e->tcell, tcell);
  rc = rc ? rc : upload(e, e->tset, tset);
  rc = rc ? rc : upload(e, e->tiled, tiled);
  rc = rc ? rc : alloc(e, e->setmat, (size_t)nset * e->sstride * tsize(e));
  if (c.scheme == 3) rc = rc ? rc : alloc(e, e->setind, (size_t)nset * e->layout.istride * tsize(e));
  std::vector<int32_t> gset((size_t)((n + 31) / 32), -1);
  for (int64_t g = 0; g < n; g += 32) {
    int32_t t = set_of[table(g)];
    for (int64_t i = g; i < n && i < g + 32; ++i)
      if (set_of[table(i)] != t) t = -1;
    gset[(size_t)(g >> 5)] = t;
  }
  rc = rc ? rc : upload(e, e->gset, gset);
  rc = rc ? rc : upload(e, e->ugrp, ugrp);
  e->nugrp = (int64_t)ugrp.size();
  if (rc) return rc;
  CK(cudaStreamSynchronize(e->stream));
  *tiles = ntile;
  return UCG_OK;
}

}  // namespace

// The matrix sets of tables [0, ntab) into the engine's interleaved tables
// for cells [first, first + count): `fill(which, t0, t1, staging)` writes
// the FP64 blocks of tables [t0, t1) into the device staging buffer, the
// pseudo-inverses (which 0, Layout::tstride each: stencil ll's rows at
// soff[ll]) or the packed smoothness matrices (which 1, Layout::istride
// each); they are expanded per cell (d_tid: cell -> table, NULL = the
// cell's own row), pseudo-inverses element by element, smoothness matrices
// by 16-byte vectors, in 512 MiB chunks.
int ucg_host::expand_tables(ucg_engine* e, int64_t first, int64_t count, int64_t ntab, const int32_t* table_id,
                            const int32_t* d_tid, const int32_t* d_rowmap, const std::function<int(int, int64_t, int64_t, double*)>& fill) {
  const Layout& Ly = e->layout;
  const int64_t n = e->n;
  const bool perm = !e->o2n.empty();
  // shared sets, where one call gives every cell's (with chunked uploads the
  // table numbers of one call say nothing about another's)
  e->ntile = 0;
  std::vector<int32_t> set_of;
  int64_t ntile = 0;
  struct Tmp {
    ucg_engine* e;
    DevBuf b;
    ~Tmp() {
      e->bytes -= (int64_t)b.bytes;
      release(b);
    }
  } d_set{e, {}};
  SetLayout SL{};
  if (table_id && first == 0 && count == n && !(e->cfg.scheme == 2 && e->cfg.iorder == 1) && !e->lsq_bulk) {
    int rc = plan_sets(e, table_id, ntab, set_of, &ntile);
    if (rc) return rc;
    if (ntile) {
      const ucg_config& c = e->cfg;
      const int vec = e->mixed ? 4 : 2;
      SL.tstride = Ly.tstride;
      SL.sstride = e->sstride;
      SL.nst = c.admis_max;
      for (int ll = 0; ll < c.admis_max; ++ll) {
        const bool low = c.ees == 5 && ll > 0;
        SL.soff[ll] = Ly.soff[ll];
        SL.sso[ll] = e->sso[ll];
        SL.nk[ll] = low ? c.imax2 : c.imax;
        SL.nd[ll] = low ? c.ideg2 : c.ideg;
        SL.stride[ll] = (SL.nd[ll] + vec - 1) / vec * vec;
      }
      if ((rc = upload(e, d_set.b, set_of))) return rc;
    }
  }
  struct Part {
    int64_t len;
    DevBuf* dst;
    int which;
  } parts[2] = {{Ly.tstride, &e->invmat, 0}, {e->cfg.scheme == 3 ? Ly.istride : 0, &e->ind, 1}};
  const size_t stage_bytes = (size_t)512 << 20;
  for (auto& pt : parts) {
    if (pt.len == 0) continue;
    int64_t per = (int64_t)(stage_bytes / (pt.len * 8));
    if (per < 1) per = 1;
    for (int64_t t0 = 0; t0 < ntab; t0 += per) {
      int64_t t1 = t0 + per < ntab ? t0 + per : ntab;
      size_t bytes = (size_t)(t1 - t0) * pt.len * 8;
      int rc = alloc(e, e->staging, bytes);
      if (rc) return rc;
      rc = fill(pt.which, t0, t1, (double*)e->staging.p);
      if (rc) return rc;
      int64_t total = (perm ? n : count) * pt.len;
      unsigned blocks = (unsigned)std::min<int64_t>((total + 255) / 256, 148 * 64);
      const double* sp = (const double*)e->staging.p;
      if (pt.which == 0 && ntile) {
        const int32_t* so = (const int32_t*)d_set.b.p;
        if (e->mixed) k_pack_sets<float><<<(unsigned)(t1 - t0), 256, 0, e->stream>>>((float*)e->setmat.p, sp, so, t0, SL);
        else k_pack_sets<double><<<(unsigned)(t1 - t0), 256, 0, e->stream>>>((double*)e->setmat.p, sp, so, t0, SL);
        e->launches++;
      }
      if (pt.which == 1 && ntile) {  // the packed triangles as they are
        SetLayout I{};
        I.tstride = I.sstride = pt.len;
        I.nst = 1;
        I.nk[0] = 1;
        I.nd[0] = I.stride[0] = (int)pt.len;
        const int32_t* so = (const int32_t*)d_set.b.p;
        if (e->mixed) k_pack_sets<float><<<(unsigned)(t1 - t0), 256, 0, e->stream>>>((float*)e->setind.p, sp, so, t0, I);
        else k_pack_sets<double><<<(unsigned)(t1 - t0), 256, 0, e->stream>>>((double*)e->setind.p, sp, so, t0, I);
        e->launches++;
      }
      if (e->mixed) {
        if (pt.which == 0)
          k_expand_il<float, double, 1><<<blocks, 256, 0, e->stream>>>((float*)pt.dst->p, sp, d_tid, first, count, pt.len, t0, t1, d_rowmap, n);
        else
          k_expand_il<float, double, 4><<<blocks, 256, 0, e->stream>>>((float*)pt.dst->p, sp, d_tid, first, count, pt.len, t0, t1, d_rowmap, n);
      } else {
        if (pt.which == 0)
          k_expand_il<double, double, 1><<<blocks, 256, 0, e->stream>>>((double*)pt.dst->p, sp, d_tid, first, count, pt.len, t0, t1, d_rowmap, n);
        else
          k_expand_il<double, double, 2><<<blocks, 256, 0, e->stream>>>((double*)pt.dst->p, sp, d_tid, first, count, pt.len, t0, t1, d_rowmap, n);
      }
      e->launches++;
      CK(cudaGetLastError());
      CK(cudaStreamSynchronize(e->stream));
    }
  }
  e->bytes -= (int64_t)e->staging.bytes;
  release(e->staging);
  CK(cudaStreamSynchronize(e->stream));
  e->ntile = ntile;
  return UCG_OK;
}

// cells [first, first + count) have their tables
void ucg_host::mark_recon(ucg_engine* e, int64_t first, int64_t count) {
  int64_t newly = 0;
  for (int64_t i = 0; i < count; ++i)
    if (!e->recon_done[first + i]) {
      e->recon_done[first + i] = 1;
      ++newly;
    }
  e->recon_cells += newly;
}

extern "C" {

int ucg_upload_recon(ucg_engine* e, const ucg_recon* r) {
  if (!e || !r) return fail(e, UCG_EINVAL, "null argument");
  const ucg_config& c = e->cfg;
  if (r->first < 0 || r->count <= 0 || r->first + r->count > e->n) return fail(e, UCG_EINVAL, "cell range out of bounds");
  if (!r->stencil || !r->invmat) return fail(e, UCG_EINVAL, "stencil and invmat are required");
  const bool weno = c.scheme == 3, cw = c.ees == 5;
  if (weno && !r->indicator) return fail(e, UCG_EINVAL, "WENO needs the INDICATOR matrices");
  if (cw && (!r->invmat2 || !r->indicator2)) return fail(e, UCG_EINVAL, "CWENO needs invmat2 and INDICATORC");
  if (!e->have_geometry) return fail(e, UCG_ESTATE, "upload the geometry before the reconstruction tables");
  cudaSetDevice(e->device);
  const int64_t first = r->first, count = r->count;
  const int A = c.admis_max;
  const int64_t ntab = r->table_id ? r->ntables : count;
  if (r->table_id) {
    if (ntab <= 0) return fail(e, UCG_EINVAL, "ntables must be positive with table_id");
    for (int64_t i = 0; i < count; ++i)
      if (r->table_id[i] < 0 || r->table_id[i] >= ntab) return fail(e, UCG_EINVAL, "table_id out of range");
  }
  DevBuf rowbuf;
  const int32_t* d_rowmap = nullptr;
  int rc = upload_stencils(e, first, count, r->stencil, rowbuf, &d_rowmap);
  if (rc) {
    release(rowbuf);
    return rc;
  }
  DevBuf tidbuf;
  int32_t* d_tid = nullptr;
  if (r->table_id) {
    CK(cudaMalloc(&tidbuf.p, count * 4));
    CK(cudaMemcpyAsync(tidbuf.p, r->table_id, count * 4, cudaMemcpyHostToDevice, e->stream));
    d_tid = (int32_t*)tidbuf.p;
  }
  // pack matrix sets into the engine's per-cell block layout on the host
  // (FP64, padding zeroed), stage them in chunks, expand per cell on the GPU
  const Layout& Ly = e->layout;
  const int ideg = c.ideg, imax = c.imax, ideg2 = c.ideg2, imax2 = c.imax2;
  const int vec = e->mixed ? 4 : 2;  // elements per 16-byte vector on the device
  auto pack_mat = [&](int64_t t, double* dst) {
    for (int64_t j = 0; j < Ly.tstride; ++j) dst[j] = 0.0;
    for (int ll = 0; ll < A; ++ll) {
      bool low = cw && ll > 0;
      int nk = low ? imax2 : imax, nd = low ? ideg2 : ideg;
      const double* src = low ? r->invmat2 + ((t * A + ll) * (int64_t)imax2) * ideg2
                              : r->invmat + ((t * A + ll) * (int64_t)imax) * ideg;
      for (int j = 0; j < nk * nd; ++j) dst[Ly.soff[ll] + j] = src[j];
    }
  };
  // upper triangle row by row, each row padded with zeros to whole 16-byte
  // vectors; off-diagonal entries hold S_de + S_ed, so the packed form gives
  // the same quadratic form as the full matrix
  auto pack_tri = [vec](const double* S, int m, double* dst) {
    int j = 0;
    for (int d = 0; d < m; ++d) {
      for (int k = d; k < m; ++k) dst[j + k - d] = k == d ? S[d * m + d] : S[d * m + k] + S[k * m + d];
      j += (m - d + vec - 1) / vec * vec;
    }
  };
  auto pack_ind = [&](int64_t t, double* dst) {
    for (int64_t j = 0; j < Ly.istride; ++j) dst[j] = 0.0;
    pack_tri(r->indicator + t * ideg * ideg, ideg, dst);
    if (cw) pack_tri(r->indicator2 + t * ideg2 * ideg2, ideg2, dst + Ly.i2off);
  };
  std::vector<double> host;
  rc = expand_tables(e, first, count, ntab, r->table_id, d_tid, d_rowmap, [&](int which, int64_t t0, int64_t t1, double* dev) {
    const int64_t len = which == 0 ? Ly.tstride : Ly.istride;
    host.resize((size_t)(t1 - t0) * len);
    for (int64_t t = t0; t < t1; ++t) {
      double* d = host.data() + (t - t0) * len;
      if (which == 0) pack_mat(t, d);
      else pack_ind(t, d);
    }
    CK(cudaMemcpyAsync(dev, host.data(), host.size() * 8, cudaMemcpyHostToDevice, e->stream));
    return (int)UCG_OK;
  });
  if (tidbuf.p) cudaFree(tidbuf.p);
  release(rowbuf);
  if (rc) return rc;
  mark_recon(e, first, count);
  return UCG_OK;
}

int ucg_set_state(ucg_engine* e, const double* u, int64_t n) {
  if (!e || !u) return fail(e, UCG_EINVAL, "null argument");
  if (n != e->n) return fail(e, UCG_EINVAL, "state size mismatch");
  cudaSetDevice(e->device);
  int rc = cells_in(e, (double*)e->Un.p, u);
  if (rc) return rc;
  CK(cudaStreamSynchronize(e->stream));
  e->have_state = true;
  e->dual_ready = false;  // a new state starts a new dual-time history
  return UCG_OK;
}

int ucg_get_state(ucg_engine* e, double* u, int64_t n) {
  if (!e || !u) return fail(e, UCG_EINVAL, "null argument");
  if (n != e->n) return fail(e, UCG_EINVAL, "state size mismatch");
  if (!e->have_state) return fail(e, UCG_ESTATE, "no state set");
  cudaSetDevice(e->device);
  int rc = cells_out(e, u, (const double*)e->Un.p);
  if (rc) return rc;
  CK(cudaStreamSynchronize(e->stream));
  return UCG_OK;
}

int ucg_compute_dt(ucg_engine* e, double cfl, double* dt) {
  if (!e || !dt || !(cfl > 0)) return fail(e, UCG_EINVAL, "bad argument");
  if (!e->have_geometry || !e->have_state) return fail(e, UCG_ESTATE, "geometry and state are needed");
  cudaSetDevice(e->device);
  int rc = cfl_device(e, cfl);
  if (rc) return rc;
  CK(cudaMemcpyAsync(dt, e->dt.p, 8, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  return UCG_OK;
}

int ucg_residual(ucg_engine* e, double* rhs) {
  if (!e) return fail(e, UCG_EINVAL, "null argument");
  if (!ready(e) || !e->have_state) return fail(e, UCG_ESTATE, "geometry, tables and state are needed");
  cudaSetDevice(e->device);
  Problem p = make_problem(e);
  int rc = launch_recon(e, p, (const double*)e->Un.p);
  if (rc) return rc;
  rc = launch_flux(e, p, 0, (const double*)e->Un.p, (const double*)e->Un.p, nullptr, 0.0);
  if (rc) return rc;
  if (rhs) {
    if ((rc = cells_out(e, rhs, (const double*)e->rhs.p))) return rc;
    CK(cudaStreamSynchronize(e->stream));
  }
  return UCG_OK;
}

int ucg_rk3_step(ucg_engine* e, double dt) {
  if (!e || !(dt > 0)) return fail(e, UCG_EINVAL, "bad argument");
  if (!ready(e) || !e->have_state) return fail(e, UCG_ESTATE, "geometry, tables and state are needed");
  cudaSetDevice(e->device);
  return rk3(e, dt);
}

int ucg_step(ucg_engine* e, double cfl, int32_t nsteps) {
  if (!e || !(cfl > 0) || nsteps < 0) return fail(e, UCG_EINVAL, "bad argument");
  if (!ready(e) || !e->have_state) return fail(e, UCG_ESTATE, "geometry, tables and state are needed");
  cudaSetDevice(e->device);
  // The time step of the first step is CALCULATE_CFL's own kernel; each
  // step's last update forms the next step's in the other of two slots.  Not
  // with MOOD, whose last cascade writes the state, nor with partition roles,
  // whose update covers only part of the cells that CALCULATE_CFL covers.
  const bool fuse = !e->cfg.mood && e->n_update == e->n;
  double* dt = (double*)e->dt.p;
  for (int s = 0; s < nsteps; ++s) {
    int rc;
    if (s == 0 || !fuse)
      if ((rc = cfl_device(e, cfl))) return rc;
    double* next = fuse && s + 1 < nsteps ? dt + (e->dt_slot ^ 1) : nullptr;
    if ((rc = rk3(e, 0.0, dt + e->dt_slot, next, cfl / 3.0))) return rc;
    if (next) e->dt_slot ^= 1;
  }
  return UCG_OK;
}

int ucg_last_dt(ucg_engine* e, double* dt) {
  if (!e || !dt) return fail(e, UCG_EINVAL, "null argument");
  cudaSetDevice(e->device);
  CK(cudaMemcpyAsync(dt, (double*)e->dt.p + e->dt_slot, 8, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  return UCG_OK;
}

int ucg_reduce(ucg_engine* e, int32_t what, double* out) {
  if (!e || !out || what < 1 || what > 4) return fail(e, UCG_EINVAL, "bad argument");
  if (!e->have_geometry || !e->have_state) return fail(e, UCG_ESTATE, "geometry and state are needed");
  cudaSetDevice(e->device);
  Problem p = make_problem(e);
  if (what == UCG_REDUCE_ENSTROPHY) {
    if (!(e->cfg.governing == 1 && e->cfg.scheme == 2 && e->cfg.iorder == 1))
      return fail(e, UCG_EINVAL, "enstrophy needs the Navier-Stokes MUSCL (IORDER 1) configuration");
    if (!ready(e)) return fail(e, UCG_ESTATE, "geometry, tables and state are needed");
    int rc = launch_recon(e, p, (const double*)e->Un.p);  // viscous least squares -> ulv
    if (rc) return rc;
  }
  int64_t nb = (e->n + 255) / 256;
  k_reduce_partial<<<(unsigned)nb, 256, 0, e->stream>>>(p, (const double*)e->Un.p, what, (double*)e->partial.p);
  k_reduce_final<<<1, 1024, 0, e->stream>>>((const double*)e->partial.p, nb, (double*)e->red.p);
  e->launches += 2;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(out, e->red.p, 8, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  return UCG_OK;
}

int ucg_check_health(ucg_engine* e) {
  if (!e) return UCG_EINVAL;
  cudaSetDevice(e->device);
  unsigned h = 0;
  CK(cudaMemcpyAsync(&h, e->health.p, sizeof(unsigned), cudaMemcpyDeviceToHost, e->stream));
  CK(cudaMemsetAsync(e->health.p, 0, sizeof(unsigned), e->stream));
  CK(cudaStreamSynchronize(e->stream));
  if (h & HEALTH_TIMEOUT) return fail(e, UCG_ETIMEOUT, "a bounded device wait gave up (reconstruction table pipeline)");
  if (h & HEALTH_NONPHYS) return fail(e, UCG_ENONPHYS, "a stage produced NaN or non-positive density/pressure");
  return UCG_OK;
}

int ucg_synchronize(ucg_engine* e) {
  if (!e) return UCG_EINVAL;
  cudaSetDevice(e->device);
  CK(cudaStreamSynchronize(e->stream));
  return UCG_OK;
}

int ucg_time_kernels(ucg_engine* e, int32_t reps, double* ms) {
  if (!e || !ms || reps < 1) return fail(e, UCG_EINVAL, "bad argument");
  if (!ready(e) || !e->have_state) return fail(e, UCG_ESTATE, "geometry, tables and state are needed");
  cudaSetDevice(e->device);
  Problem p = make_problem(e);
  cudaEvent_t ev[5];
  for (auto& x : ev) CK(cudaEventCreate(&x));
  double acc[4] = {0, 0, 0, 0};
  int rc = UCG_OK;
  const bool split = !(e->cfg.scheme == 2 && e->cfg.iorder == 1);  // least squares, then the rest
  // r = -1: one untimed pass (first launches load the kernels' modules)
  for (int r = -1; r < reps && !rc; ++r) {
    cudaEventRecord(ev[0], e->stream);
    e->mark = split ? ev[4] : nullptr;
    rc = launch_recon(e, p, (const double*)e->Un.p);
    e->mark = nullptr;
    cudaEventRecord(ev[1], e->stream);
    if (!rc) rc = launch_flux(e, p, 0, (const double*)e->Un.p, (const double*)e->Un.p, nullptr, 0.0);
    cudaEventRecord(ev[2], e->stream);
    if (!rc) rc = cfl_device(e, 0.5);
    cudaEventRecord(ev[3], e->stream);
    cudaEventSynchronize(ev[3]);
    if (r < 0) continue;
    float t;
    for (int k = 0; k < 3; ++k) {
      cudaEventElapsedTime(&t, ev[k], ev[k + 1]);
      acc[k] += t;
    }
    cudaEventElapsedTime(&t, ev[0], split ? ev[4] : ev[1]);
    acc[3] += t;
  }
  for (auto& x : ev) cudaEventDestroy(x);
  if (rc) return rc;
  for (int k = 0; k < 4; ++k) ms[k] = acc[k] / reps;
  CK(cudaGetLastError());
  return UCG_OK;
}

int ucg_mood_state(ucg_engine* e, int32_t* order, int32_t* recalc) {
  if (!e) return UCG_EINVAL;
  if (!e->cfg.mood) return fail(e, UCG_EINVAL, "MOOD is off (cfg.mood 0)");
  const int64_t n = e->n;
  std::vector<int8_t> a((size_t)n), b((size_t)n);
  CK(cudaStreamSynchronize(e->stream));
  CK(cudaMemcpy(a.data(), e->mord.p, (size_t)n, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(b.data(), e->mprev.p, (size_t)n, cudaMemcpyDeviceToHost));
  for (int64_t c = 0; c < n; ++c) {
    const int64_t o = e->n2o.empty() ? c : e->n2o[c];  // caller's cell at device position c
    if (order) order[o] = a[c];
    if (recalc) recalc[o] = b[c];
  }
  return UCG_OK;
}

int ucg_set_wait_limit(ucg_engine* e, int64_t polls) {
  if (!e) return UCG_EINVAL;
  e->lsq_wait = polls < 0 ? -1 : (long)polls;
  return UCG_OK;
}

int ucg_shared_sets(const ucg_engine* e, int64_t* cells, int64_t* sets) {
  if (!e) return UCG_EINVAL;
  if (cells) *cells = e->ntile ? e->ntiled : 0;
  if (sets) *sets = e->ntile ? e->nset : 0;
  return UCG_OK;
}

int ucg_cell_order(const ucg_engine* e, int32_t* renumbered, int32_t* n2o, double* cost) {
  if (!e) return UCG_EINVAL;
  if (!e->have_geometry) return UCG_ESTATE;
  if (renumbered) *renumbered = e->n2o.empty() ? 0 : 1;
  if (n2o)
    for (int64_t c = 0; c < e->n; ++c) n2o[c] = e->n2o.empty() ? (int32_t)c : e->n2o[c];
  if (cost) {
    cost[0] = e->cost_caller;
    cost[1] = e->cost_rcm;
  }
  return UCG_OK;
}

void* ucg_get_stream(ucg_engine* e) { return e ? (void*)e->stream : nullptr; }
int64_t ucg_launch_count(const ucg_engine* e) { return e ? e->launches : 0; }
int64_t ucg_device_bytes(const ucg_engine* e) { return e ? e->bytes : 0; }

int ucg_last_error(const ucg_engine* e, char* buf, int32_t len) {
  if (!e || !buf || len <= 0) return UCG_EINVAL;
  std::snprintf(buf, (size_t)len, "%s", e->err.c_str());
  return UCG_OK;
}

}  // extern "C"
