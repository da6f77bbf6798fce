// evp_dyn.cu -- the 2D adapter of include/evp1d.h (evp1d_dyn_*): the
// dyn_evp1d_init / dyn_evp1d_run / dyn_evp1d_finalize interface on global 2D
// arrays, on top of the 1D solver.
//
// The per-timestep conversions are the transfer kernels' index map
// (evp_transfer.cu): they read the list points' cells of the caller's arrays
// and the ice masks (convert_2d_1d_dyn and set_skipMe,
// integration/ice_dyn_evp1d.F90:521-537, 818-882), halo velocities 0
// (:880-881), and write the results to the list points' cells
// (convert_1d_2d_dyn, :884-947).  Arrays that the GPU cannot address are copied
// whole to the device and back.  Cells outside the list keep the values the
// caller passed.
#include <cstdint>
#include <string>
#include <vector>

#include "evp1d.h"
#include "evp_handle.h"
#include "evp_internal.h"

namespace {

// 2D fields of one call on the device, in this order: the 12 per-call inputs
// (strength, cdn_ocn, aiu, uocn, vocn, waterxU, wateryU, forcexU, forceyU,
// umassdti, fmU, Tbu), the 12 stresses, strintxU, strintyU, Cb, uvel, vvel.
constexpr int kIn2d = 12;
constexpr int kF2d = kIn2d + 12 + 3 + 2;  // 29

#define DYN_TRY(x)                                                         \
  do {                                                                     \
    cudaError_t e_ = (x);                                                  \
    if (e_ != cudaSuccess)                                                 \
      return evp::error(e_ == cudaErrorMemoryAllocation ? EVP1D_ERR_NOMEM  \
                                                       : EVP1D_ERR_CUDA,   \
                        "%s: %s", #x, cudaGetErrorString(e_));             \
  } while (0)

}  // namespace

struct evp1d_dyn_handle {
  int nx = 0, ny = 0, na = 0, navel = 0;
  evp1d_t *h = nullptr;
  int32_t *cell = nullptr;   // device: 2D cell (0-based, i fastest) of each list point
  double *f2d = nullptr;     // device: kF2d x nx*ny doubles
  int32_t *mask2d = nullptr; // device: icetmask, iceumask
};

extern "C" {

int evp1d_dyn_init(evp1d_dyn_t **handle, int nx, int ny, int nghost,
                   const int32_t *tmask, const double *dyT, const double *dxT,
                   const double *uarear, const double *HTE, const double *HTN,
                   const evp1d_params *params, int device) {
  if (!handle || !tmask || !dyT || !dxT || !uarear || !HTE || !HTN || !params)
    return evp::error(EVP1D_ERR_INVALID_ARG, "NULL argument");
  *handle = nullptr;
  if (nx < 2 || ny < 2 || nghost < 1)
    return evp::error(EVP1D_ERR_INVALID_ARG, "need nx, ny >= 2 and nghost >= 1");
  if ((long long)nx * ny > 0x7fffffffLL)
    return evp::error(EVP1D_ERR_INVALID_ARG, "nx*ny too large for int32 cell indices");
  int na = 0, navel = 0;
  int rc = evp1d_build_index(nx, ny, nghost, tmask, 0, 0, &na, &navel, nullptr, nullptr,
                             nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr);
  if (rc != EVP1D_OK && rc != EVP1D_ERR_INVALID_ARG) return rc;
  std::vector<int32_t> ti((size_t)na + 1), tj((size_t)na + 1), tij((size_t)navel + 1),
      nb((size_t)6 * (na + 1));
  int32_t *nbp[6];
  for (int k = 0; k < 6; k++) nbp[k] = nb.data() + (size_t)k * (na + 1);
  rc = evp1d_build_index(nx, ny, nghost, tmask, na, navel, &na, &navel, ti.data(), tj.data(),
                         tij.data(), nbp[0], nbp[1], nbp[2], nbp[3], nbp[4], nbp[5]);
  if (rc != EVP1D_OK) return rc;
  // static 1D geometry (convert_2d_1d_init, :803-815): HTEm1 = HTE(i-1,j),
  // HTNm1 = HTN(i,j-1)
  std::vector<int32_t> cell((size_t)na + 1);
  std::vector<double> g((size_t)7 * (na + 1));
  double *G[7];
  for (int k = 0; k < 7; k++) G[k] = g.data() + (size_t)k * (na + 1);
  for (int w = 0; w < na; w++) {
    const size_t c = (size_t)(ti[w] - 1) + (size_t)(tj[w] - 1) * (size_t)nx;
    cell[w] = (int32_t)c;
    G[0][w] = dxT[c];
    G[1][w] = dyT[c];
    G[2][w] = HTE[c];
    G[3][w] = HTN[c];
    G[4][w] = HTE[c - 1];
    G[5][w] = HTN[c - (size_t)nx];
    G[6][w] = uarear[c];
  }
  evp1d_dyn_t *d = new evp1d_dyn_handle();
  d->nx = nx;
  d->ny = ny;
  d->na = na;
  d->navel = navel;
  rc = evp1d_init(&d->h, na, navel, nbp[0], nbp[1], nbp[2], nbp[3], nbp[4], nbp[5], G[0],
                  G[1], G[2], G[3], G[4], G[5], G[6], params, device);
  if (rc != EVP1D_OK) {
    delete d;
    return rc;
  }
  if (na > 0) {
    const size_t cells = (size_t)nx * ny;
    cudaError_t e = evp::device_alloc(&d->cell, sizeof(int32_t) * (size_t)na);
    if (e == cudaSuccess) e = evp::device_alloc(&d->f2d, sizeof(double) * kF2d * cells);
    if (e == cudaSuccess) e = evp::device_alloc(&d->mask2d, sizeof(int32_t) * 2 * cells);
    if (e == cudaSuccess)
      e = cudaMemcpy(d->cell, cell.data(), sizeof(int32_t) * (size_t)na, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      evp1d_dyn_finalize(d);
      return evp::error(e == cudaErrorMemoryAllocation ? EVP1D_ERR_NOMEM : EVP1D_ERR_CUDA,
                        "2D adapter buffers: %s", cudaGetErrorString(e));
    }
  }
  *handle = d;
  return EVP1D_OK;
}

int evp1d_dyn_run(evp1d_dyn_t *d, int ndte, const evp1d_dyn_fields *io) {
  evp::NvtxRange nvtx_range("evp1d_dyn_run");
  if (!d || !io) return evp::error(EVP1D_ERR_INVALID_ARG, "NULL argument");
  const double *in[kIn2d] = {io->strength, io->cdn_ocn, io->aiu, io->uocn, io->vocn,
                             io->waterxU, io->wateryU, io->forcexU, io->forceyU,
                             io->umassdti, io->fmU, io->Tbu};
  for (int k = 0; k < kIn2d; k++)
    if (!in[k] || !io->stress[k]) return evp::error(EVP1D_ERR_INVALID_ARG, "NULL field");
  if (!io->strintxU || !io->strintyU || !io->Cb || !io->uvel || !io->vvel ||
      !io->icetmask || !io->iceumask)
    return evp::error(EVP1D_ERR_INVALID_ARG, "NULL field");
  if (ndte < 0) return evp::error(EVP1D_ERR_INVALID_ARG, "ndte = %d < 0", ndte);
  if (d->na == 0) return EVP1D_OK;
  evp1d_t *h = d->h;
  evp::DeviceProblem &P = h->d;
  DYN_TRY(cudaSetDevice(P.device));
  const size_t cells = (size_t)d->nx * d->ny;
  evp::UploadFields f;
  evp::DownloadFields o;
  for (int k = 0; k < 12; k++) {
    f.in[k] = in[k];
    f.stress[k] = io->stress[k];
    o.stress[k] = io->stress[k];
  }
  f.u = o.u = io->uvel;
  f.v = o.v = io->vvel;
  f.strintx = o.strintx = io->strintxU;
  f.strinty = o.strinty = io->strintyU;
  f.Cb = o.Cb = io->Cb;
  f.skT = io->icetmask;
  f.skU = io->iceumask;
  f.mask = f.zero_halo = true;
  f.n_f = f.n_uv = o.n_f = o.n_u = cells;
  f.map_f = o.map_f = d->cell;
  f.stage = o.stage = d->f2d;
  f.stage_step = o.stage_step = cells;
  f.istage = d->mask2d;
  evp::adjoint_invalidate(h->adj);
  h->uinit_explicit = false;
  int rc = evp::settle(h, evp::problem_upload(&P, f, h->p.rhow, false));
  if (rc != EVP1D_OK) return rc;
  h->uploaded = true;
  h->sets_differ = false;
  rc = evp::settle(h, evp1d_subcycles(h, ndte));
  if (rc != EVP1D_OK) return rc;
  int code = 0;
  rc = evp::settle(h, evp::problem_download(&P, o, &code));
  if (rc != EVP1D_OK) return rc;
  return code ? evp::timeout_error(code) : EVP1D_OK;
}

int evp1d_dyn_finalize(evp1d_dyn_t *d) {
  if (!d) return EVP1D_OK;
  int rc = EVP1D_OK;
  if (d->h) {
    cudaSetDevice(d->h->d.device);
    if (d->cell) cudaFree(d->cell);
    if (d->f2d) cudaFree(d->f2d);
    if (d->mask2d) cudaFree(d->mask2d);
    rc = evp1d_finalize(d->h);
  }
  delete d;
  return rc;
}

int evp1d_dyn_sizes(evp1d_dyn_t *d, int *na, int *navel) {
  if (!d || !na || !navel) return evp::error(EVP1D_ERR_INVALID_ARG, "NULL argument");
  *na = d->na;
  *navel = d->navel;
  return EVP1D_OK;
}

}  // extern "C"
