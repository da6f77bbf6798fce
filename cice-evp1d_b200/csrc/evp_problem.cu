// evp_problem.cu -- device arena of one 1D problem and the kernels' views of it.
#include <vector>

#include "evp_internal.h"

namespace evp {

namespace {

#define CUDA_TRY(x)                                                        \
  do {                                                                     \
    cudaError_t e_ = (x);                                                  \
    if (e_ != cudaSuccess)                                                 \
      return error(e_ == cudaErrorMemoryAllocation ? EVP1D_ERR_NOMEM       \
                                                   : EVP1D_ERR_CUDA,       \
                   "%s: %s", #x, cudaGetErrorString(e_));                  \
  } while (0)

#define TRY(x)               \
  do {                       \
    int rc_ = (x);           \
    if (rc_) return rc_;     \
  } while (0)

size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

// Bump allocator over one cudaMalloc.
struct Carve {
  char *base = nullptr;
  size_t off = 0;
  template <class T>
  void take(T **p, size_t count) {
    const size_t b = align_up((count > 0 ? count : 1) * sizeof(T));
    if (base) *p = (T *)(base + off);
    off += b;
  }
};

int h2d(void *dst, const void *src, size_t bytes, cudaStream_t st) {
  if (bytes == 0) return EVP1D_OK;
  CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
  return EVP1D_OK;
}

void layout(DeviceProblem *d, Carve &c, size_t nhalo_total, size_t nuvx_total,
            size_t ndep_total) {
  const size_t R = (size_t)d->res_blocks * (size_t)d->res_threads;
  const size_t S = (size_t)d->nslots, U = (size_t)d->nuv, T = (size_t)d->ntiles;
  c.take(&d->err, 1);
  c.take(&d->cflags, 1);
  c.take(&d->meta, S);
  c.take(&d->lcor, S);
  c.take(&d->halo_lcc, nhalo_total);
  c.take(&d->halo_lcor, nhalo_total);
  c.take(&d->uvx_off, T);
  c.take(&d->uvx_cnt, T);
  c.take(&d->uvx_idx, nuvx_total);
  c.take(&d->tile_meta, 8 * T);
  c.take(&d->tile_rec, (size_t)kRecInts * T);
  c.take(&d->cblk, (size_t)kConstFields * kConstTileSlots * T);
  c.take(&d->run_off, (size_t)d->nruns + 1);
  c.take(&d->dep_off, T + 1);
  c.take(&d->dep_idx, ndep_total);
  c.take(&d->epoch, T);
  c.take(&d->tile_off, T);
  c.take(&d->tile_cnt, T);
  c.take(&d->halo_off, T);
  c.take(&d->halo_cnt, T);
  c.take(&d->halo_idx, nhalo_total);
  c.take(&d->slot_of_point, (size_t)d->na);
  c.take(&d->point_of_slot, S);
  c.take(&d->tile_of_quad, S / kSlotAlign);
  for (int k = 0; k < 6; k++) c.take(&d->nb[k], S);
  c.take(&d->lnb, S);
  c.take(&d->flags, S);
  for (int k = 0; k < kNumGeo; k++) c.take(&d->geo[k], S);
  for (int k = 0; k < kNumDyn; k++) c.take(&d->dyn[k], S);
  for (int b = 0; b < 2; b++) {
    for (int k = 0; k < 12; k++) c.take(&d->stress[b][k], S);
    c.take(&d->u[b], U);
    c.take(&d->v[b], U);
  }
  c.take(&d->strintx, S);
  c.take(&d->strinty, S);
  c.take(&d->Cb, S);
  for (int k = 0; k < 8; k++) c.take(&d->str[k], U);
  if (d->res_blocks > 0) {
    c.take(&d->res_slot, R);
    c.take(&d->res_cnt, (size_t)d->res_blocks);
    c.take(&d->res_corner, 4 * R);
    c.take(&d->res_str, R);
    c.take(&d->res_mail, 2 * S);
  }
  c.take(&d->stage, (size_t)32 * (size_t)(d->navel > 0 ? d->navel : 1));
}

}  // namespace

int problem_create(DeviceProblem *d, int device, const TilePlan &plan,
                   const ResidentPlan &res, const double *const geo[kNumGeo]) {
  d->device = device;
  d->na = plan.na;
  d->navel = plan.navel;
  d->nslots = plan.nslots;
  d->nhs = plan.nhalo_slots;
  d->nuv = plan.nslots + plan.nhalo_slots;
  d->ntiles = plan.ntiles;
  d->nruns = plan.nruns;
  d->from_coords = plan.from_coords;
  CUDA_TRY(cudaSetDevice(device));
  CUDA_TRY(cudaStreamCreateWithFlags(&d->stream, cudaStreamNonBlocking));
  CUDA_TRY(cudaDeviceGetAttribute(&d->nctas, cudaDevAttrMultiProcessorCount, device));
  int short_of;
  const cudaError_t e = tma_prepare(&short_of);
  if (short_of)
    return error(EVP1D_ERR_CUDA, "the subcycle kernel was compiled with fewer than the %d "
                 "registers a thread that its roles share out", short_of);
  if (e != cudaSuccess) return error(EVP1D_ERR_CUDA, "subcycle kernel: %s", cudaGetErrorString(e));
  if (res.nblocks > 0 && resident_prepare(device, res.quad, res.cls, res.nblocks)) {
    d->res_quad = res.quad;
    d->res_blocks = res.nblocks;
    d->res_threads = res.threads;
    d->res_cls = res.cls;
  }
  pinned_hold(d);
  Carve sizing;
  layout(d, sizing, plan.halo_idx.size(), plan.uvx_idx.size(), plan.dep_idx.size());
  CUDA_TRY(device_alloc(&d->arena, sizing.off));
  d->arena_bytes = sizing.off;
  Carve c;
  c.base = (char *)d->arena;
  layout(d, c, plan.halo_idx.size(), plan.uvx_idx.size(), plan.dep_idx.size());
  cudaStream_t st = d->stream;
  CUDA_TRY(cudaMemsetAsync(d->arena, 0, d->arena_bytes, st));
  if (d->na == 0) {
    CUDA_TRY(cudaStreamSynchronize(st));
    return EVP1D_OK;
  }
  const size_t T = (size_t)d->ntiles * sizeof(int32_t);
  const size_t S4 = (size_t)d->nslots * sizeof(int32_t);
  TRY(h2d(d->run_off, plan.run_off.data(), plan.run_off.size() * sizeof(int32_t), st));
  TRY(h2d(d->dep_off, plan.dep_off.data(), plan.dep_off.size() * sizeof(int32_t), st));
  TRY(h2d(d->dep_idx, plan.dep_idx.data(), plan.dep_idx.size() * sizeof(int32_t), st));
  TRY(h2d(d->tile_off, plan.tile_off.data(), T, st));
  TRY(h2d(d->tile_cnt, plan.tile_cnt.data(), T, st));
  TRY(h2d(d->halo_off, plan.halo_off.data(), T, st));
  TRY(h2d(d->halo_cnt, plan.halo_cnt.data(), T, st));
  TRY(h2d(d->halo_idx, plan.halo_idx.data(), plan.halo_idx.size() * sizeof(int32_t), st));
  TRY(h2d(d->slot_of_point, plan.slot_of_point.data(), (size_t)d->na * sizeof(int32_t), st));
  TRY(h2d(d->point_of_slot, plan.point_of_slot.data(), S4, st));
  std::vector<int32_t> quad((size_t)d->nslots / kSlotAlign);
  for (int t = 0; t < d->ntiles; t++)
    for (int s = plan.tile_off[t]; s < plan.tile_off[t] + plan.tile_cnt[t]; s += kSlotAlign)
      quad[s / kSlotAlign] = t;
  TRY(h2d(d->tile_of_quad, quad.data(), quad.size() * sizeof(int32_t), st));
  const std::vector<int32_t> *nbv[6] = {&plan.ee, &plan.ne, &plan.se,
                                        &plan.nw, &plan.sw, &plan.sse};
  for (int k = 0; k < 6; k++) TRY(h2d(d->nb[k], nbv[k]->data(), S4, st));
  TRY(h2d(d->lnb, plan.lnb.data(), S4, st));
  TRY(h2d(d->meta, plan.lnb.data(), S4, st));
  TRY(h2d(d->lcor, plan.lcor.data(), S4, st));
  const size_t H4 = plan.halo_idx.size() * sizeof(uint32_t);
  TRY(h2d(d->halo_lcc, plan.halo_lcc.data(), H4, st));
  TRY(h2d(d->halo_lcor, plan.halo_lcor.data(), H4, st));
  TRY(h2d(d->uvx_off, plan.uvx_off.data(), T, st));
  TRY(h2d(d->uvx_cnt, plan.uvx_cnt.data(), T, st));
  TRY(h2d(d->uvx_idx, plan.uvx_idx.data(), plan.uvx_idx.size() * sizeof(int32_t), st));
  std::vector<int32_t> tm((size_t)8 * d->ntiles, 0);
  for (int t = 0; t < d->ntiles; t++) {
    int32_t *q = tm.data() + (size_t)8 * t;
    q[0] = plan.tile_off[t];
    q[1] = plan.tile_cnt[t];
    q[2] = plan.uvx_off[t];
    q[3] = plan.uvx_cnt[t];
    q[4] = plan.halo_off[t];
    q[5] = plan.halo_cnt[t];
  }
  TRY(h2d(d->tile_meta, tm.data(), tm.size() * sizeof(int32_t), st));
  std::vector<int32_t> rec((size_t)kRecInts * d->ntiles, 0);
  for (int t = 0; t < d->ntiles; t++) {
    int32_t *q = rec.data() + (size_t)kRecInts * t;
    const int nx = plan.uvx_cnt[t], nh = plan.halo_cnt[t];
    q[0] = plan.tile_off[t];
    q[1] = plan.tile_cnt[t];
    q[2] = nx;
    q[3] = nh;
    for (int x = 0; x < nx; x++) q[kRecUvx + x] = plan.uvx_idx[plan.uvx_off[t] + x];
    for (int h = 0; h < nh; h++) {
      q[kRecHalo + h] = plan.halo_idx[plan.halo_off[t] + h];
      q[kRecHLcor + h] = (int32_t)plan.halo_lcor[plan.halo_off[t] + h];
      q[kRecHLcc + h] = (int32_t)plan.halo_lcc[plan.halo_off[t] + h];
    }
  }
  TRY(h2d(d->tile_rec, rec.data(), rec.size() * sizeof(int32_t), st));
  if (d->res_blocks > 0) {
    TRY(h2d(d->res_slot, res.slot.data(), res.slot.size() * sizeof(int32_t), st));
    TRY(h2d(d->res_cnt, res.cnt.data(), res.cnt.size() * sizeof(int32_t), st));
    TRY(h2d(d->res_corner, res.corner.data(), res.corner.size() * sizeof(int32_t), st));
    TRY(h2d(d->res_str, res.str.data(), res.str.size() * sizeof(uint32_t), st));
  }
  // geometry: reference order -> staging -> slots
  PermBatch b;
  for (int k = 0; k < kNumGeo; k++) {
    double *src = d->stage + (size_t)k * d->navel;
    TRY(h2d(src, geo[k], (size_t)d->na * sizeof(double), st));
    b.src[b.n] = src;
    b.dst[b.n] = d->geo[k];
    b.n++;
  }
  launch_scatter(b, d->nslots, d->point_of_slot, st);
  // every slot skipped until an upload (padding slots stay so), and the
  // constant blocks' geometry and padding
  launch_skip_all(d->nslots, d->flags, d->lnb, d->meta, st);
  TRY(problem_fill_const(d));
  CUDA_TRY(cudaGetLastError());
  CUDA_TRY(cudaStreamSynchronize(st));
  return EVP1D_OK;
}

void problem_destroy(DeviceProblem *d) {
  if (d->stream) {
    cudaSetDevice(d->device);
    cudaStreamSynchronize(d->stream);
  }
  if (d->arena) cudaFree(d->arena);
  if (d->uv_pos) cudaFree(d->uv_pos);
  pinned_release(d);
  d->uv_pos = nullptr;
  if (d->stream) cudaStreamDestroy(d->stream);
  d->arena = nullptr;
  d->stream = nullptr;
}

int problem_fill_const(DeviceProblem *d) {
  if (d->ntiles == 0) return EVP1D_OK;
  const double *src[kConstFields - 1] = {
      d->geo[kDxT],  d->geo[kDyT],    d->geo[kHTE],    d->geo[kHTN],    d->geo[kHTEm1],
      d->geo[kHTNm1], d->dyn[kStrength], d->dyn[kKvrel], d->dyn[kUocn], d->dyn[kVocn],
      d->dyn[kWaterx], d->dyn[kWatery], d->dyn[kForcex], d->dyn[kForcey], d->dyn[kUmassdti],
      d->dyn[kFm],   d->geo[kUarear], d->dyn[kTbu],    d->dyn[kUinit],  d->dyn[kVinit]};
  CUDA_TRY(cudaMemsetAsync(d->cflags, 0, sizeof(int), d->stream));
  launch_const_blocks(d->ntiles, d->tile_off, d->tile_cnt, src, d->meta, d->lcor, d->cblk,
                      d->cflags, d->stream);
  CUDA_TRY(cudaGetLastError());
  return EVP1D_OK;
}

DevState problem_inplace_view(const DeviceProblem &d) {
  DevState s;
  const int c = d.cur;
  s.na = d.nslots;
  s.navel = d.nuv;
  s.ee = d.nb[0];
  s.ne = d.nb[1];
  s.se = d.nb[2];
  s.nw = d.nb[3];
  s.sw = d.nb[4];
  s.sse = d.nb[5];
  s.flags = d.flags;
  s.dxT = d.geo[kDxT];
  s.dyT = d.geo[kDyT];
  s.HTE = d.geo[kHTE];
  s.HTN = d.geo[kHTN];
  s.HTEm1 = d.geo[kHTEm1];
  s.HTNm1 = d.geo[kHTNm1];
  s.uarear = d.geo[kUarear];
  s.strength = d.dyn[kStrength];
  s.Cw = d.dyn[kCw];
  s.aiu = d.dyn[kAiu];
  s.uocn = d.dyn[kUocn];
  s.vocn = d.dyn[kVocn];
  s.waterx = d.dyn[kWaterx];
  s.watery = d.dyn[kWatery];
  s.forcex = d.dyn[kForcex];
  s.forcey = d.dyn[kForcey];
  s.umassdti = d.dyn[kUmassdti];
  s.fm = d.dyn[kFm];
  s.Tbu = d.dyn[kTbu];
  s.uinit = d.dyn[kUinit];
  s.vinit = d.dyn[kVinit];
  for (int k = 0; k < 12; k++) s.stress[k] = d.stress[c][k];
  s.u = d.u[c];
  s.v = d.v[c];
  for (int k = 0; k < 8; k++) s.str[k] = d.str[k];
  s.strintx = d.strintx;
  s.strinty = d.strinty;
  s.Cb = d.Cb;
  return s;
}

FusedArgs problem_fused_args(const DeviceProblem &d, int from) {
  FusedArgs a;
  const int to = 1 - from;
  a.ntiles = d.ntiles;
  a.nruns = d.nruns;
  a.run_off = d.run_off;
  a.tile_off = d.tile_off;
  a.tile_cnt = d.tile_cnt;
  a.halo_off = d.halo_off;
  a.halo_cnt = d.halo_cnt;
  a.halo_idx = d.halo_idx;
  a.flags = d.flags;
  a.ee = d.nb[0];
  a.ne = d.nb[1];
  a.se = d.nb[2];
  a.lnb = d.lnb;
  a.dxT = d.geo[kDxT];
  a.dyT = d.geo[kDyT];
  a.HTE = d.geo[kHTE];
  a.HTN = d.geo[kHTN];
  a.HTEm1 = d.geo[kHTEm1];
  a.HTNm1 = d.geo[kHTNm1];
  a.uarear = d.geo[kUarear];
  a.strength = d.dyn[kStrength];
  a.kvrel = d.dyn[kKvrel];
  a.uocn = d.dyn[kUocn];
  a.vocn = d.dyn[kVocn];
  a.waterx = d.dyn[kWaterx];
  a.watery = d.dyn[kWatery];
  a.forcex = d.dyn[kForcex];
  a.forcey = d.dyn[kForcey];
  a.umassdti = d.dyn[kUmassdti];
  a.fm = d.dyn[kFm];
  a.Tbu = d.dyn[kTbu];
  a.uinit = d.dyn[kUinit];
  a.vinit = d.dyn[kVinit];
  a.u_in = d.u[from];
  a.v_in = d.v[from];
  a.u_out = d.u[to];
  a.v_out = d.v[to];
  for (int k = 0; k < 12; k++) {
    a.s_in[k] = d.stress[from][k];
    a.s_out[k] = d.stress[to][k];
  }
  a.strintx = d.strintx;
  a.strinty = d.strinty;
  a.Cb = d.Cb;
  for (int k = 0; k < 8; k++) a.str_out[k] = d.str[k];
  return a;
}

TmaArgs problem_tma_args(const DeviceProblem &d, int from) {
  TmaArgs a;
  const int to = 1 - from;
  a.ntiles = d.ntiles;
  a.nruns = d.nruns;
  a.run_off = d.run_off;
  a.tile_off = d.tile_off;
  a.tile_cnt = d.tile_cnt;
  a.halo_off = d.halo_off;
  a.halo_cnt = d.halo_cnt;
  a.halo_idx = d.halo_idx;
  a.uvx_off = d.uvx_off;
  a.uvx_cnt = d.uvx_cnt;
  a.uvx_idx = d.uvx_idx;
  a.meta = d.meta;
  a.lcor = d.lcor;
  a.halo_lcc = d.halo_lcc;
  a.halo_lcor = d.halo_lcor;
  a.tile_meta = d.tile_meta;
  a.tile_rec = d.tile_rec;
  const int geo_order[6] = {kDxT, kDyT, kHTE, kHTN, kHTEm1, kHTNm1};
  for (int k = 0; k < 6; k++) a.sg[k] = d.geo[geo_order[k]];
  a.sg[6] = d.dyn[kStrength];
  a.cblk = d.cblk;
  a.cflags = d.cflags;
  a.compact = d.compact_allowed;
  a.u[0] = d.u[from];
  a.v[0] = d.v[from];
  a.u[1] = d.u[to];
  a.v[1] = d.v[to];
  for (int k = 0; k < 12; k++) {
    a.s[0][k] = d.stress[from][k];
    a.s[1][k] = d.stress[to][k];
  }
  a.strintx = d.strintx;
  a.strinty = d.strinty;
  a.Cb = d.Cb;
  for (int k = 0; k < 8; k++) a.str_out[k] = d.str[k];
  a.dep_off = d.dep_off;
  a.dep_idx = d.dep_idx;
  a.err = d.err;
  return a;
}

cudaError_t problem_launch_resident(DeviceProblem *d, const Params &p, int nsub, bool last,
                                    double *const s_in[12], double *const s_out[12],
                                    const double *u_in, const double *v_in, double *u_out,
                                    double *v_out, size_t uv_step) {
  ResidentArgs a;
  a.nslots = d->nslots;
  a.slot = d->res_slot;
  a.cnt = d->res_cnt;
  a.corner = d->res_corner;
  a.str_idx = d->res_str;
  a.flags = d->flags;
  const int geo_order[6] = {kDxT, kDyT, kHTE, kHTN, kHTEm1, kHTNm1};
  for (int k = 0; k < 6; k++) a.sg[k] = d->geo[geo_order[k]];
  a.sg[6] = d->dyn[kStrength];
  const double *uf[kTmaStepuFields] = {
      d->dyn[kKvrel],  d->dyn[kUocn],     d->dyn[kVocn], d->dyn[kWaterx],
      d->dyn[kWatery], d->dyn[kForcex],   d->dyn[kForcey], d->dyn[kUmassdti],
      d->dyn[kFm],     d->geo[kUarear],   d->dyn[kTbu],  d->dyn[kUinit],
      d->dyn[kVinit]};
  for (int k = 0; k < kTmaStepuFields; k++) a.uf[k] = uf[k];
  for (int k = 0; k < 12; k++) {
    a.s_in[k] = s_in[k];
    a.s_out[k] = s_out[k];
  }
  a.u_in = u_in;
  a.v_in = v_in;
  a.u_out = u_out;
  a.v_out = v_out;
  a.uv_step = uv_step;
  a.strintx = d->strintx;
  a.strinty = d->strinty;
  a.Cb = d->Cb;
  for (int k = 0; k < 8; k++) a.str_out[k] = d->str[k];
  a.nsub = nsub;
  a.last = last;
  a.mail = d->res_mail;
  a.seq = d->res_seq;
  a.err = d->err;
  d->res_seq += (unsigned)nsub;
  return launch_resident(a, p, d->res_quad, d->res_cls, d->res_threads, d->res_blocks, d->stream);
}

int problem_take_error(DeviceProblem *d, int *code) {
  int v = 0;
  int *word = pinned_word(d), *to = word ? word : &v;
  CUDA_TRY(cudaMemcpyAsync(to, d->err, sizeof(int), cudaMemcpyDeviceToHost, d->stream));
  CUDA_TRY(cudaStreamSynchronize(d->stream));
  v = *to;
  if (v) CUDA_TRY(cudaMemsetAsync(d->err, 0, sizeof(int), d->stream));
  *code = v;
  return EVP1D_OK;
}

}  // namespace evp
