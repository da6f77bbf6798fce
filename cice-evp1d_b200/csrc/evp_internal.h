// evp_internal.h -- library-internal state shared by the C-ABI translation
// units (not part of the public ABI).
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "evp1d.h"
#include "evp_kernels.cuh"
#include "evp_resident.h"
#include "evp_tiles.h"

namespace evp {

// Record `fmt` as this thread's last error message and return `code`.
int error(int code, const char *fmt, ...);
// EVP1D_ERR_TIMEOUT for the error word's `code`.
int timeout_error(int code);

// A named NVTX range over a scope, so that the public calls show on a
// profiler's timeline (header-only NVTX; without a profiler it does nothing).
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};

// Every device allocation of the library: cudaMalloc, unless the failure
// injection of evp1d_debug_fail_alloc picks this allocation, which then
// fails with cudaErrorMemoryAllocation and allocates nothing.
cudaError_t device_alloc(void **p, size_t bytes);
template <class T>
cudaError_t device_alloc(T **p, size_t bytes) {
  return device_alloc(reinterpret_cast<void **>(p), bytes);
}

// A launch whose blocks wait on one another, so all must be resident at once.
// Refused (launch_refused of its result; nothing has been launched) where less
// of the device is free to this context, and by evp1d_debug_refuse_launch.
cudaError_t launch_cooperative(const void *kernel, dim3 grid, dim3 block, void **args,
                               size_t smem, cudaStream_t st);
bool launch_refused(cudaError_t e);

// Per-call input fields in the order they are staged and scattered.
enum DynField {
  kStrength, kCw, kAiu, kUocn, kVocn, kWaterx, kWatery, kForcex, kForcey,
  kUmassdti, kFm, kTbu, kUinit, kVinit, kKvrel, kNumDyn
};
enum GeoField { kDxT, kDyT, kHTE, kHTN, kHTEm1, kHTNm1, kUarear, kNumGeo };

// The 1D problem on one GPU in slot order (tiles of the TilePlan), with the
// reference's halo slots appended after the nslots list slots for u, v, str.
struct DeviceProblem {
  int device = 0;
  cudaStream_t stream = nullptr;
  int na = 0, navel = 0, nslots = 0, nhs = 0, nuv = 0, ntiles = 0;
  bool from_coords = false;
  void *arena = nullptr;
  size_t arena_bytes = 0;
  // tile plan
  int nruns = 0;                 // CTAs of the subcycle kernel
  int32_t *run_off = nullptr;    // [nruns + 1] tile ranges of the runs
  int32_t *tile_off = nullptr, *tile_cnt = nullptr, *halo_off = nullptr;
  int32_t *halo_cnt = nullptr, *halo_idx = nullptr;
  int32_t *slot_of_point = nullptr, *point_of_slot = nullptr;
  int32_t *tile_of_quad = nullptr;  // tile of slots 4q..4q+3
  // batched: caller's position of each list point, then each halo slot
  int32_t *uv_pos = nullptr;
  int *err_host = nullptr;  // page-locked copy of the error word (pinned_word)
  bool pins = false;        // holds a reference to the page-locked pool
  unsigned pin_gen = 0;     // as it was then
  int32_t *nb[6] = {};  // ee ne se nw sw sse, slot space
  uint32_t *lnb = nullptr;   // static packed stepu neighbours
  uint32_t *meta = nullptr;  // lnb | skip flags << 30 (per call)
  uint32_t *lcor = nullptr;  // packed stress corner velocity indices
  uint32_t *halo_lcc = nullptr, *halo_lcor = nullptr;
  int32_t *uvx_off = nullptr, *uvx_cnt = nullptr, *uvx_idx = nullptr;
  int32_t *dep_off = nullptr, *dep_idx = nullptr;  // subcycle dependencies (TilePlan)
  unsigned *epoch = nullptr;     // per-tile counters of a multi-subcycle launch
  int32_t *tile_meta = nullptr;  // 8 int32 per tile (see TmaArgs)
  int32_t *tile_rec = nullptr;   // kRecInts int32 per tile (producer records)
  double *cblk = nullptr;        // per-call constants, kConstFields x 256 per tile
  int *err = nullptr;        // device error word of the bounded waits
  // device word of launch_const_blocks' field checks: 0 when every Tbu of the
  // call is +0 and every uinit, vinit finite (TmaArgs::compact)
  int *cflags = nullptr;
  bool compact_allowed = true;  // EVP1D_COMPACT=0 at init turns the short part off
  int nctas = 0;             // SM count of the device
  uint8_t *flags = nullptr;
  double *geo[kNumGeo] = {};
  double *dyn[kNumDyn] = {};
  double *stress[2][12] = {};
  double *u[2] = {}, *v[2] = {};
  double *strintx = nullptr, *strinty = nullptr, *Cb = nullptr;
  double *str[8] = {};
  double *stage = nullptr;  // reference-order staging, 32 x navel doubles
  int cur = 0;              // buffer holding the current state
  // resident plan (evp_resident.h), res_blocks == 0: none
  int res_blocks = 0, res_threads = 0, res_cls = 0;
  bool res_quad = false;
  int32_t *res_slot = nullptr, *res_cnt = nullptr, *res_corner = nullptr;
  uint32_t *res_str = nullptr;
  double4 *res_mail = nullptr;  // 2 x nslots velocity mailboxes
  unsigned res_seq = 1;         // number of the next launch's first subcycle
};

// Allocate and fill the static part from a tile plan and reference-order
// geometry (host).  Creates the stream.
int problem_create(DeviceProblem *d, int device, const TilePlan &plan,
                   const ResidentPlan &res, const double *const geo[kNumGeo]);
void problem_destroy(DeviceProblem *d);

// The host arrays of one call.  Per-point fields have n_f elements, point p
// at map_f[p] (null: at p); u and v have n_uv, at map_uv[p] (null: as the
// fields; halo slots at their own index).  `stage` is device staging for
// arrays the GPU cannot address, stage_step doubles apart: 0..11 the inputs,
// 12..23 the stresses, strintx, strinty, Cb, u, v, uinit, vinit; istage has
// room for the two skip arrays.
struct UploadFields {
  const double *in[12] = {}, *stress[12] = {};
  const double *u = nullptr, *v = nullptr, *uinit = nullptr, *vinit = nullptr;
  const double *strintx = nullptr, *strinty = nullptr, *Cb = nullptr;
  const int32_t *skT = nullptr, *skU = nullptr;
  bool mask = false;       // skT, skU are ice masks (nonzero: not skipped)
  bool zero_halo = false;  // halo velocities are 0, not read
  size_t n_f = 0, n_uv = 0;
  const int32_t *map_f = nullptr, *map_uv = nullptr;  // device
  double *stage = nullptr;
  size_t stage_step = 0;
  int32_t *istage = nullptr;
};
// Where one call's results go (null: not wanted); u and v: n_u elements where
// the array is staged (the list points come first there), str: n_str.
struct DownloadFields {
  double *stress[12] = {}, *u = nullptr, *v = nullptr, *strintx = nullptr, *strinty = nullptr;
  double *Cb = nullptr, *str[8] = {};
  size_t n_f = 0, n_u = 0, n_str = 0;
  const int32_t *map_f = nullptr, *map_uv = nullptr;
  double *stage = nullptr;
  size_t stage_step = 0;
};
// n slot-ordered arrays to the caller's host arrays (na points each, reference
// order); waits for the stream.
int problem_gather_to_host(DeviceProblem *d, int n, const double *const *src,
                           double *const *host);
// Page-locked memory shared by the handles of the process, allocated once
// their calls have made enough copies without it and freed with the last
// handle: a page of words, one per handle, and one staging buffer of
// kPinnedStage bytes that a call borrows.  All are safe from several threads.
void pinned_hold(DeviceProblem *d);  // takes a reference
void pinned_release(DeviceProblem *d);
int *pinned_word(DeviceProblem *d);  // the handle's word; null: none (yet)
// Whether the GPU can address the `bytes` bytes of host memory at p
// (page-locked or managed, the whole range, `align`ed); *dev: at which address.
bool device_view(const void *p, size_t bytes, size_t align, void **dev);
// Fields host -> device: state in both sets, slot-ordered inputs, drag factor
// (aiu*rhow)*Cw, constant blocks; str zeroed; uvel_init/vvel_init default to
// the velocities; cur = 0.  With `wait` the arrays may be changed afterwards.
int problem_upload(DeviceProblem *d, const UploadFields &f, double rhow, bool wait);
// Results device -> host; waits for the stream.  *code: the error word of the
// bounded waits, cleared; if it is set, no result has been written.
int problem_download(DeviceProblem *d, const DownloadFields &f, int *code);
// Rebuild the per-tile constant blocks from the slot arrays (after the
// per-call fields or the drag factor changed), with the field checks in
// cflags.
int problem_fill_const(DeviceProblem *d);

// Views for the kernels.
DevState problem_inplace_view(const DeviceProblem &d);
FusedArgs problem_fused_args(const DeviceProblem &d, int from);
TmaArgs problem_tma_args(const DeviceProblem &d, int from);
// One resident launch of nsub subcycles from the state (u_in, v_in, s_in) to
// s_out and, uv_step == 0, (u_out, v_out); see ResidentArgs.  Takes nsub
// mailbox numbers (a refused launch too, which changes nothing else).
cudaError_t problem_launch_resident(DeviceProblem *d, const Params &p, int nsub, bool last,
                                    double *const s_in[12], double *const s_out[12],
                                    const double *u_in, const double *v_in, double *u_out,
                                    double *v_out, size_t uv_step);
// Read and clear the device error word (0 if no bounded wait ran out).
int problem_take_error(DeviceProblem *d, int *code);

}  // namespace evp
