// evp_resident.h -- host-side plan of the resident solver (internal).
//
// Where a problem fits the SMs' registers and shared memory (up to about 98k
// points on 148), a call's subcycles run in one launch whose CTAs keep their
// points on chip from the first subcycle to the last
// (evp_kernels_resident.cu).  The list is cut into
// blocks, one per CTA.  A block owns its points and recomputes `stress` at
// its forward halo, the nw/sw/sse neighbours other blocks own, so that only
// velocities travel between blocks: those of points that another block's
// stress reads ("exported" points).
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "evp_tiles.h"

namespace evp {

// Widths the kernel is compiled for: a block's compute set (owned points, then
// forward halo) has at most that many positions.  Up to kResMaxThreads a thread
// each; of a wider block the positions beyond take four lanes each
// (k_resident), as far as shared memory holds their constants.
constexpr int kResMaxThreads = 512;
constexpr int kResWidths[] = {128, 256, 384, kResMaxThreads, 736};
constexpr int kResMaxWidth = 736;
constexpr int kResMinWidth = 128;  // four warps, one per scheduler
// Small problems take four lanes per point (k_resident_quad), in blocks of up to
// kQuadMaxWidth points: below that one thread per point leaves an SM's
// schedulers a warp each, whose 2300 cycles of stress are instruction latency.
constexpr int kQuadMinWidth = 32, kQuadMaxWidth = 128;
// ResidentPlan::str bits
constexpr uint32_t kResExport = 1u << 30;

struct ResidentPlan {
  int nblocks = 0;
  int threads = 0;  // per block: compute positions (a multiple of 32; quad: of 8)
  bool quad = false;  // four lanes per compute position
  int cls = 0;      // the kResWidths entry the kernel runs at
  std::vector<int32_t> cnt;   // [nblocks] owned points; positions below cnt are owned
  // [nblocks * threads]: device slot of each position, -1 for none
  std::vector<int32_t> slot;
  // [nblocks * threads * 4]: where a position's stress reads the velocities of
  // cc, ee, ne, se: >= 0 an owned position of the block; < 0 the u/v slot ~x:
  // another block's point (~x < nslots), or one of the reference's halo slots,
  // whose velocities stay as given
  std::vector<int32_t> corner;
  // [nblocks * threads] owned positions: str positions of nw, sw, sse (10 bits
  // each; `cls` = the zero slot) and kResExport
  std::vector<uint32_t> str;
};

// Plan for at most `max_blocks` CTAs from the problem's tile plan (its slots
// and rebuilt coordinates) and 0-based neighbour vectors.  False where the
// problem does not fit the widest blocks, has no grid layout, or where its
// neighbour relations are not each other's inverse (ee and nw, ne and sw, se
// and sse; grids' are): the kernels' two-deep mailboxes and their results in
// place need every wait to be mutual, whichever points a call skips.
// `quad`: blocks for four lanes per point where the problem is small enough.
bool build_resident_plan(int na, const int32_t *const nb0[6], const TilePlan &tiles,
                         int max_blocks, ResidentPlan *plan, bool quad = true);

// Decode every index of `plan` and compare it with the neighbour vectors.
// Returns the number of violations; *first (if not null) describes the first.
long long verify_resident_plan(const ResidentPlan &plan, int na, const int32_t *const nb0[6],
                               const TilePlan &tiles, std::string *first);

}  // namespace evp
