// resident_plan_shim.cpp -- test helper (host only): builds the tile plan and
// the resident plan of a problem (csrc/evp_tiles.cpp, evp_resident.cpp) and
// runs the resident plan's verifier, optionally after planting a mistake.
#include <cstdint>
#include <string>

#include "evp_resident.h"

extern "C" {

// 0-based neighbour vectors ee, ne, se, nw, sw, sse, back to back ([6 * na]).
// Returns the number of violations (-1: the problem has no resident plan);
// stats: blocks, threads per block, width class, largest compute set, halo
// points, exported points.
long long resident_plan(int na, int navel, const int32_t *nb, int max_blocks, int plant,
                        long long stats[6]) {
  const int32_t *nbp[6];
  for (int k = 0; k < 6; k++) nbp[k] = nb + (size_t)k * na;
  evp::TilePlan T;
  evp::build_tile_plan(na, navel, nbp, nullptr, nullptr, &T);
  evp::ResidentPlan R;
  if (!evp::build_resident_plan(na, nbp, T, max_blocks, &R)) return -1;
  long long most = 0, halo = 0, exported = 0;
  for (int b = 0; b < R.nblocks; b++) {
    int n = 0;
    for (int k = 0; k < R.threads; k++) {
      const size_t at = (size_t)b * R.threads + k;
      if (R.slot[at] < 0) continue;
      n++;
      if (k >= R.cnt[b]) halo++;
      if (R.str[at] & evp::kResExport) exported++;
    }
    if (n > most) most = n;
  }
  const long long st[6] = {R.nblocks, R.threads, R.cls, most, halo, exported};
  for (int k = 0; k < 6; k++) stats[k] = st[k];
  const size_t mid = (size_t)(R.nblocks / 2) * R.threads;
  if (plant == 1) R.corner[4 * mid + 1] += 1;
  if (plant == 2) R.str[mid] ^= 1u;
  if (plant == 3) R.slot[mid] = R.slot[mid + 1];
  if (plant == 4) R.str[mid + R.cnt[R.nblocks / 2] - 1] ^= evp::kResExport;
  if (plant == 5) R.cnt[R.nblocks / 2] -= 1;
  std::string first;
  return evp::verify_resident_plan(R, na, nbp, T, &first);
}
}
