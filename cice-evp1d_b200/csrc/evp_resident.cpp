// evp_resident.cpp -- plan of the resident solver (evp_resident.h).
//
// Points are ordered in strips about as wide as a block is high (the block
// that results is close to a square, which keeps its halo short: a block of
// o points recomputes about 2*sqrt(o)), and cut in that order into blocks of
// the longest prefix whose compute set fits.  Within a block the points whose
// stress reads only the block's own velocities come first, so that the warps
// that wait for another block's velocities are few and run last.
#include "evp_resident.h"

#include <algorithm>
#include <cmath>
#include <cstdio>

namespace evp {

namespace {

struct Cut {
  int w = 0;                   // strip width of `order`
  std::vector<int32_t> order;  // list points, block after block
  std::vector<int32_t> off;    // [nblocks + 1]
};

// Blocks of at most `threads` compute positions and `owned` owned points, or
// nothing once more than `max_blocks` are needed.
bool cut_blocks(int na, const int32_t *const nb0[6], const TilePlan &T, int threads, int owned,
                int max_blocks, Cut *cut) {
  const int w = std::max(4, std::min(63, (int)std::lround(std::sqrt((double)threads))));
  if (cut->w != w) {
    cut->w = w;
    std::vector<std::pair<uint64_t, int32_t>> key((size_t)na);
    for (int p = 0; p < na; p++) {
      const uint64_t i = (uint64_t)T.ci[p], j = (uint64_t)T.cj[p];
      key[p] = {((uint64_t)T.piece[p] << 40) | ((i / w) << 23) | (j << 6) | (i % w), p};
    }
    std::sort(key.begin(), key.end());
    cut->order.resize((size_t)na);
    for (int p = 0; p < na; p++) cut->order[p] = key[p].second;
  }
  cut->off.assign(1, 0);
  std::vector<int32_t> own((size_t)na, -1), halo((size_t)na, -1);
  for (int k = 0; k < na;) {
    const int b = (int)cut->off.size() - 1;
    if (b == max_blocks) return false;
    int nh = 0, best = 1, len = 0;
    while (k + len < na && len < owned && len + nh <= threads + 32) {
      const int p = cut->order[k + len++];
      own[p] = b;
      if (halo[p] == b) nh--;
      for (int r = 3; r < 6; r++) {
        const int q = nb0[r][p];
        if (q < na && own[q] != b && halo[q] != b) {
          halo[q] = b;
          nh++;
        }
      }
      // not monotone: a point can join that was a halo point
      if (len + nh <= threads) best = len;
    }
    for (int q = best; q < len; q++) own[cut->order[k + q]] = -1;
    k += best;
    cut->off.push_back(k);
  }
  return true;
}

// Whether nw of ee, sw of ne, sse of se and back return to the point wherever
// both ends are list points; *first: a point where they do not.  Then the
// blocks that read a corner velocity of a T point are those that own one of
// its corners, and every one of them computes the point: a point that is not
// skipped makes all of them wait for one another, a skipped one none, so
// waiting is mutual under every mask.  (Symmetry between blocks over all
// points is not enough: a mask can leave only one side's points.)
bool inverse_relations(int na, const int32_t *const nb0[6], int *first) {
  for (int r = 0; r < 6; r++)
    for (int p = 0; p < na; p++) {
      const int q = nb0[r][p];
      if (q < na && nb0[(r + 3) % 6][q] != p) {
        *first = p;
        return false;
      }
    }
  return true;
}

}  // namespace

bool build_resident_plan(int na, const int32_t *const nb0[6], const TilePlan &T, int max_blocks,
                         ResidentPlan *plan, bool quad) {
  ResidentPlan &R = *plan;
  R = ResidentPlan();
  // 17 bits of strip, row and piece in the sort key
  int one_way;
  if (na <= 0 || !T.from_coords || max_blocks < 1 || na > (1 << 17) ||
      !inverse_relations(na, nb0, &one_way))
    return false;
  const double o = std::ceil((double)na / max_blocks);
  const double least = o + 1.8 * std::sqrt(o);
  Cut cut;
  int threads = std::max((int)std::ceil(least / 8.0) * 8, kQuadMinWidth);
  for (; quad && threads <= kQuadMaxWidth; threads += 8)
    if (cut_blocks(na, nb0, T, threads, threads, max_blocks, &cut)) break;
  R.quad = quad && threads <= kQuadMaxWidth;
  if (!R.quad) {
    threads = std::max((int)std::ceil(least / 32.0) * 32, kResMinWidth);
    for (;; threads += 32) {
      if (threads > kResMaxWidth) return false;
      // wider than a CTA: a second stepu pass only where it cannot be avoided
      if (threads > kResMaxThreads &&
          cut_blocks(na, nb0, T, threads, kResMaxThreads, max_blocks, &cut))
        break;
      if (cut_blocks(na, nb0, T, threads, threads, max_blocks, &cut)) break;
    }
  }
  const int nb = (int)cut.off.size() - 1;
  R.nblocks = nb;
  R.threads = threads;
  for (int c : kResWidths)
    if (c >= threads) {
      R.cls = c;
      break;
    }
  std::vector<int32_t> owner((size_t)na);
  for (int b = 0; b < nb; b++)
    for (int k = cut.off[b]; k < cut.off[b + 1]; k++) owner[cut.order[k]] = b;
  const size_t N = (size_t)nb * threads;
  R.cnt.resize(nb);
  R.slot.assign(N, -1);
  R.corner.assign(4 * N, 0);
  R.str.assign(N, 0);
  std::vector<char> exported((size_t)na, 0);
  std::vector<int32_t> pos((size_t)na, -1);       // position in the point's own block
  std::vector<int32_t> hpos((size_t)na, -1), hblk((size_t)na, -1);
  std::vector<std::vector<int32_t>> members((size_t)nb);
  for (int b = 0; b < nb; b++) {
    auto reads_other = [&](int p) {
      for (int r = 0; r < 3; r++)
        if (nb0[r][p] < na && owner[nb0[r][p]] != b) return true;
      return false;
    };
    std::vector<int32_t> &m = members[b];
    m.assign(cut.order.begin() + cut.off[b], cut.order.begin() + cut.off[b + 1]);
    std::stable_partition(m.begin(), m.end(), [&](int p) { return !reads_other(p); });
    R.cnt[b] = (int32_t)m.size();
    for (size_t k = 0; k < m.size(); k++) pos[m[k]] = (int32_t)k;
  }
  for (int b = 0; b < nb; b++) {
    const size_t base = (size_t)b * threads;
    std::vector<int32_t> m = members[b];
    const int cnt = R.cnt[b];
    for (int k = 0; k < cnt; k++) {
      uint32_t packed = 0;
      for (int r = 3; r < 6; r++) {
        const int q = nb0[r][m[k]];
        uint32_t at = (uint32_t)R.cls;
        if (q < na && owner[q] == b) {
          at = (uint32_t)pos[q];
        } else if (q < na) {
          if (hblk[q] != b) {
            hblk[q] = b;
            hpos[q] = (int32_t)m.size();
            m.push_back(q);
          }
          at = (uint32_t)hpos[q];
        }
        packed |= at << (10 * (r - 3));
      }
      R.str[base + k] = packed;
    }
    for (size_t k = 0; k < m.size(); k++) {
      R.slot[base + k] = T.slot_of_point[m[k]];
      for (int r = 0; r < 4; r++) {
        const int q = r == 0 ? m[k] : nb0[r - 1][m[k]];
        int32_t at;
        if (q >= na) {
          at = ~(T.nslots + (q - na));
        } else if (owner[q] == b) {
          at = pos[q];
        } else {
          at = ~T.slot_of_point[q];
          exported[q] = 1;
        }
        R.corner[4 * (base + k) + r] = at;
      }
    }
  }
  for (int p = 0; p < na; p++)
    if (exported[p]) R.str[(size_t)owner[p] * threads + pos[p]] |= kResExport;
  return true;
}

long long verify_resident_plan(const ResidentPlan &R, int na, const int32_t *const nb0[6],
                               const TilePlan &T, std::string *first) {
  long long bad = 0;
  auto wrong = [&](const char *what, int b, int k) {
    if (bad++ == 0 && first) {
      char buf[128];
      snprintf(buf, sizeof buf, "resident block %d position %d: %s", b, k, what);
      *first = buf;
    }
  };
  const int M = R.threads;
  const size_t N = (size_t)R.nblocks * M;
  if (M % (R.quad ? 8 : 32) || (R.quad && M > kQuadMaxWidth) || M > R.cls ||
      R.cls > kResMaxWidth || R.slot.size() != N || R.str.size() != N ||
      R.corner.size() != 4 * N || R.cnt.size() != (size_t)R.nblocks) {
    wrong("sizes", -1, -1);
    return bad;
  }
  auto point = [&](int32_t s) { return s >= 0 && s < T.nslots ? T.point_of_slot[s] : -1; };
  std::vector<int32_t> owner((size_t)na, -1);
  std::vector<char> exported((size_t)na, 0), wanted((size_t)na, 0);
  for (int b = 0; b < R.nblocks; b++)
    for (int k = 0; k < M; k++) {
      const int32_t s = R.slot[(size_t)b * M + k];
      if (s == -1 && k >= R.cnt[b]) continue;
      const int p = point(s);
      if (p < 0) {
        wrong("not a point's slot", b, k);
      } else if (k < R.cnt[b]) {
        if (owner[p] != -1) wrong("owned twice", b, k);
        owner[p] = b;
        if (R.str[(size_t)b * M + k] & kResExport) exported[p] = 1;
      }
    }
  if (bad) return bad;
  std::vector<uint64_t> pairs;
  for (int b = 0; b < R.nblocks; b++)
    for (int k = 0; k < M; k++) {
      const size_t at = (size_t)b * M + k;
      const int p = point(R.slot[at]);
      if (p < 0) continue;
      for (int r = 0; r < 4; r++) {
        const int q = r == 0 ? p : nb0[r - 1][p];
        const int32_t c = R.corner[4 * at + r];
        if (c >= 0) {
          if (c >= R.cnt[b] || q >= na || point(R.slot[(size_t)b * M + c]) != q)
            wrong("own velocity position", b, k);
        } else if (q >= na) {
          if (~c != T.nslots + (q - na)) wrong("halo velocity slot", b, k);
        } else {
          if (point(~c) != q || owner[q] == b) wrong("polled velocity slot", b, k);
          wanted[q] = 1;
          pairs.push_back((uint64_t)b << 32 | (uint32_t)owner[q]);
        }
      }
      if (k >= R.cnt[b]) continue;
      for (int r = 3; r < 6; r++) {
        const int q = nb0[r][p];
        const int x = (int)(R.str[at] >> (10 * (r - 3))) & 1023;
        if (q >= na ? x != R.cls : (x >= M || point(R.slot[(size_t)b * M + x]) != q))
          wrong("str position", b, k);
      }
    }
  for (int p = 0; p < na; p++) {
    if (owner[p] < 0) wrong("a point no block owns", -1, p);
    if (exported[p] != wanted[p]) wrong("export mark", owner[p], p);
  }
  int one_way;
  if (!inverse_relations(na, nb0, &one_way))
    wrong("neighbour relations that are not each other's inverse", -1, one_way);
  std::sort(pairs.begin(), pairs.end());
  for (uint64_t x : pairs)
    if (!std::binary_search(pairs.begin(), pairs.end(), (x & 0xffffffffu) << 32 | x >> 32))
      wrong("a block reads from one that does not read from it", (int)(x >> 32), -1);
  return bad;
}

}  // namespace evp
