// cuts3d.h -- how the fused 3D half steps (sweep3d.cu) cut their tiles in z.
#pragma once
#include <algorithm>

namespace fomo {

constexpr int kMaxGrid3 = 1184;  // most persistent CTAs of a half step

// Segments that the list of a grid of ntiles tiles has room for.
constexpr long long segs3_room(long long ntiles) { return ntiles + 4LL * kMaxGrid3; }

// The last `tiles` tiles are cut in `chunks` (chunk-major), the ones before them are whole
// z columns.
struct Cuts3 {
  int tiles, chunks;
};

// ntiles tiles of nz planes for G persistent CTAs.
// Every tile is cut into ten z chunks where that gives idle CTAs work or evens
// out the last wave: up to 0.7 acoustic or 0.5 elastic tiles per CTA, and if a chunk has 12
// planes (its pipeline has to fill) up to 9/8 elastic tiles per CTA and as many acoustic
// ones as the list has room for (526).  Otherwise the tiles are whole columns and only the
// last wave is cut, in four.
// us per step, last wave in four -> all in ten (layers included, order 8):
//   acoustic 249x238x209 (153 tiles) 461 -> 404, 128x118x138 157 -> 113,
//   328x328x268 (264) 790 -> 743, 388x388x288 (364) 1184 -> 1041, but in shorter chunks
//   548x328x108 (456) 498 -> 528, 428x418x38 (420) 193 -> 213;
//   elastic 148x148x128 (55 tiles) 253 -> 216, 249x238x209 (153) 828 -> 793, but 348x168x38
//   (144) 151 -> 174, order 10 310x270x250 (220) 1296 -> 1298, 368x368x268 (351) 1849 -> 1899.
inline Cuts3 cuts3(bool elastic, int ntiles, int nz, int G) {
  const long long nt = ntiles, room = segs3_room(nt);
  const int n = std::min(10, nz / 5);
  const bool few = elastic ? 2 * nt <= G : 10 * nt <= 7LL * G;
  const bool tall = nz >= 120 && (!elastic || 8 * nt <= 9LL * G);
  if (n > 1 && (few || tall) && n * nt <= room) return {ntiles, n};
  return {std::min({ntiles, G, kMaxGrid3}), nz >= 64 ? 4 : 1};
}

}  // namespace fomo
