// cuts3d.h -- how the fused 3D half steps (sweep3d.cu) cut their tiles in z.
#pragma once
#include <algorithm>
#include <functional>
#include <queue>
#include <vector>

namespace fomo {

constexpr int kMaxGrid3 = 1184;  // most persistent CTAs of a half step

// Segments that the list of a grid of ntiles tiles has room for.
constexpr long long segs3_room(long long ntiles) { return ntiles + 4LL * kMaxGrid3; }

// The last `tiles` tiles are cut in `chunks` (chunk-major), the ones before them are whole
// z columns.
struct Cuts3 {
  int tiles, chunks;
};

// Planes until the last of G CTAs is done that take the segments of a cut in order, each
// worth its planes and the two it takes to fill its pipeline.
inline long long span3(const Cuts3& c, int ntiles, int nz, int G) {
  std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free_at;
  for (int k = 0; k < G; ++k) free_at.push(0);
  long long end = 0;
  auto take = [&](int planes) {
    const long long t = free_at.top() + planes + 2;
    free_at.pop();
    free_at.push(t);
    end = std::max(end, t);
  };
  for (int k = c.tiles; k < ntiles; ++k) take(nz);
  for (int k = 0; k < c.chunks; ++k)
    for (int t = 0; t < c.tiles; ++t)
      take((int)((long long)nz * (k + 1) / c.chunks - (long long)nz * k / c.chunks));
  return end;
}

// ntiles tiles of nz planes for G persistent CTAs on nsm SMs.
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
// Ten chunks lose where they are one round of the CTAs more than the four would be, or only
// more pipelines to fill, so they also have to end sooner by span3.  That holds
// for elastic steps (a CTA per SM); two acoustic CTAs share an SM's rate, so there it says
// something only where the four chunks leave an SM to every CTA.
//   elastic 108x108x68 (32 tiles) 92 -> 98, order 6 118x115x77 (36) 85 -> 101, 72x154x99 (33)
//   134 -> 141, order 2 217x250x147 (144) 358 -> 375, but 147x42x94 (15) 112 -> 98;
//   acoustic 48x48x72 (8 tiles) 73 -> 76, order 4 194x70x64 (35) 58 -> 64, order 10 50x33x76 (6)
//   67 -> 73, but 48x115x58 (18) 162 -> 70, 45x183x80 (28) 74 -> 67.
// Of 332 listed and random grids none is more than 1.3 % slower by this choice than with the
// last wave in four; it passes by 26 gains of over 2 %, the largest 23 %.  Of 216 random grids
// that the rule was not made on none is more than 0.5 % slower (geometric mean 1.31 times faster).
inline Cuts3 cuts3(bool elastic, int ntiles, int nz, int G, int nsm) {
  const long long nt = ntiles;
  const Cuts3 last{std::min({ntiles, G, kMaxGrid3}), nz >= 64 ? 4 : 1};
  const Cuts3 ten{ntiles, std::min(10, nz / 5)};
  const bool few = elastic ? 2 * nt <= G : 10 * nt <= 7LL * G;
  const bool tall = nz >= 120 && (!elastic || 8 * nt <= 9LL * G);
  if (ten.chunks <= 1 || !(few || tall) || ten.chunks * nt > segs3_room(nt)) return last;
  const bool alone = elastic || 4 * nt <= nsm;
  return !alone || span3(ten, ntiles, nz, G) < span3(last, ntiles, nz, G) ? ten : last;
}

}  // namespace fomo
