// resident2d.cuh -- 2D time loops whose state stays on the chip.
//
// Small and mid-size 2D runs (up to about 1 M shot-cells) are bound by launch
// latency in the two-phase form: a step is one or two dependent launches whose
// cells fill the chip for a few microseconds.  Here one cooperative launch runs
// many steps.  Every CTA (one per SM) owns a tile of one shot's padded grid and
// keeps the tile's wavefields, with a halo, and materials in shared memory for
// the whole launch; only halo cells travel between CTAs.
//
// Halo exchange.  After a half step each CTA publishes the cells its
// neighbours read as 8-byte words {value, epoch} in its part of a buffer in global
// memory, and reads its own halo from its neighbours' parts, polling each word until it
// carries the epoch of the half step.  A word is one 64-bit access, so value and flag
// arrive together: no fence, no separate flag, one L2 round trip per exchange.
// The buffer is double-buffered by step parity: a tile overwrites the words of
// step k at step k + 2, after it has read its neighbours' words of step k + 1,
// which they publish only once they have read step k.  Neighbours are mutual:
// tiles are at least N + 1 cells wide and high.  Every poll is bounded (about a
// second on the global timer, recorded in *err); after that the tile stops waiting,
// and the host runs the steps again as launches, which wait for nobody.
//
// What it measured (us per step, order 8, nbc 50 where none is given, this form / replayed
// two-phase launches, in blocks per thread from 200 k inner cells):
// acoustic 240x200 4.5 / 8.0, 400x300 nbc 100 6.0 / 12.3, 4 shots of 240x200 7.6 / 14.2,
// eight 13.2 / 18.7, 1000x800 12.6 / 14.1 (materials from L2); elastic 240x200 6.3 / 9.4,
// 501x397 10.4 / 16.1, 640x560 nbc 20 12.5 / 14.0; scalar 240x200 2.1 / 3.6, 500x400 2.7 / 5.1,
// 1000x800 5.5 / 6.1; coupled 400x300 nbc 100 10.2 / 13.4.  It is the faster form up to the
// largest grids that fit, at order 10 too.  With the updates taken out, the exchange and the
// barriers alone take 1.3 of the 2.1 us of a scalar step and, for its two exchanges, 2.6 of
// the 4.5 us of an acoustic step (240x200; 4.1 of 12.6 at 1000x800).  The rest is issue and
// latency of the phases between barriers: 46 to 49 % of the issue slots are used, at 20
// warps per SM (30 for scalar 240x200), by more integer than floating point instructions.
//
// A tile computes its own cells and a one-cell ring around them (the inward
// neighbours of the Higdon terms), so the ring's old values come with the halo and the
// pre-correction neighbours never travel.  Threads own blocks of CX x R cells: the x window
// comes as words of CX floats, the z window lives in registers.  The per-cell arithmetic
// is the two-phase kernels' sequence, so results are equal bit for bit.
#pragma once
#include <stdint.h>

#include <algorithm>

#include "solver2d_kernels.cuh"
#include "tma.cuh"

namespace fomo {
namespace res {

// Blocks of cells per thread (columns x rows) and the most threads of a CTA (one CTA
// per SM): the smallest block that covers the tile runs the step, since few warps
// with long blocks leave the phases between two barriers bound by latency (acoustic
// 240x200, nbc 50, us per step: 1 x 1 4.61, 4 x 1 4.61, 4 x 2 5.08, 4 x 4 7.10; 400x300, nbc
// 100: 4 x 1 6.19, 4 x 2 6.60, 4 x 4 7.91).
struct Form {
  int CX, R, threads;
};
constexpr Form kForms[] = {{1, 1, 1024}, {4, 1, 640}, {4, 2, 512}, {4, 4, 512}};
constexpr int kNumForms = 4;
constexpr int kSmallBlock = 4;  // cells of blocks that always have their materials on the chip

// Decomposition and shared-memory geometry of one run (the same for every tile;
// tiles differ by at most one column or row).
struct Geom {
  int nx, nz, ld;      // padded grid, row pitch
  long long plane;
  int M, nbc;          // fd_order / 2, Higdon zone
  int gx, gz;          // tiles per shot
  int nq, ngr;         // quads of columns per extended row, groups of R extended rows
  int nb;              // blocks per extended row
  int pitch, rows;     // haloed arrays (floats per row, rows)
  int words;           // start of the word tables in shared memory (floats)
  int per;             // words a tile publishes per half step, at most
  int gmat;            // materials are read from global memory (they do not fit on the chip)
};

// First column / row of tile i of `parts`.  Tiles start one column past a multiple
// of four, so a tile's quads (which begin with the ring column left of it) are
// aligned in the grid: one extra quad per row holds both ring columns, and a
// quad's words in global memory move as vectors.
__host__ __device__ inline int tile_x(int n, int parts, int i) {
  if (i <= 0) return 0;
  if (i >= parts) return n;
  return 1 + 4 * (int)((long long)((n + 2) / 4) * i / parts);
}
__host__ __device__ inline int tile_z(int n, int parts, int i) {
  return (int)((long long)n * i / parts);
}

// Source / receiver cells of a tile, sorted by the thread that owns them.
struct Entries {
  const int* off;   // [tiles + 1]
  const int2* key;  // {thread, cell k * CX + j of the thread's block}
  const int* ent;   // index into the run's CellTags entries
  CellTags tags;    // tag unused
};

struct Tile {
  int shot, x0, z0, TW, TH;
  int off;          // columns of the first quad left of the tile (the ring column, or 0)
  int q, gr;        // this thread's block column and row group
  int e0, e1;       // this thread's entries
  bool act;         // the thread owns a block
};

template <int N>
struct Shape {
  static constexpr int H = N + 1;             // halo width
  static constexpr int L = (N + 3) & ~3;      // columns left of the extended row (multiple of 4)
};

__device__ __forceinline__ Tile tile_of(const Geom& g, const Entries& E) {
  Tile t;
  const int per = g.gx * g.gz;
  t.shot = blockIdx.x / per;
  const int b = blockIdx.x - t.shot * per, tz = b / g.gx, tx = b - tz * g.gx;
  t.x0 = tile_x(g.nx, g.gx, tx);
  t.TW = tile_x(g.nx, g.gx, tx + 1) - t.x0;
  t.z0 = tile_z(g.nz, g.gz, tz);
  t.TH = tile_z(g.nz, g.gz, tz + 1) - t.z0;
  t.off = t.x0 > 0 ? 1 : 0;
  t.gr = threadIdx.x / g.nb;
  t.q = threadIdx.x - t.gr * g.nb;
  t.act = t.gr < g.ngr;
  // this thread's range of the tile's entries (sorted by thread)
  int lo = E.off[blockIdx.x], hi = E.off[blockIdx.x + 1];
  const int end = hi;
  while (lo < hi) {
    const int m = (lo + hi) >> 1;
    if (E.key[m].x < (int)threadIdx.x) lo = m + 1;
    else hi = m;
  }
  t.e0 = t.e1 = lo;
  while (t.e1 < end && E.key[t.e1].x == (int)threadIdx.x) ++t.e1;
  return t;
}

__device__ __forceinline__ void ll_put(uint64_t* p, float v, uint32_t epoch) {
  const uint64_t w = ((uint64_t)epoch << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ uint64_t ll_get(const uint64_t* p) {
  uint64_t w;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}

// The words a tile publishes lie one after another in its own part of the plane
// set, in the order of its put table, so puts and gets move whole sectors.
// A word that a tile reads: its place there (-1: outside the grid) and in shared memory.
struct Word {
  int g, s;
};
// Publishes the words of a table (shared-memory places) at ll.  The tables are built
// once per launch: the region arithmetic in the step loop cost as many instructions
// as the stencils.
__device__ __forceinline__ void words_put(const int* tab, int n, uint64_t* ll, const float* sm,
                                          uint32_t epoch) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) ll_put(ll + i, sm[tab[i]], epoch);
}
// K words per thread are polled together: a round trip covers all that are still missing.
template <int K>
__device__ __forceinline__ void words_get(const Word* tab, int n, const uint64_t* ll, float* sm,
                                          uint32_t epoch, bool& live, int* err) {
  for (int base = threadIdx.x; base < n; base += K * blockDim.x) {
    Word e[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      e[k].g = -1;
      if (base + k * blockDim.x < n) e[k] = tab[base + k * blockDim.x];
    }
    uint64_t t0 = 0;
    bool any = true;
    for (int spin = 1; any; ++spin) {
      uint64_t w[K];
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (e[k].g >= 0) w[k] = ll_get(ll + e[k].g);
      any = false;
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (e[k].g >= 0) {
          if ((uint32_t)(w[k] >> 32) == epoch || !live) {
            sm[e[k].s] = __uint_as_float((uint32_t)w[k]);
            e[k].g = -1;
          } else {
            any = true;
          }
        }
      if ((spin & 1023) == 0) {
        const uint64_t t = tma::global_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > 1000000000ull) {
          atomicOr(err, 8);
          live = false;
        }
      }
    }
  }
}

// A region of one field's halo.  strip: lo columns left and hi right of the tile, rows
// -1 .. TH.  band: lo rows above and hi below, columns -1 .. TW.  rows / cols: the ring
// rows above and below, the ring columns left and right.
enum RegionKind { kStrip, kBand, kRows, kCols };
struct Region {
  int kind, lo, hi, field;
};

// CX consecutive floats, loaded and stored as one word.
template <int CX>
struct Vec {
  float v[CX];
  __device__ __forceinline__ float operator[](int j) const { return v[j]; }
};
template <int CX>
__device__ __forceinline__ Vec<CX> ldv(const float* p) {
  Vec<CX> r;
  if constexpr (CX == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    r.v[0] = q.x;
    r.v[1] = q.y;
    r.v[2] = q.z;
    r.v[3] = q.w;
  } else {
    r.v[0] = *p;
  }
  return r;
}
template <int CX>
__device__ __forceinline__ void stv(float* p, const float (&u)[CX]) {
  if constexpr (CX == 4) *reinterpret_cast<float4*>(p) = make_float4(u[0], u[1], u[2], u[3]);
  else *p = u[0];
}

// The row window of a block at p: at least N columns on both sides, w[L + j] = cell j.
template <int N, int CX>
struct XWin {
  static constexpr int G = (N + CX - 1) / CX, L = G * CX;
  float w[2 * L + CX];
  __device__ __forceinline__ void load(const float* p) {
#pragma unroll
    for (int i = -G; i <= G; ++i) {
      const Vec<CX> v = ldv<CX>(p + i * CX);
#pragma unroll
      for (int j = 0; j < CX; ++j) w[L + i * CX + j] = v[j];
    }
  }
  // backward / forward staggered difference at cell j
  __device__ __forceinline__ float dm(int j, const Coef& c) const {
    float acc = 0.0f;
#pragma unroll
    for (int l = 1; l <= N; ++l)
      acc = __fmaf_rn(c.a[l - 1], __fsub_rn(w[L + j + l - 1], w[L + j - l]), acc);
    return acc;
  }
  __device__ __forceinline__ float dp(int j, const Coef& c) const {
    float acc = 0.0f;
#pragma unroll
    for (int l = 1; l <= N; ++l)
      acc = __fmaf_rn(c.a[l - 1], __fsub_rn(w[L + j + l], w[L + j - l + 1]), acc);
    return acc;
  }
};
// z differences of a register window w of rows, the cell's row at index o
template <int N, int CX, int NW>
__device__ __forceinline__ float zdm(const Vec<CX> (&w)[NW], int o, int j, const Coef& c) {
  float acc = 0.0f;
#pragma unroll
  for (int l = 1; l <= N; ++l)
    acc = __fmaf_rn(c.a[l - 1], __fsub_rn(w[o + l - 1][j], w[o - l][j]), acc);
  return acc;
}
template <int N, int CX, int NW>
__device__ __forceinline__ float zdp(const Vec<CX> (&w)[NW], int o, int j, const Coef& c) {
  float acc = 0.0f;
#pragma unroll
  for (int l = 1; l <= N; ++l)
    acc = __fmaf_rn(c.a[l - 1], __fsub_rn(w[o + l][j], w[o - l + 1][j]), acc);
  return acc;
}

// Column / row classification of the thread's block (kernels_fused.jl:28-52).
struct Class {
  unsigned own = 0;    // bit k * CX + j: a cell of the tile (not the ring)
  unsigned inner = 0;  // bit: inside the stencil's range
  unsigned frame = 0;  // bit: own Higdon cell
  int x, z;            // grid cell of (k, j) = (0, 0)
  // Values the step loop derives its tests and addresses from.  Without this the
  // compiler hoists every derived value out of the loop and spills them.
  __device__ __forceinline__ void refresh() {
    asm volatile("" : "+r"(own), "+r"(inner), "+r"(frame), "+r"(x), "+r"(z));
  }
  __device__ __forceinline__ int side(int p, int n, int nbc) const {
    return p <= nbc ? 1 : (p >= n - 1 - nbc ? -1 : 0);
  }
};
template <int CX, int R>
__device__ __forceinline__ Class classify(const Geom& g, const Tile& t, bool sponge) {
  Class b;
  b.x = t.x0 - t.off + CX * t.q;
  b.z = t.z0 + t.gr * R - 1;
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int j = 0; j < CX; ++j) {
      const int x = b.x + j, z = b.z + k, lx = CX * t.q + j - t.off, lz = t.gr * R + k - 1;
      const unsigned bit = 1u << (k * CX + j);
      const bool own = t.act && lx >= 0 && lx < t.TW && lz >= 0 && lz < t.TH;
      if (own) b.own |= bit;
      if (x >= g.M && x < g.nx - g.M && z >= g.M && z < g.nz - g.M) b.inner |= bit;
      if (!sponge && own && x >= 1 && x <= g.nx - 2 && z >= 1 && z <= g.nz - 2 &&
          (b.side(x, g.nx, g.nbc) != 0 || b.side(z, g.nz, g.nbc) != 0))
        b.frame |= bit;
    }
  return b;
}
// The run of one resident launch: geometry, steps and acquisition.
struct Run {
  Geom g;
  Coef c;
  float dtx, dtz;
  HabcDev h;
  Entries E;
  uint64_t* ll;        // [parity][half step][tiles][g.per]
  int it0, nsteps;     // first step (1-based), steps of this launch
  int snap_interval, pad, nxi, nzi;  // interior snapshots (0: none)
  float* snaps;
  int* err;
};

// Copies a tile of a grid plane into shared memory: element (r, col) is the cell
// (x0 + col - left, z0 + r - top), zero outside the grid or where src is null.
__device__ __forceinline__ void load_tile(const Geom& g, const Tile& t, const float* src, float* dst,
                                          int pitch, int rows, int left, int top) {
  for (int i = threadIdx.x; i < rows * pitch; i += blockDim.x) {
    const int r = i / pitch, col = i - r * pitch;
    const int x = t.x0 + col - left, z = t.z0 + r - top;
    dst[i] = (src && x >= 0 && x < g.nx && z >= 0 && z < g.nz) ? __ldg(src + (long long)z * g.ld + x)
                                                               : 0.0f;
  }
}

// A thread's view of its tile: where its block lies and the moves between
// registers, shared memory and the exchange planes that every solver shares.
// "Haloed" arrays hold the tile with N + 1 cells around it (pitch g.pitch), "extended"
// ones the tile and its ring (pitch 4 g.nq).
template <int N, int CX, int R>
struct Work {
  static constexpr int L = Shape<N>::L;
  static constexpr unsigned kRow = (1u << CX) - 1u;
  Tile t;
  Class cl;
  int hb, eb;       // the block in haloed / extended arrays
  int pitch, ep;
  bool live = true;

  __device__ __forceinline__ Work(const Run& run, bool sponge)
      : t(tile_of(run.g, run.E)), cl(classify<CX, R>(run.g, t, sponge)) {
    pitch = run.g.pitch;
    ep = 4 * run.g.nq;
    hb = (t.gr * R + N) * pitch + L + CX * t.q;
    eb = t.gr * R * ep + CX * t.q;
  }
  __device__ __forceinline__ void refresh() {
    cl.refresh();
    asm volatile("" : "+r"(hb), "+r"(eb));
  }
  __device__ __forceinline__ void load(const Run& run, float* A, const float* src) const {
    load_tile(run.g, t, src, A, pitch, run.g.rows, L + t.off, N + 1);
  }
  __device__ __forceinline__ void load_ext(const Run& run, float* A, const float* src) const {
    load_tile(run.g, t, src, A, ep, run.g.ngr * R, t.off, 1);
  }
  // Row k of the block in a material plane, from its extended array or, where the
  // materials stay off the chip, from L2 (a row outside the grid reads the nearest one: its
  // cells take no update).
  __device__ __forceinline__ Vec<CX> mat(const Run& run, const float* A, const float* plane,
                                         int k) const {
    if (CX * R <= kSmallBlock || !run.g.gmat) return ldv<CX>(A + eb + k * ep);
    const float* p = plane + (long long)min(max(cl.z + k, 0), run.g.nz - 1) * run.g.ld + cl.x;
    Vec<CX> r;
    if constexpr (CX == 4) {
      const float4 q = __ldg(reinterpret_cast<const float4*>(p));
      r.v[0] = q.x;
      r.v[1] = q.y;
      r.v[2] = q.z;
      r.v[3] = q.w;
    } else {
      r.v[0] = cl.x < run.g.nx ? __ldg(p) : 0.0f;
    }
    return r;
  }
  // the block's cells of a material plane (zero outside the grid)
  __device__ __forceinline__ void load_own(const Run& run, float (&m)[R][CX], const float* src) const {
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < CX; ++j) {
        const int x = cl.x + j, z = cl.z + k;
        m[k][j] = (t.act && x >= 0 && x < run.g.nx && z >= 0 && z < run.g.nz)
                      ? __ldg(src + (long long)z * run.g.ld + x)
                      : 0.0f;
      }
  }
  __device__ __forceinline__ void store(const Run& run, const float* A, float* dst) const {
    for (int i = threadIdx.x; i < t.TW * t.TH; i += blockDim.x) {
      const int r = i / t.TW, col = i - r * t.TW;
      dst[(long long)(t.z0 + r) * run.g.ld + t.x0 + col] = A[(r + N + 1) * pitch + col + L + t.off];
    }
  }
  __device__ __forceinline__ int dist(const Run& run, int k, int j) const {
    const int x = cl.x + j, z = cl.z + k;
    return min(min(x, run.g.nx - 1 - x), min(z, run.g.nz - 1 - z));
  }
  // ... of a cell that may lie outside the grid, as an index of the ramps
  __device__ __forceinline__ int dist_in(const Run& run, int k, int j) const {
    return min(max(dist(run, k, j), 0), run.h.wstride - 1);
  }
  // sponge.jl:55-78
  __device__ __forceinline__ float damp(const Run& run, const float* wt, int k, int j, float u) const {
    const int d = dist(run, k, j);
    return d >= 0 && d < run.h.nbc ? __fmul_rn(u, wt[d]) : u;
  }
  __device__ __forceinline__ bool inner(int k, int j) const { return cl.inner >> (k * CX + j) & 1; }
  // pre-correction values of the block into an extended array
  __device__ __forceinline__ void stage(float* U, const float (&u)[R][CX]) const {
#pragma unroll
    for (int k = 0; k < R; ++k)
      stv<CX>(U + eb + k * ep, u[k]);
  }
  // Higdon values (kernels_det.jl:22-57) of the block's own frame cells: u their
  // pre-correction values, also in U; F the old values.  Without branches per cell: every
  // cell evaluates both side terms (of itself where it has no such side) and selects.
  __device__ __forceinline__ void blend_row(const Run& run, const HabcDev& h, const float* wt, int kind, int k,
                                            float (&u)[CX], const float* U, const float* F) const {
    const Geom& g = run.g;
    const float* w = wt + kind * h.wstride;
    const unsigned m = cl.frame >> (CX * k) & kRow;
    const int e = eb + k * ep, q = hb + k * pitch;
    const int sz = cl.side(cl.z + k, g.nz, g.nbc);
    const Vec<CX> f = ldv<CX>(F + q), uz = ldv<CX>(U + e + sz * ep),
                  fz = ldv<CX>(F + q + sz * pitch);
    const float ul = U[e - 1], ur = U[e + CX], fl = F[q - 1], fr = F[q + CX];
    float r[CX];
#pragma unroll
    for (int j = 0; j < CX; ++j) {
      const int sx = cl.side(cl.x + j, g.nx, g.nbc);
      const float fo = f[j], wj = w[dist_in(run, k, j)], om = __fsub_rn(1.0f, wj);
      const float ux = sx > 0 ? (j == CX - 1 ? ur : u[j == CX - 1 ? j : j + 1])
                              : (j == 0 ? ul : u[j == 0 ? 0 : j - 1]);
      const float fx = sx > 0 ? (j == CX - 1 ? fr : f[j == CX - 1 ? j : j + 1])
                              : (j == 0 ? fl : f[j == 0 ? 0 : j - 1]);
      const float a = higdon_side(h, ux, fo, fx);
      const float b = higdon_side(h, uz[j], fo, fz[j]);
      const float s = sx != 0 && sz != 0 ? __fmul_rn(__fmul_rn(om, 0.5f), __fadd_rn(a, b))
                                         : __fmul_rn(om, sx != 0 ? a : b);
      r[j] = m >> j & 1 ? __fmaf_rn(wj, u[j], s) : u[j];
    }
#pragma unroll
    for (int j = 0; j < CX; ++j) u[j] = r[j];
  }
  // A barrier after the stores of U, the blend of NF fields (hs: the second one's Higdon
  // terms where they differ), a barrier.
  template <int NF>
  __device__ __forceinline__ void blend(const Run& run, const float* wt, const int (&kind)[NF],
                                        float (*const (&u)[NF])[CX], float* const (&U)[NF],
                                        float* const (&F)[NF],
                                        const HabcDev* hs = nullptr) const {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < R; ++k)
      if (cl.frame >> (CX * k) & kRow) {
#pragma unroll
        for (int f = 0; f < NF; ++f) blend_row(run, f == 1 && hs ? *hs : run.h, wt, kind[f], k, u[f][k], U[f], F[f]);
      }
    __syncthreads();
  }
  // own cells of the block into a haloed array
  __device__ __forceinline__ void keep(float* A, const float (&u)[R][CX]) const {
#pragma unroll
    for (int k = 0; k < R; ++k) {
      float* p = A + hb + k * pitch;
      const unsigned m = cl.own >> (CX * k) & kRow;
      if (m == kRow) {
        stv<CX>(p, u[k]);
      } else if (m) {
#pragma unroll
        for (int j = 0; j < CX; ++j)
          if (m >> j & 1) p[j] = u[k][j];
      }
    }
  }
  // Words of a region of a tile TW x TH as it publishes them: the cells its
  // left / upper neighbour reads, then those of the right / lower one, row by row.
  static __device__ int region_n(const Region& r, int TW, int TH) {
    return r.kind == kStrip ? (r.lo + r.hi) * TH : r.kind == kBand ? (r.lo + r.hi) * TW
           : r.kind == kRows ? 2 * TW : 2 * TH;
  }
  // ... the place of own cell (lx, lz) among them, read from the other side of
  // the tile (`low`: by the right / lower neighbour)
  static __device__ int region_at(const Region& r, int TW, int TH, int lx, int lz, bool low) {
    const int lo = r.lo, hi = r.hi;
    if (r.kind == kStrip) return low ? hi * TH + lz * lo + lx - (TW - lo) : lz * hi + lx;
    if (r.kind == kBand) return low ? hi * TW + (lz - (TH - lo)) * TW + lx : lz * TW + lx;
    if (r.kind == kRows) return low ? TW + lx : lx;
    return low ? TH + lz : lz;
  }
  // Fills the put table (shared-memory places, in publishing order); haloed array f starts
  // at f * hn.  Returns its length.
  __device__ int put_words(int* tab, const Region* reg, int nreg, int hn) const {
    int n0 = 0;
    for (int r = 0; r < nreg; ++r) {
      const int lo = reg[r].lo, hi = reg[r].hi, n = region_n(reg[r], t.TW, t.TH);
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int lx, lz;
        if (reg[r].kind == kStrip) {
          const bool low = i >= hi * t.TH;
          const int q = low ? i - hi * t.TH : i, wd = low ? lo : hi;
          lz = q / wd;
          lx = q - lz * wd + (low ? t.TW - lo : 0);
        } else if (reg[r].kind == kBand) {
          const bool low = i >= hi * t.TW;
          const int q = low ? i - hi * t.TW : i;
          lz = q / t.TW;
          lx = q - lz * t.TW;
          if (low) lz += t.TH - lo;
        } else if (reg[r].kind == kRows) {
          lx = i % t.TW;
          lz = i < t.TW ? 0 : t.TH - 1;
        } else {
          lz = i % t.TH;
          lx = i < t.TH ? 0 : t.TW - 1;
        }
        tab[n0 + i] = reg[r].field * hn + (lz + N + 1) * pitch + lx + L + t.off;
      }
      n0 += n;
    }
    return n0;
  }
  // Fills the get table: the words this tile reads of the regions of its neighbours,
  // whose parts of the plane set are `per` words each.
  __device__ int get_words(const Run& run, Word* tab, const Region* reg, int nreg, int hn,
                           int per) const {
    const Geom& g = run.g;
    const int tz = (blockIdx.x / g.gx) % g.gz, tx = blockIdx.x % g.gx;
    int n0 = 0;
    for (int r = 0; r < nreg; ++r) {
      const int kind = reg[r].kind, lo = reg[r].lo, hi = reg[r].hi;
      const int W = t.TW + 2, H = t.TH + 2;  // with the ring
      const int n = kind == kStrip ? (lo + hi) * H : kind == kBand ? (lo + hi) * W
                    : kind == kRows ? 2 * t.TW : 2 * t.TH;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        int lx, lz;
        if (kind == kStrip) {  // lo columns left, then hi right, rows -1 .. TH
          const bool left = i < lo * H;
          const int q = left ? i : i - lo * H, wd = left ? lo : hi;
          lz = q / wd - 1;
          lx = q - (lz + 1) * wd + (left ? -lo : t.TW);
        } else if (kind == kBand) {  // lo rows above, then below, columns -1 .. TW
          const int k = i / W;
          lx = i - k * W - 1;
          lz = k < lo ? k - lo : t.TH + k - lo;
        } else if (kind == kRows) {
          lx = i % t.TW;
          lz = i < t.TW ? -1 : t.TH;
        } else {
          lz = i % t.TH;
          lx = i < t.TH ? -1 : t.TW;
        }
        const int x = t.x0 + lx, z = t.z0 + lz;
        Word w{-1, reg[r].field * hn + (lz + N + 1) * pitch + lx + L + t.off};
        if (x >= 0 && x < g.nx && z >= 0 && z < g.nz) {
          // the neighbour that owns the cell, and the place among the words it puts
          const int ux = tx + (lx < 0 ? -1 : lx >= t.TW ? 1 : 0);
          const int uz = tz + (lz < 0 ? -1 : lz >= t.TH ? 1 : 0);
          const int ax = tile_x(g.nx, g.gx, ux), az = tile_z(g.nz, g.gz, uz);
          const int TW = tile_x(g.nx, g.gx, ux + 1) - ax, TH = tile_z(g.nz, g.gz, uz + 1) - az;
          int at = 0;
          for (int p = 0; p < r; ++p) at += region_n(reg[p], TW, TH);
          const bool low = kind == kStrip || kind == kCols ? lx < 0 : lz < 0;
          at += region_at(reg[r], TW, TH, x - ax, z - az, low);
          w.g = ((t.shot * g.gz + uz) * g.gx + ux) * per + at;
        }
        tab[n0 + i] = w;
      }
      n0 += n;
    }
    return n0;
  }
  // interior snapshot of the block (fused_kernels.jl:192-195)
  __device__ __forceinline__ void snapshot(const Run& run, float* snaps, int it,
                                           const float (&u)[R][CX]) const {
    float* sn = snaps + (long long)(it / run.snap_interval - 1) * run.nxi * run.nzi;
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < CX; ++j) {
        const int x = cl.x + j - run.pad, z = cl.z + k - run.pad;
        if ((cl.own >> (k * CX + j) & 1) && x >= 0 && x < run.nxi && z >= 0 && z < run.nzi)
          sn[(long long)z * run.nxi + x] = u[k][j];
      }
  }
};

// ---- host side -------------------------------------------------------------
struct Plan {
  bool ok = false;
  Geom g{};
  int form = 0, threads = 0, tiles = 0;
  size_t smem = 0;
  // per-tile entries (host copies; uploaded by the caller)
  std::vector<int> off, ent;
  std::vector<int2> key;
};

// What a solver keeps in shared memory: `hal` haloed arrays, `ext` arrays over the
// extended tile, `mats` materials (in registers where blocks have up to mreg cells,
// else extended arrays, or off the chip where those do not fit) and the words of its regions (counts per kind).
struct Needs {
  int hal, ext, mats, mreg, strips, bands, rows, cols;
  int wide;  // strips and bands are 2N + 1 + wide cells wide in all
  int forms; // block forms in use: the elastic and coupled updates spill some words in
             // every form (52 / 96 bytes stored / loaded at 4 x 1, order 8), in 4 x 4 blocks
             // so many that launches are faster (elastic 700x600 30.2 us per step against 23.2)
};
constexpr Needs kAcousticNeeds{3, 2, 3, 8, 2, 2, 1, 1, 0, 4};
constexpr Needs kElasticNeeds{5, 3, 5, 0, 4, 4, 1, 1, 0, 3};
constexpr Needs kScalarNeeds{1, 1, 1, 8, 1, 1, 0, 0, 1, 4};
constexpr Needs kCoupledNeeds{4, 2, 8, 0, 2, 2, 2, 2, 1, 3};
// Chooses the tiles of a run (extra: floats of the weight ramps); ok = false when it
// does not fit on the chip.
Plan make_plan(const Needs& needs, int N, int nx, int nz, int ld, int nbc, int ns, int nsm,
               int extra);
// Floats of the weight ramps (or the sponge's damping table).
inline int smem_extra(int wstride, int nbc_sponge) { return std::max(3 * wstride, nbc_sponge) + 4; }
// Distributes the cells of the run's tags over the tiles' threads.
void plan_entries(Plan& p, int ns, const CellTagHost& tags);

// A run's tables in the context workspace: taken from the arena, then uploaded on st
// with the exchange buffer cleared, which completes the device pointers of `run`.
struct Tables {
  size_t off = 0, key = 0, ent = 0, ll = 0, ll_words = 0;
};
Tables take_tables(Arena& ar, const Plan& p);
cudaError_t upload_tables(cudaStream_t st, char* ws, const Plan& p, const Tables& t,
                          const CellTags& tags, Run& run);
// Runs of more steps than this keep their state on the chip when it fits.  The line is
// not where the time turns: on chip a call is the faster one from 10 to 50 steps on (call
// ms, on chip / launched, at 50, 100 and 300 steps: acoustic 400x300 nbc 100 0.7 / 1.2,
// 1.1 / 2.0, 2.4 / 4.7; 1000x800 2.0 / 2.1, 2.7 / 2.9, 5.4 / 6.2; elastic 501x397 1.1 / 1.5,
// 1.7 / 2.6, 3.9 / 5.9; coupled 400x300 1.0 / 1.3, 1.6 / 2.2, 3.7 / 5.1).  Up to here runs keep
// the replayed launches, whose number callers read in the stats and tests fix at 300 steps.
constexpr int kMinSteps = 300;
int sm_count(int device);

// Device planes of a launch: materials and the state read (null: zero) and written.
struct Fields {
  // acoustic bx, bz, kappa; elastic bx, bz, lam, l2m, mut; scalar c2; coupled the
  // eight planes of CoupledMedium
  const float* mat[8];
  // acoustic vx, vz, p; elastic vx, vz, txx, tzz, txz; scalar u^n, u^{n-1}; coupled P, S,
  // dP/dt, dS/dt
  const float* in[5];
  float* out[5];
};
// Centered-difference coefficients (scalar, coupled).
struct Centered {
  float c0;               // scalar 2 c0 of the Laplacian, coupled c0
  float d1[5], d2[5];     // first (coupled) and second differences
  float dt, ih, ih2;      // coupled
  HabcDev hs;             // coupled: the S fields' Higdon terms
  float* snaps_s;
};
cudaError_t launch_scalar(cudaStream_t st, int N, const Plan& p, const Run& run, const Fields& f,
                          const Centered& c);
cudaError_t launch_coupled(cudaStream_t st, int N, const Plan& p, const Run& run, const Fields& f,
                           const Centered& c);
cudaError_t launch_acoustic(cudaStream_t st, int N, bool sponge, const Plan& p, const Run& run,
                            const Fields& f);
cudaError_t launch_elastic(cudaStream_t st, int N, bool sponge, const Plan& p, const Run& run,
                           const Fields& f);

// switch over the block forms: M(index, CX, R, threads)
#define FOMO_RES_FORMS3(M) M(0, 1, 1, 1024) M(1, 4, 1, 640) M(2, 4, 2, 512)
#define FOMO_RES_FORMS(M) FOMO_RES_FORMS3(M) M(3, 4, 4, 512)

template <class Kern, class... More>
cudaError_t launch_resident(cudaStream_t st, Kern kern, const Plan& p, const Run& run,
                            const Fields& f, const More&... more) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       227 * 1024);
  if (e != cudaSuccess) return e;
  Run r = run;
  Fields ff = f;
  void* args[] = {&r, &ff, const_cast<More*>(&more)...};
  return cudaLaunchCooperativeKernel((const void*)kern, dim3(p.tiles), dim3(p.threads), args,
                                     p.smem, st);
}

}  // namespace res
}  // namespace fomo
