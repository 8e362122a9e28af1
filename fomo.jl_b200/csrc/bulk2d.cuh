// bulk2d.cuh -- two-phase kernels of large 2D grids.
//
// The cell-per-thread kernels (solver2d_kernels.cuh) load every stencil operand as a
// word of its own: 41 loads per acoustic cell and step, bound by issue at a third of the
// bandwidth.  Away from the edges a thread here owns 4 x R cells: 16-byte loads, the z
// window in registers, the x window from three words, so an acoustic cell costs about
// five loaded words per half step.  One launch covers the grid: its first blocks take the
// four edge rectangles (Higdon zone or sponge), a quad of a row per thread, which evaluates
// the interior-ward neighbour row (and cell) again; the others the inner rectangle.
// Same per-cell arithmetic, equal bit for bit.
// Acoustic, order 8, nbc 50, us per step, cell-per-thread / this: 700x600 16.8 / 12.9, 1000x800
// 22.7 / 14.2, 1400x1000 31.5 / 17.8, 2000x1600 68.2 / 37.3 (4.6 TB/s of the 48 B that the two half
// steps move per cell; the working set of 130 MB is just over L2), 8 shots of 600x500
// 63.9 / 42.0.  Elastic: 700x600 24.5 / 18.2, 1000x800 34.9 / 22.0, 1400x1000 65.8 / 31.3,
// 2000x1600 157 / 67.5.  Scalar: 1000x800 10.9 / 6.8, 2000x1600 25.9 / 17.6.
#pragma once
#include "resident2d.cuh"

namespace fomo {
namespace bulk {

constexpr int kW = 128;  // columns of an inner tile: a warp of 4-cell threads
constexpr int kThreads = 256;
// CTAs per SM that the acoustic kernels' registers are bounded to: without the bound
// (2 to 3) too few loads are in flight to cover the latency (64 uneven
// shots 466 us per step, with 4 349, with 5 372).  At 4 some forms spill a few words (8 to 12
// bytes untagged, the tagged order-8 pressure kernel 96 / 104), at 5 all of them many.
constexpr int ac_blocks(int N) { return N <= 4 ? 4 : 3; }

// The inner rectangle [x0, x1) x [z0, z1) (x0, x1 multiples of 4), its tiles, and the
// quads (4 cells of a row) of the edge rectangles: above and below it (full rows), left
// and right of it.
struct Split {
  int x0, x1, z0, z1;
  int tx, tiles;            // tiles per row, tiles
  int nq, lq, rq;           // quads per row: full, left, right
  int top, bottom, left;    // first quad after the top, bottom and left rectangles
  int quads, edge;          // edge quads, edge blocks
};

// edge: cells within this distance of the grid's edge are not inner cells.
inline Split make_split(const Geo2& g, int edge, int rows) {
  Split s;
  s.x0 = (edge + 3) & ~3;
  s.x1 = std::max(s.x0, (g.nx - edge) & ~3);
  s.z0 = edge;
  s.z1 = std::max(s.z0, g.nz - edge);
  s.tx = (s.x1 - s.x0 + kW - 1) / kW;
  s.tiles = s.tx * ((s.z1 - s.z0 + rows - 1) / rows);
  s.nq = (g.nx + 3) / 4;
  s.lq = s.x0 / 4;
  s.rq = (g.nx - s.x1 + 3) / 4;
  s.top = s.nq * s.z0;
  s.bottom = s.top + s.nq * (g.nz - s.z1);
  s.left = s.bottom + s.lq * (s.z1 - s.z0);
  s.quads = s.left + s.rq * (s.z1 - s.z0);
  s.edge = (s.quads + kThreads - 1) / kThreads;
  return s;
}

// First cell of edge quad i.
__device__ __forceinline__ void edge_quad(const Split& s, int i, int& x, int& z) {
  int n = s.nq, xa = 0, za = 0;
  if (i >= s.left) {
    i -= s.left;
    n = s.rq;
    xa = s.x1;
    za = s.z0;
  } else if (i >= s.bottom) {
    i -= s.bottom;
    n = s.lq;
    za = s.z0;
  } else if (i >= s.top) {
    i -= s.top;
    za = s.z1;
  }
  const int r = i / n;
  x = xa + 4 * (i - r * n);
  z = za + r;
}

__device__ __forceinline__ res::Vec<4> ldg4(const float* __restrict__ p) {
  const float4 q = __ldg(reinterpret_cast<const float4*>(p));
  return res::Vec<4>{{q.x, q.y, q.z, q.w}};
}
// ... of a word that this step does not read again: it leaves L2 first, so that the
// fields which the next half step reads stay (acoustic 2000x1600 41.7 -> 37.3 us per step,
// order 4 39.6 -> 35.5; sizes that fit in L2 unchanged).
__device__ __forceinline__ res::Vec<4> lds4(const float* __restrict__ p) {
  const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
  return res::Vec<4>{{q.x, q.y, q.z, q.w}};
}
template <int N>
struct GWin : res::XWin<N, 4> {
  using B = res::XWin<N, 4>;
  __device__ __forceinline__ void load(const float* __restrict__ p) {
#pragma unroll
    for (int i = -B::G; i <= B::G; ++i) {
      const res::Vec<4> v = ldg4(p + 4 * i);
#pragma unroll
      for (int j = 0; j < 4; ++j) this->w[B::L + 4 * i + j] = v[j];
    }
  }
};
__device__ __forceinline__ void stg4(float* p, const float (&u)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(u[0], u[1], u[2], u[3]);
}

// A quad's row window and z window near the grid's edge: words that would lie outside
// the rows read the quad itself, rows outside the grid the nearest one.  Such values only
// reach cells outside the stencil's range, which keep their old values.
template <int N>
__device__ __forceinline__ void edge_window(const Geo2& g, const float* __restrict__ f, int x, int z,
                                            GWin<N>& w) {
  using B = res::XWin<N, 4>;
  const float* __restrict__ p = f + (long long)z * g.ld + x;
#pragma unroll
  for (int i = -B::G; i <= B::G; ++i) {
    const bool in = x + 4 * i >= 0 && x + 4 * i < g.ld;
    const res::Vec<4> v = ldg4(in ? p + 4 * i : p);
#pragma unroll
    for (int j = 0; j < 4; ++j) w.w[B::L + 4 * i + j] = v[j];
  }
}
// rows z - lo .. z - lo + 2N - 1
template <int N>
__device__ __forceinline__ void edge_rows(const Geo2& g, const float* __restrict__ f, int x, int z,
                                          int lo, res::Vec<4> (&w)[2 * N]) {
#pragma unroll
  for (int i = 0; i < 2 * N; ++i)
    w[i] = ldg4(f + (long long)min(max(z - lo + i, 0), g.nz - 1) * g.ld + x);
}

// Higdon values of an edge quad for NF fields (kernels_det.jl:22-57): u pre-correction
// values of the quad (replaced), v those of the row z + sz, e those of the cell beside the quad on
// its interior-ward x side; F the old fields.
template <int NF>
__device__ __forceinline__ void edge_blend(const Geo2& g, const HabcDev& h, int x, int z, int sz,
                                           const int (&kind)[NF], float (&u)[NF][4],
                                           const float (&v)[NF][4], const float (&e)[NF],
                                           const float* const (&F)[NF]) {
  const long long p = (long long)z * g.ld + x;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    const res::Vec<4> o = ldg4(F[f] + p), oz = ldg4(F[f] + p + (long long)sz * g.ld);
    float r[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int xx = x + j;
      const int sx = xx <= g.nbc ? 1 : (xx >= g.nx - 1 - g.nbc ? -1 : 0);
      r[j] = u[f][j];
      if (xx < 1 || xx > g.nx - 2 || (sx == 0 && sz == 0)) continue;
      const int dist = min(min(xx, g.nx - 1 - xx), min(z, g.nz - 1 - z));
      const float w = habc_weight(h, kind[f], dist);
      const bool out = sx > 0 ? j == 3 : j == 0;  // the x neighbour lies outside the quad
      const int jn = sx > 0 ? (j == 3 ? 3 : j + 1) : (j == 0 ? 0 : j - 1);
      const float ux = out ? e[f] : u[f][jn];
      const float fx = sx == 0 ? 0.0f : (out ? __ldg(F[f] + p + j + sx) : o[jn]);
      if (sx != 0 && sz != 0)
        r[j] = higdon_corner(w, u[f][j], higdon_side(h, ux, o[j], fx),
                             higdon_side(h, v[f][j], o[j], oz[j]));
      else
        r[j] = higdon_edge(w, u[f][j], sx != 0 ? higdon_side(h, ux, o[j], fx)
                                               : higdon_side(h, v[f][j], o[j], oz[j]));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) u[f][j] = r[j];
  }
}
// Sides of an edge quad: sz of its row (0 on the grid's outermost rows, which the frame
// leaves out), ex the column of the x neighbour beside the quad (-1: none needed).
__device__ __forceinline__ bool edge_sides(const Geo2& g, int x, int z, int& sz, int& ex) {
  if (z < 1 || z > g.nz - 2) return false;
  sz = z <= g.nbc ? 1 : (z >= g.nz - 1 - g.nbc ? -1 : 0);
  ex = x + 3 <= g.nbc && x + 3 <= g.nx - 2 ? x + 4 : (x >= g.nx - 1 - g.nbc && x > g.nbc ? x - 1 : -1);
  return true;
}
__device__ __forceinline__ void edge_store(const Geo2& g, float* f, int x, const float (&u)[4]) {
  if (x + 3 < g.nx) {
    stg4(f, u);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (x + j < g.nx) f[j] = u[j];
  }
}

// Pre-correction velocities / pressure of an edge quad (ac_vel_at, ac_prs_at).
template <int N>
__device__ __forceinline__ void ac_vel_quad(const Geo2& g, const Coef& c, float dtx, float dtz,
                                            const float* __restrict__ p0,
                                            const float* __restrict__ vx0,
                                            const float* __restrict__ vz0,
                                            const float* __restrict__ bx,
                                            const float* __restrict__ bz, int x, int z,
                                            float (&u)[2][4]) {
  const long long p = (long long)z * g.ld + x;
  const res::Vec<4> ox = ldg4(vx0 + p), oz = ldg4(vz0 + p), mx = ldg4(bx + p), mz = ldg4(bz + p);
  GWin<N> xw;
  edge_window<N>(g, p0, x, z, xw);
  res::Vec<4> w[2 * N];
  edge_rows<N>(g, p0, x, z, N - 1, w);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool in = interior2(g, x + j, z);
    const float ux = __fmaf_rn(__fmul_rn(mx[j], dtx), xw.dm(j, c), ox[j]);
    const float uz = __fmaf_rn(__fmul_rn(mz[j], dtz), res::zdp<N, 4>(w, N - 1, j, c), oz[j]);
    u[0][j] = in ? ux : ox[j];
    u[1][j] = in ? uz : oz[j];
  }
}
template <int N>
__device__ __forceinline__ void ac_prs_quad(const Geo2& g, const Coef& c, float dtx, float dtz,
                                            const float* __restrict__ vx,
                                            const float* __restrict__ vz,
                                            const float* __restrict__ p0,
                                            const float* __restrict__ kappa, int x, int z,
                                            float (&u)[1][4]) {
  const long long p = (long long)z * g.ld + x;
  const res::Vec<4> op = ldg4(p0 + p), ka = ldg4(kappa + p);
  GWin<N> xw;
  edge_window<N>(g, vx, x, z, xw);
  res::Vec<4> w[2 * N];
  edge_rows<N>(g, vz, x, z, N, w);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float v = __fmaf_rn(
        ka[j], __fmaf_rn(xw.dp(j, c), dtx, __fmul_rn(res::zdm<N, 4>(w, N, j, c), dtz)), op[j]);
    u[0][j] = interior2(g, x + j, z) ? v : op[j];
  }
}

// First cell (4 columns, R rows) of this thread in inner tile b; false outside.
template <int R>
__device__ __forceinline__ bool inner_cells(const Split& s, int b, int& x, int& z, int& rows) {
  const int ty = b / s.tx;
  x = s.x0 + (b - ty * s.tx) * kW + 4 * (threadIdx.x & 31);
  z = s.z0 + (ty * (kThreads / 32) + (threadIdx.x >> 5)) * R;
  rows = s.z1 - z;
  return x < s.x1 && rows > 0;
}

// Block `blk` of the acoustic velocity half step of one shot.
template <int N, int R, bool SP>
__device__ __forceinline__ void ac_vel_block(int blk, const Geo2& g, const Split& s, const Coef& c,
                                             float dtx, float dtz, const HabcDev& h,
                                             const float* __restrict__ p0,
                                             const float* __restrict__ vx0,
                                             const float* __restrict__ vz0,
                                             const float* __restrict__ bx,
                                             const float* __restrict__ bz,
                                             float* __restrict__ vx1, float* __restrict__ vz1) {
  int x, z;
  if (blk < s.edge) {
    const int i = blk * kThreads + threadIdx.x;
    if (i >= s.quads) return;
    edge_quad(s, i, x, z);
    float u[2][4];
    ac_vel_quad<N>(g, c, dtx, dtz, p0, vx0, vz0, bx, bz, x, z, u);
    int sz, ex;
    if constexpr (SP) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u[0][j] = x + j < g.nx ? sponge_damp(g, h, x + j, z, u[0][j]) : 0.0f;
        u[1][j] = x + j < g.nx ? sponge_damp(g, h, x + j, z, u[1][j]) : 0.0f;
      }
    } else if (edge_sides(g, x, z, sz, ex)) {
      float v[2][4] = {}, e[2] = {};
      if (sz) ac_vel_quad<N>(g, c, dtx, dtz, p0, vx0, vz0, bx, bz, x, z + sz, v);
      if (ex >= 0) ac_vel_at<N>(g, c, dtx, dtz, p0, vx0, vz0, bx, bz, ex, z, e[0], e[1]);
      edge_blend<2>(g, h, x, z, sz, {0, 1}, u, v, e, {vx0, vz0});
    }
    const long long p = (long long)z * g.ld + x;
    edge_store(g, vx1 + p, x, u[0]);
    edge_store(g, vz1 + p, x, u[1]);
    return;
  }
  int rows;
  if (!inner_cells<R>(s, blk - s.edge, x, z, rows)) return;
  const long long q = (long long)z * g.ld + x;
  constexpr int NWIN = R + 2 * N - 1;
  res::Vec<4> w[NWIN];  // p rows z - (N - 1) .. (rows past the rectangle are still in the grid)
#pragma unroll
  for (int i = 0; i < NWIN; ++i)
    w[i] = ldg4(p0 + q + (long long)min(i - (N - 1), rows - 1 + N) * g.ld);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (k >= rows) break;
    const long long e = q + (long long)k * g.ld;
    GWin<N> xw;
    xw.load(p0 + e);
    const res::Vec<4> ox = lds4(vx0 + e), oz = lds4(vz0 + e), mx = lds4(bx + e), mz = lds4(bz + e);
    float ux[4], uz[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      ux[j] = __fmaf_rn(__fmul_rn(mx[j], dtx), xw.dm(j, c), ox[j]);
      uz[j] = __fmaf_rn(__fmul_rn(mz[j], dtz), res::zdp<N, 4>(w, N - 1 + k, j, c), oz[j]);
    }
    stg4(vx1 + e, ux);
    stg4(vz1 + e, uz);
  }
}
template <int N, int R, bool SP>
__global__ void __launch_bounds__(kThreads, ac_blocks(N))
    k_ac_vel_bulk(Geo2 g, Split s, Coef c, float dtx, float dtz, HabcDev h,
                  const float* __restrict__ p0, const float* __restrict__ vx0,
                  const float* __restrict__ vz0, const float* __restrict__ bx,
                  const float* __restrict__ bz, float* __restrict__ vx1,
                  float* __restrict__ vz1) {
  const long long so = (long long)blockIdx.z * g.plane;
  ac_vel_block<N, R, SP>(blockIdx.x, g, s, c, dtx, dtz, h, p0 + so, vx0 + so, vz0 + so, bx, bz,
                         vx1 + so, vz1 + so);
}

// Block `blk` of the pressure half step.  TG: inject into p and record p, vx, vz on tagged
// cells (step *t.it0 + j0 + 1).
template <int N, int R, bool SP, bool TG>
__device__ __forceinline__ void ac_prs_block(int blk, int shot, const Geo2& g, const Split& s,
                                             const Coef& c, float dtx, float dtz, const HabcDev& h,
                                             const float* __restrict__ p0,
                                             const float* __restrict__ vx1,
                                             const float* __restrict__ vz1,
                                             const float* __restrict__ kappa,
                                             float* __restrict__ p1, const CellTags& t, int j0) {
  auto tagged = [&](int e, long long p, float u) {
    const long long k = (long long)(*t.it0 + j0);
    const int4 E = t.ent[e];
    u = tag_inject(t, E, k, shot, u);
    tag_record(t, E, k, shot, u, __ldg(vx1 + p), __ldg(vz1 + p));
    return u;
  };
  int x, z;
  if (blk < s.edge) {
    const int i = blk * kThreads + threadIdx.x;
    if (i >= s.quads) return;
    edge_quad(s, i, x, z);
    float u[1][4];
    ac_prs_quad<N>(g, c, dtx, dtz, vx1, vz1, p0, kappa, x, z, u);
    int sz, ex;
    if constexpr (SP) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        u[0][j] = x + j < g.nx ? sponge_damp(g, h, x + j, z, u[0][j]) : 0.0f;
    } else if (edge_sides(g, x, z, sz, ex)) {
      float v[1][4] = {}, e[1] = {};
      if (sz) ac_prs_quad<N>(g, c, dtx, dtz, vx1, vz1, p0, kappa, x, z + sz, v);
      if (ex >= 0) e[0] = ac_prs_at<N>(g, c, dtx, dtz, vx1, vz1, p0, kappa, ex, z);
      edge_blend<1>(g, h, x, z, sz, {2}, u, v, e, {p0});
    }
    const long long p = (long long)z * g.ld + x;
    if constexpr (TG) {  // sources and receivers may lie in the edge rectangles' inner cells
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + j < g.nx) {
          const int e = __ldg(t.tag + p + j);
          if (e >= 0) u[0][j] = tagged(e, p + j, u[0][j]);
        }
    }
    edge_store(g, p1 + p, x, u[0]);
    return;
  }
  int rows;
  if (!inner_cells<R>(s, blk - s.edge, x, z, rows)) return;
  const long long q = (long long)z * g.ld + x;
  constexpr int NWIN = R + 2 * N - 1;
  res::Vec<4> w[NWIN];  // vz rows z - N ..
#pragma unroll
  for (int i = 0; i < NWIN; ++i)
    w[i] = ldg4(vz1 + q + (long long)min(i - N, rows - 1 + N) * g.ld);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (k >= rows) break;
    const long long e = q + (long long)k * g.ld;
    GWin<N> xw;
    xw.load(vx1 + e);
    const res::Vec<4> op = lds4(p0 + e), ka = lds4(kappa + e);
    float u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      u[j] = __fmaf_rn(ka[j],
                       __fmaf_rn(xw.dp(j, c), dtx, __fmul_rn(res::zdm<N, 4>(w, N + k, j, c), dtz)),
                       op[j]);
    if constexpr (TG) {
      const int4 tg = __ldg(reinterpret_cast<const int4*>(t.tag + e));
      if (tg.x >= 0) u[0] = tagged(tg.x, e, u[0]);
      if (tg.y >= 0) u[1] = tagged(tg.y, e + 1, u[1]);
      if (tg.z >= 0) u[2] = tagged(tg.z, e + 2, u[2]);
      if (tg.w >= 0) u[3] = tagged(tg.w, e + 3, u[3]);
    }
    stg4(p1 + e, u);
  }
}
template <int N, int R, bool SP, bool TG>
__global__ void __launch_bounds__(kThreads, ac_blocks(N))
    k_ac_prs_bulk(Geo2 g, Split s, Coef c, float dtx, float dtz, HabcDev h,
                  const float* __restrict__ p0, const float* __restrict__ vx1,
                  const float* __restrict__ vz1, const float* __restrict__ kappa,
                  float* __restrict__ p1, CellTags t, int j0) {
  const long long so = (long long)blockIdx.z * g.plane;
  ac_prs_block<N, R, SP, TG>(blockIdx.x, blockIdx.z, g, s, c, dtx, dtz, h, p0 + so, vx1 + so,
                             vz1 + so, kappa, p1 + so, t, j0);
}

// Pre-correction velocities / stresses of an edge quad (el_vel_at, el_str_at).
template <int N>
__device__ __forceinline__ void el_vel_quad(const Geo2& g, const Coef& c, float dtx, float dtz,
                                            const ElFields& a, const ElMat& m, int x, int z,
                                            float (&u)[2][4]) {
  const long long p = (long long)z * g.ld + x;
  float zx[4], zz[4];
  {
    res::Vec<4> w[2 * N];
    edge_rows<N>(g, a.txz, x, z, N, w);
#pragma unroll
    for (int j = 0; j < 4; ++j) zx[j] = __fmul_rn(dtz, res::zdm<N, 4>(w, N, j, c));
    edge_rows<N>(g, a.tzz, x, z, N - 1, w);
#pragma unroll
    for (int j = 0; j < 4; ++j) zz[j] = __fmul_rn(dtz, res::zdp<N, 4>(w, N - 1, j, c));
  }
  GWin<N> xw;
  edge_window<N>(g, a.txx, x, z, xw);
  const res::Vec<4> ox = ldg4(a.vx + p), oz = ldg4(a.vz + p), bx = ldg4(m.bx + p),
                    bz = ldg4(m.bz + p);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float v = __fmaf_rn(bx[j], __fmaf_rn(dtx, xw.dm(j, c), zx[j]), ox[j]);
    u[0][j] = interior2(g, x + j, z) ? v : ox[j];
  }
  edge_window<N>(g, a.txz, x, z, xw);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float v = __fmaf_rn(bz[j], __fmaf_rn(dtx, xw.dp(j, c), zz[j]), oz[j]);
    u[1][j] = interior2(g, x + j, z) ? v : oz[j];
  }
}
template <int N>
__device__ __forceinline__ void el_str_quad(const Geo2& g, const Coef& c, float dtx, float dtz,
                                            const float* __restrict__ vx,
                                            const float* __restrict__ vz, const ElFields& a,
                                            const ElMat& m, int x, int z, float (&u)[3][4]) {
  const long long p = (long long)z * g.ld + x;
  float ez[4], sh[4];
  {
    res::Vec<4> w[2 * N];
    edge_rows<N>(g, vz, x, z, N, w);
#pragma unroll
    for (int j = 0; j < 4; ++j) ez[j] = __fmul_rn(res::zdm<N, 4>(w, N, j, c), dtz);
    edge_rows<N>(g, vx, x, z, N - 1, w);
#pragma unroll
    for (int j = 0; j < 4; ++j) sh[j] = res::zdp<N, 4>(w, N - 1, j, c);
  }
  GWin<N> xw;
  edge_window<N>(g, vx, x, z, xw);
  const res::Vec<4> oxx = ldg4(a.txx + p), ozz = ldg4(a.tzz + p), oxz = ldg4(a.txz + p);
  const res::Vec<4> la = ldg4(m.lam + p), l2 = ldg4(m.l2m + p), mu = ldg4(m.mut + p);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float ex = __fmul_rn(xw.dp(j, c), dtx);
    const bool in = interior2(g, x + j, z);
    u[0][j] = in ? __fadd_rn(oxx[j], __fmaf_rn(l2[j], ex, __fmul_rn(la[j], ez[j]))) : oxx[j];
    u[1][j] = in ? __fadd_rn(ozz[j], __fmaf_rn(la[j], ex, __fmul_rn(l2[j], ez[j]))) : ozz[j];
  }
  edge_window<N>(g, vz, x, z, xw);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float v = __fmaf_rn(mu[j], __fmaf_rn(sh[j], dtz, __fmul_rn(xw.dm(j, c), dtx)), oxz[j]);
    u[2][j] = interior2(g, x + j, z) ? v : oxz[j];
  }
}

template <int N, int R, bool SP>
__global__ void __launch_bounds__(kThreads)
    k_el_vel_bulk(Geo2 g, Split s, Coef c, float dtx, float dtz, HabcDev h, ElFields a, ElMat m,
                  float* __restrict__ vx1, float* __restrict__ vz1) {
  const long long so = (long long)blockIdx.z * g.plane;
  a.vx += so; a.vz += so; a.txx += so; a.tzz += so; a.txz += so;
  int x, z;
  if ((int)blockIdx.x < s.edge) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= s.quads) return;
    edge_quad(s, i, x, z);
    float u[2][4];
    el_vel_quad<N>(g, c, dtx, dtz, a, m, x, z, u);
    int sz, ex;
    if constexpr (SP) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        u[0][j] = x + j < g.nx ? sponge_damp(g, h, x + j, z, u[0][j]) : 0.0f;
        u[1][j] = x + j < g.nx ? sponge_damp(g, h, x + j, z, u[1][j]) : 0.0f;
      }
    } else if (edge_sides(g, x, z, sz, ex)) {
      float v[2][4] = {}, e[2] = {};
      if (sz) el_vel_quad<N>(g, c, dtx, dtz, a, m, x, z + sz, v);
      if (ex >= 0) el_vel_at<N>(g, c, dtx, dtz, a, m, ex, z, e[0], e[1]);
      edge_blend<2>(g, h, x, z, sz, {0, 1}, u, v, e, {a.vx, a.vz});
    }
    const long long p = so + (long long)z * g.ld + x;
    edge_store(g, vx1 + p, x, u[0]);
    edge_store(g, vz1 + p, x, u[1]);
    return;
  }
  int rows;
  if (!inner_cells<R>(s, blockIdx.x - s.edge, x, z, rows)) return;
  const long long q = (long long)z * g.ld + x;
  constexpr int NWIN = R + 2 * N - 1;
  float zx[R][4], zz[R][4];
  {  // one register window at a time
    res::Vec<4> w[NWIN];
#pragma unroll
    for (int i = 0; i < NWIN; ++i)
      w[i] = ldg4(a.txz + q + (long long)min(i - N, rows - 1 + N) * g.ld);
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) zx[k][j] = __fmul_rn(dtz, res::zdm<N, 4>(w, N + k, j, c));
#pragma unroll
    for (int i = 0; i < NWIN; ++i)
      w[i] = ldg4(a.tzz + q + (long long)min(i - (N - 1), rows - 1 + N) * g.ld);
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) zz[k][j] = __fmul_rn(dtz, res::zdp<N, 4>(w, N - 1 + k, j, c));
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (k >= rows) break;
    const long long e = q + (long long)k * g.ld;
    GWin<N> xw;
    xw.load(a.txx + e);
    const res::Vec<4> ox = lds4(a.vx + e), oz = lds4(a.vz + e), bx = lds4(m.bx + e),
                      bz = lds4(m.bz + e);
    float u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      u[j] = __fmaf_rn(bx[j], __fmaf_rn(dtx, xw.dm(j, c), zx[k][j]), ox[j]);
    stg4(vx1 + so + e, u);
    xw.load(a.txz + e);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      u[j] = __fmaf_rn(bz[j], __fmaf_rn(dtx, xw.dp(j, c), zz[k][j]), oz[j]);
    stg4(vz1 + so + e, u);
  }
}

// TG: inject into txx, tzz and record vx, vz on tagged cells (step *t.it0 + j0 + 1).
template <int N, int R, bool SP, bool TG>
__global__ void __launch_bounds__(kThreads)
    k_el_str_bulk(Geo2 g, Split s, Coef c, float dtx, float dtz, HabcDev h, ElFields a,
                  const float* __restrict__ vx1, const float* __restrict__ vz1, ElMat m,
                  float* __restrict__ txx1, float* __restrict__ tzz1, float* __restrict__ txz1,
                  CellTags t, int j0) {
  const long long so = (long long)blockIdx.z * g.plane;
  a.txx += so; a.tzz += so; a.txz += so;
  vx1 += so;
  vz1 += so;
  auto tagged = [&](int e, long long p, float& sxx, float& szz) {
    const long long k = (long long)(*t.it0 + j0);
    const int4 E = t.ent[e];
    sxx = tag_inject(t, E, k, blockIdx.z, sxx);
    szz = tag_inject(t, E, k, blockIdx.z, szz);
    tag_record(t, E, k, blockIdx.z, __ldg(vx1 + p), __ldg(vz1 + p), 0.0f);
  };
  int x, z;
  if ((int)blockIdx.x < s.edge) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= s.quads) return;
    edge_quad(s, i, x, z);
    float u[3][4];
    el_str_quad<N>(g, c, dtx, dtz, vx1, vz1, a, m, x, z, u);
    int sz, ex;
    if constexpr (SP) {
#pragma unroll
      for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          u[f][j] = x + j < g.nx ? sponge_damp(g, h, x + j, z, u[f][j]) : 0.0f;
    } else if (edge_sides(g, x, z, sz, ex)) {
      float v[3][4] = {}, e[3] = {};
      if (sz) el_str_quad<N>(g, c, dtx, dtz, vx1, vz1, a, m, x, z + sz, v);
      if (ex >= 0) el_str_at<N>(g, c, dtx, dtz, vx1, vz1, a, m, ex, z, e[0], e[1], e[2]);
      edge_blend<3>(g, h, x, z, sz, {2, 2, 2}, u, v, e, {a.txx, a.tzz, a.txz});
    }
    const long long p = (long long)z * g.ld + x;
    if constexpr (TG) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + j < g.nx) {
          const int e = __ldg(t.tag + p + j);
          if (e >= 0) tagged(e, p + j, u[0][j], u[1][j]);
        }
    }
    edge_store(g, txx1 + so + p, x, u[0]);
    edge_store(g, tzz1 + so + p, x, u[1]);
    edge_store(g, txz1 + so + p, x, u[2]);
    return;
  }
  int rows;
  if (!inner_cells<R>(s, blockIdx.x - s.edge, x, z, rows)) return;
  const long long q = (long long)z * g.ld + x;
  constexpr int NWIN = R + 2 * N - 1;
  float ez[R][4], sh[R][4];
  {
    res::Vec<4> w[NWIN];
#pragma unroll
    for (int i = 0; i < NWIN; ++i)
      w[i] = ldg4(vz1 + q + (long long)min(i - N, rows - 1 + N) * g.ld);
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) ez[k][j] = __fmul_rn(res::zdm<N, 4>(w, N + k, j, c), dtz);
#pragma unroll
    for (int i = 0; i < NWIN; ++i)
      w[i] = ldg4(vx1 + q + (long long)min(i - (N - 1), rows - 1 + N) * g.ld);
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) sh[k][j] = res::zdp<N, 4>(w, N - 1 + k, j, c);
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (k >= rows) break;
    const long long e = q + (long long)k * g.ld;
    GWin<N> xw;
    xw.load(vx1 + e);
    float sxx[4], szz[4], sxz[4];
    {
      const res::Vec<4> oxx = lds4(a.txx + e), ozz = lds4(a.tzz + e), la = lds4(m.lam + e),
                        l2 = lds4(m.l2m + e);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float ex = __fmul_rn(xw.dp(j, c), dtx);
        sxx[j] = __fadd_rn(oxx[j], __fmaf_rn(l2[j], ex, __fmul_rn(la[j], ez[k][j])));
        szz[j] = __fadd_rn(ozz[j], __fmaf_rn(la[j], ex, __fmul_rn(l2[j], ez[k][j])));
      }
    }
    xw.load(vz1 + e);
    const res::Vec<4> oxz = lds4(a.txz + e), mu = lds4(m.mut + e);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      sxz[j] = __fmaf_rn(mu[j], __fmaf_rn(sh[k][j], dtz, __fmul_rn(xw.dm(j, c), dtx)), oxz[j]);
    if constexpr (TG) {
      const int4 tg = __ldg(reinterpret_cast<const int4*>(t.tag + e));
      if (tg.x >= 0) tagged(tg.x, e, sxx[0], szz[0]);
      if (tg.y >= 0) tagged(tg.y, e + 1, sxx[1], szz[1]);
      if (tg.z >= 0) tagged(tg.z, e + 2, sxx[2], szz[2]);
      if (tg.w >= 0) tagged(tg.w, e + 3, sxx[3], szz[3]);
    }
    stg4(txx1 + so + e, sxx);
    stg4(tzz1 + so + e, szz);
    stg4(txz1 + so + e, sxz);
  }
}

// scalar2d leapfrog (sc_at): u2 from u1, u0.
template <int N>
__device__ __forceinline__ float sc_cell(const D2Coef& c, float uc, float u0, float c2,
                                         const float (&nb)[N]) {
  float lap = __fmul_rn(c.two_c0, uc);
#pragma unroll
  for (int l = 0; l < N; ++l) lap = __fmaf_rn(c.d[l], nb[l], lap);
  return __fmaf_rn(c2, lap, __fsub_rn(__fmul_rn(2.0f, uc), u0));
}
template <int N>
__device__ __forceinline__ void sc_quad(const Geo2& g, const D2Coef& c,
                                        const float* __restrict__ u1,
                                        const float* __restrict__ u0,
                                        const float* __restrict__ c2, int x, int z,
                                        float (&u)[1][4]) {
  using B = res::XWin<N, 4>;
  const long long p = (long long)z * g.ld + x;
  const res::Vec<4> o = ldg4(u0 + p), m = ldg4(c2 + p);
  GWin<N> xw;
  edge_window<N>(g, u1, x, z, xw);
  res::Vec<4> a[2 * N], b[1];
  edge_rows<N>(g, u1, x, z, N, a);  // rows z - N .. z + N - 1
  b[0] = ldg4(u1 + (long long)min(z + N, g.nz - 1) * g.ld + x);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float nb[N];
#pragma unroll
    for (int l = 1; l <= N; ++l)
      nb[l - 1] = __fadd_rn(__fadd_rn(__fadd_rn(xw.w[B::L + j + l], xw.w[B::L + j - l]),
                                      l == N ? b[0][j] : a[l == N ? 0 : N + l][j]),
                            a[N - l][j]);
    const float uc = xw.w[B::L + j];
    const float v = sc_cell<N>(c, uc, o[j], m[j], nb);
    u[0][j] = interior2(g, x + j, z) ? v : uc;
  }
}
template <int N, int R, bool TG>
__global__ void __launch_bounds__(kThreads)
    k_sc_bulk(Geo2 g, Split s, D2Coef c, HabcDev h, const float* __restrict__ u1,
              const float* __restrict__ u0, const float* __restrict__ c2, float* __restrict__ u2,
              CellTags t, int j0) {
  auto tagged = [&](int e, float u) {
    const long long k = (long long)(*t.it0 + j0);
    const int4 E = t.ent[e];
    u = tag_inject(t, E, k, 0, u);
    tag_record(t, E, k, 0, u, 0.0f, 0.0f);
    return u;
  };
  int x, z;
  if ((int)blockIdx.x < s.edge) {
    const int i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= s.quads) return;
    edge_quad(s, i, x, z);
    float u[1][4];
    sc_quad<N>(g, c, u1, u0, c2, x, z, u);
    int sz, ex;
    if (edge_sides(g, x, z, sz, ex)) {
      float v[1][4] = {}, e[1] = {};
      if (sz) sc_quad<N>(g, c, u1, u0, c2, x, z + sz, v);
      if (ex >= 0) e[0] = sc_at<N>(g, c, u1, u0, c2, ex, z);
      edge_blend<1>(g, h, x, z, sz, {2}, u, v, e, {u1});
    }
    const long long p = (long long)z * g.ld + x;
    if constexpr (TG) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (x + j < g.nx) {
          const int e = __ldg(t.tag + p + j);
          if (e >= 0) u[0][j] = tagged(e, u[0][j]);
        }
    }
    edge_store(g, u2 + p, x, u[0]);
    return;
  }
  int rows;
  if (!inner_cells<R>(s, blockIdx.x - s.edge, x, z, rows)) return;
  const long long q = (long long)z * g.ld + x;
  constexpr int NWIN = R + 2 * N;
  res::Vec<4> w[NWIN];
#pragma unroll
  for (int i = 0; i < NWIN; ++i) w[i] = ldg4(u1 + q + (long long)min(i - N, rows - 1 + N) * g.ld);
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (k >= rows) break;
    const long long e = q + (long long)k * g.ld;
    GWin<N> xw;
    xw.load(u1 + e);
    const res::Vec<4> o = lds4(u0 + e), m = lds4(c2 + e);
    float u[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float nb[N];
#pragma unroll
      for (int l = 1; l <= N; ++l)
        nb[l - 1] = __fadd_rn(__fadd_rn(__fadd_rn(xw.w[GWin<N>::L + j + l], xw.w[GWin<N>::L + j - l]),
                                        w[N + k + l][j]),
                              w[N + k - l][j]);
      u[j] = sc_cell<N>(c, w[N + k][j], o[j], m[j], nb);
    }
    if constexpr (TG) {
      const int4 tg = __ldg(reinterpret_cast<const int4*>(t.tag + e));
      if (tg.x >= 0) u[0] = tagged(tg.x, u[0]);
      if (tg.y >= 0) u[1] = tagged(tg.y, u[1]);
      if (tg.z >= 0) u[2] = tagged(tg.z, u[2]);
      if (tg.w >= 0) u[3] = tagged(tg.w, u[3]);
    }
    stg4(u2 + e, u);
  }
}

}  // namespace bulk
}  // namespace fomo
