// resident2d_el.cu -- elastic2d time loop with its state on the chip
// (elastic2d/fused_kernels.jl:21-124, kernels_det.jl:22-57, sponge.jl:30-78).
#include <type_traits>

#include "resident2d.cuh"

namespace fomo {
namespace res {
namespace {

// Shared memory (floats): vx, vz, txx, tzz, txz haloed; the five materials and the
// three arrays of pre-correction values over the extended tile; weight
// ramps; word tables.
template <int N, int CX, int R, int THREADS, bool SP>
__global__ void __launch_bounds__(THREADS, 1)
    k_res_el(const __grid_constant__ Run run, const __grid_constant__ Fields f) {
  constexpr int NWIN = R + 2 * N - 1;
  extern __shared__ __align__(16) float sm[];
  const Geom& g = run.g;
  const Coef& c = run.c;
  Work<N, CX, R> w(run, SP);
  const int hn = g.rows * w.pitch, en = g.ngr * R * w.ep;
  float* VX = sm;
  float* VZ = VX + hn;
  float* XX = VZ + hn;
  float* ZZ = XX + hn;
  float* XZ = ZZ + hn;
  float* M = XZ + hn;  // bx, bz, lam, l2m, mut
  float* U = M + (g.gmat ? 0 : 5 * en);
  float* wt = U + 3 * en;
  const long long so = (long long)w.t.shot * g.plane;
#pragma unroll
  for (int i = 0; i < 5; ++i) w.load(run, VX + i * hn, f.in[i] ? f.in[i] + so : nullptr);
  if (!g.gmat)
    for (int i = 0; i < 5; ++i) w.load_ext(run, M + i * en, f.mat[i]);
  const int nwt = SP ? run.h.nbc : 3 * run.h.wstride;
  for (int i = threadIdx.x; i < nwt; i += blockDim.x) wt[i] = __ldg(run.h.wtab + i);
  // halo regions: vx, vz and txz are read along x and z, txx along x and tzz along z (and
  // in the ring)
  const Region rv[4] = {{kStrip, N, N + 1, 0}, {kBand, N, N + 1, 0}, {kStrip, N + 1, N, 1},
                        {kBand, N + 1, N, 1}};
  const Region rs[6] = {{kStrip, N + 1, N, 2}, {kRows, 0, 0, 2},      {kBand, N, N + 1, 3},
                        {kCols, 0, 0, 3},      {kStrip, N, N + 1, 4}, {kBand, N + 1, N, 4}};
  Word* tvg = reinterpret_cast<Word*>(sm + g.words);
  const int nvg = w.get_words(run, tvg, rv, 4, hn, g.per);
  Word* tsg = tvg + nvg;
  const int nsg = w.get_words(run, tsg, rs, 6, hn, g.per);
  int* tvp = reinterpret_cast<int*>(tsg + nsg);
  const int nvp = w.put_words(tvp, rv, 4, hn);
  int* tsp = tvp + nvp;
  const int nsp = w.put_words(tsp, rs, 6, hn);
  const bool blend = __syncthreads_or(w.cl.frame != 0);
  for (int step = 0; step < run.nsteps; ++step) {
    const int it = run.it0 + step;
    w.refresh();
    const int hb = w.hb, pitch = w.pitch;
    // this step's buffers of the two half steps, and this tile's parts
    uint64_t* l0 = run.ll + (long long)(it & 1) * 2 * gridDim.x * g.per;
    uint64_t* l1 = l0 + (long long)gridDim.x * g.per;
    const long long part = (long long)blockIdx.x * g.per;
    const uint32_t ev = 2u * (uint32_t)it - 1u, es = 2u * (uint32_t)it;
    // ---- velocity ----
    {
      float ux[R][CX], uz[R][CX];
      if (w.t.act) {
        {
          // z sums first: one register window at a time
          Vec<CX> r[NWIN];
#pragma unroll
          for (int i = 0; i < NWIN; ++i) r[i] = ldv<CX>(XZ + hb + (i - N) * pitch);
#pragma unroll
          for (int k = 0; k < R; ++k)
#pragma unroll
            for (int j = 0; j < CX; ++j) ux[k][j] = __fmul_rn(run.dtz, zdm<N, CX>(r, N + k, j, c));
#pragma unroll
          for (int i = 0; i < NWIN; ++i) r[i] = ldv<CX>(ZZ + hb + (i - (N - 1)) * pitch);
#pragma unroll
          for (int k = 0; k < R; ++k)
#pragma unroll
            for (int j = 0; j < CX; ++j) uz[k][j] = __fmul_rn(run.dtz, zdp<N, CX>(r, N - 1 + k, j, c));
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
          XWin<N, CX> xw;
          const int h = hb + k * pitch;
          xw.load(XX + h);
          const Vec<CX> ox = ldv<CX>(VX + h), bx = w.mat(run, M, f.mat[0], k);
#pragma unroll
          for (int j = 0; j < CX; ++j) {
            const float u = __fmaf_rn(bx[j], __fmaf_rn(run.dtx, xw.dm(j, c), ux[k][j]),
                                      ox[j]);
            ux[k][j] = w.inner(k, j) ? u : ox[j];
            if constexpr (SP) ux[k][j] = w.damp(run, wt, k, j, ux[k][j]);
          }
          xw.load(XZ + h);
          const Vec<CX> oz = ldv<CX>(VZ + h), bz = w.mat(run, M + en, f.mat[1], k);
#pragma unroll
          for (int j = 0; j < CX; ++j) {
            const float u = __fmaf_rn(bz[j], __fmaf_rn(run.dtx, xw.dp(j, c), uz[k][j]),
                                      oz[j]);
            uz[k][j] = w.inner(k, j) ? u : oz[j];
            if constexpr (SP) uz[k][j] = w.damp(run, wt, k, j, uz[k][j]);
          }
        }
        if (blend) {
          w.stage(U, ux);
          w.stage(U + en, uz);
        }
      }
      if (blend) w.template blend<2>(run, wt, {0, 1}, {ux, uz}, {U, U + en}, {VX, VZ});
      w.keep(VX, ux);
      w.keep(VZ, uz);
    }
    __syncthreads();
    words_put(tvp, nvp, l0 + part, sm, ev);
    words_get<4>(tvg, nvg, l0, sm, ev, w.live, run.err);
    __syncthreads();
    // ---- stress, injection, recording ----
    float sx[R][CX], sz[R][CX], sq[R][CX];
    if (w.t.act) {
      {
        Vec<CX> r[NWIN];
#pragma unroll
        for (int i = 0; i < NWIN; ++i) r[i] = ldv<CX>(VZ + hb + (i - N) * pitch);
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
          for (int j = 0; j < CX; ++j) sz[k][j] = __fmul_rn(zdm<N, CX>(r, N + k, j, c), run.dtz);  // ez
#pragma unroll
        for (int i = 0; i < NWIN; ++i) r[i] = ldv<CX>(VX + hb + (i - (N - 1)) * pitch);
#pragma unroll
        for (int k = 0; k < R; ++k)
#pragma unroll
          for (int j = 0; j < CX; ++j) sq[k][j] = zdp<N, CX>(r, N - 1 + k, j, c);  // dvx/dz
      }
#pragma unroll
      for (int k = 0; k < R; ++k) {
        XWin<N, CX> xw;
        const int h = hb + k * pitch;
        xw.load(VX + h);
        const Vec<CX> oxx = ldv<CX>(XX + h), ozz = ldv<CX>(ZZ + h);
        const Vec<CX> la = w.mat(run, M + 2 * en, f.mat[2], k), l2 = w.mat(run, M + 3 * en, f.mat[3], k);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          const float ex = __fmul_rn(xw.dp(j, c), run.dtx), ez = sz[k][j];
          const float lam = la[j], l2m = l2[j];
          const float a = __fadd_rn(oxx[j], __fmaf_rn(l2m, ex, __fmul_rn(lam, ez)));
          const float b = __fadd_rn(ozz[j], __fmaf_rn(lam, ex, __fmul_rn(l2m, ez)));
          const bool in = w.inner(k, j);
          sx[k][j] = in ? a : oxx[j];
          sz[k][j] = in ? b : ozz[j];
          if constexpr (SP) {
            sx[k][j] = w.damp(run, wt, k, j, sx[k][j]);
            sz[k][j] = w.damp(run, wt, k, j, sz[k][j]);
          }
        }
        xw.load(VZ + h);
        const Vec<CX> oxz = ldv<CX>(XZ + h), mu = w.mat(run, M + 4 * en, f.mat[4], k);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          const float u = __fmaf_rn(mu[j],
                                    __fmaf_rn(sq[k][j], run.dtz,
                                              __fmul_rn(xw.dm(j, c), run.dtx)),
                                    oxz[j]);
          sq[k][j] = w.inner(k, j) ? u : oxz[j];
          if constexpr (SP) sq[k][j] = w.damp(run, wt, k, j, sq[k][j]);
        }
      }
      if (blend) {
        w.stage(U, sx);
        w.stage(U + en, sz);
        w.stage(U + 2 * en, sq);
      }
    }
    if (blend)
      w.template blend<3>(run, wt, {2, 2, 2}, {sx, sz, sq}, {U, U + en, U + 2 * en}, {XX, ZZ, XZ});
    w.keep(XX, sx);
    w.keep(ZZ, sz);
    w.keep(XZ, sq);
    for (int e = w.t.e0; e < w.t.e1; ++e) {
      const int cell = run.E.key[e].y, q = hb + (cell / CX) * pitch + cell % CX;
      const int4 E = run.E.tags.ent[run.E.ent[e]];
      const float a = tag_inject(run.E.tags, E, it - 1, w.t.shot, XX[q]);
      const float b = tag_inject(run.E.tags, E, it - 1, w.t.shot, ZZ[q]);
      XX[q] = a;
      ZZ[q] = b;
      tag_record(run.E.tags, E, it - 1, w.t.shot, VX[q], VZ[q], 0.0f);
#pragma unroll
      for (int k = 0; k < R; ++k)
#pragma unroll
        for (int j = 0; j < CX; ++j)
          if (cell == k * CX + j) {
            sx[k][j] = a;
            sz[k][j] = b;
          }
    }
    if (run.snap_interval && it % run.snap_interval == 0) {
      float v[R][CX];
#pragma unroll
      for (int k = 0; k < R; ++k)
#pragma unroll
        for (int j = 0; j < CX; ++j) v[k][j] = w.t.act ? VZ[hb + k * pitch + j] : 0.0f;
      w.snapshot(run, run.snaps, it, v);
    }
    __syncthreads();
    words_put(tsp, nsp, l1 + part, sm, es);
    words_get<4>(tsg, nsg, l1, sm, es, w.live, run.err);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 5; ++i) w.store(run, VX + i * hn, f.out[i] + so);
}

}  // namespace

cudaError_t launch_elastic(cudaStream_t st, int N, bool sponge, const Plan& p, const Run& run,
                           const Fields& f) {
#define FOMO_RES_F(I, CX, R, T)                                                          \
  case I:                                                                               \
    return sponge ? launch_resident(st, k_res_el<NN, CX, R, T, true>, p, run, f)         \
                  : launch_resident(st, k_res_el<NN, CX, R, T, false>, p, run, f);
  auto go = [&](auto n) -> cudaError_t {
    constexpr int NN = decltype(n)::value;
    switch (p.form) { FOMO_RES_FORMS3(FOMO_RES_F) }
    return cudaErrorInvalidValue;
  };
#undef FOMO_RES_F
  switch (N) {
    case 1: return go(std::integral_constant<int, 1>{});
    case 2: return go(std::integral_constant<int, 2>{});
    case 3: return go(std::integral_constant<int, 3>{});
    case 4: return go(std::integral_constant<int, 4>{});
    case 5: return go(std::integral_constant<int, 5>{});
  }
  return cudaErrorInvalidValue;
}

}  // namespace res
}  // namespace fomo
