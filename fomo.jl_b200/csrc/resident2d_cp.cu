// resident2d_cp.cu -- coupled2d time loop with its state on the chip
// (coupled2d/update_fields.jl:27-141, kernels_det.jl:22-57).
#include <type_traits>

#include "resident2d.cuh"

namespace fomo {
namespace res {
namespace {

// Sums of one potential at a block's cells: centered first differences along x and z and
// the Laplacian (one fma per term, as cp_vel_at).
template <int N, int CX, int R>
struct Sums {
  float dx[R][CX], dz[R][CX], lap[R][CX], mid[R][CX];
  __device__ __forceinline__ void load(const float* A, int hb, int pitch, const Centered& c) {
    constexpr int NWIN = R + 2 * N, L = XWin<N, CX>::L;
    Vec<CX> zw[NWIN];
#pragma unroll
    for (int i = 0; i < NWIN; ++i) zw[i] = ldv<CX>(A + hb + (i - N) * pitch);
#pragma unroll
    for (int k = 0; k < R; ++k) {
      XWin<N, CX> xw;
      xw.load(A + hb + k * pitch);
#pragma unroll
      for (int j = 0; j < CX; ++j) {
        const float u = zw[N + k][j];
        float gx = 0.0f, gz = 0.0f, lx = __fmul_rn(c.c0, u), lz = lx;
#pragma unroll
        for (int l = 1; l <= N; ++l) {
          const float c1 = c.d1[l - 1], c2 = c.d2[l - 1];
          const float xp = xw.w[L + j + l], xm = xw.w[L + j - l];
          const float zp = zw[N + k + l][j], zm = zw[N + k - l][j];
          gx = __fmaf_rn(c1, __fsub_rn(xp, xm), gx);
          gz = __fmaf_rn(c1, __fsub_rn(zp, zm), gz);
          lx = __fmaf_rn(c2, __fadd_rn(xp, xm), lx);
          lz = __fmaf_rn(c2, __fadd_rn(zp, zm), lz);
        }
        dx[k][j] = __fmul_rn(gx, c.ih);
        dz[k][j] = __fmul_rn(gz, c.ih);
        lap[k][j] = __fmul_rn(__fadd_rn(lx, lz), c.ih2);
        mid[k][j] = u;
      }
    }
  }
};

// Shared memory (floats): P, S, dP/dt, dS/dt haloed; two arrays of pre-correction values
// and the eight medium planes over the extended tile; weight ramps; word tables.
template <int N, int CX, int R, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
    k_res_cp(const __grid_constant__ Run run, const __grid_constant__ Fields f,
             const __grid_constant__ Centered c) {
  extern __shared__ __align__(16) float sm[];
  const Geom& g = run.g;
  Work<N, CX, R> w(run, false);
  const int hn = g.rows * w.pitch, en = g.ngr * R * w.ep;
  float* P = sm;
  float* S = P + hn;
  float* DP = S + hn;
  float* DS = DP + hn;
  float* U0 = DS + hn;
  float* U1 = U0 + en;
  float* ME = U1 + en;  // alpha, beta, their x and z derivatives, Laplacians
  float* wt = ME + (g.gmat ? 0 : 8 * en);
  for (int i = 0; i < 4; ++i) w.load(run, P + i * hn, f.in[i]);
  if (!g.gmat)
    for (int i = 0; i < 8; ++i) w.load_ext(run, ME + i * en, f.mat[i]);
  for (int i = threadIdx.x; i < 3 * run.h.wstride; i += blockDim.x) wt[i] = __ldg(run.h.wtab + i);
  // halo regions: dP/dt and dS/dt in the ring, P and S along x and z
  const Region rv[4] = {{kRows, 0, 0, 2}, {kCols, 0, 0, 2}, {kRows, 0, 0, 3}, {kCols, 0, 0, 3}};
  const Region rp[4] = {{kStrip, N + 1, N + 1, 0}, {kBand, N + 1, N + 1, 0},
                        {kStrip, N + 1, N + 1, 1}, {kBand, N + 1, N + 1, 1}};
  Word* tvg = reinterpret_cast<Word*>(sm + g.words);
  const int nvg = w.get_words(run, tvg, rv, 4, hn, g.per);
  Word* tpg = tvg + nvg;
  const int npg = w.get_words(run, tpg, rp, 4, hn, g.per);
  int* tvp = reinterpret_cast<int*>(tpg + npg);
  const int nvp = w.put_words(tvp, rv, 4, hn);
  int* tpp = tvp + nvp;
  const int npp = w.put_words(tpp, rp, 4, hn);
  const bool blend = __syncthreads_or(w.cl.frame != 0);
  for (int step = 0; step < run.nsteps; ++step) {
    const int it = run.it0 + step;
    w.refresh();
    const int hb = w.hb, pitch = w.pitch;
    uint64_t* l0 = run.ll + (long long)(it & 1) * 2 * gridDim.x * g.per;
    uint64_t* l1 = l0 + (long long)gridDim.x * g.per;
    const long long part = (long long)blockIdx.x * g.per;
    const uint32_t ev = 2u * (uint32_t)it - 1u, ep2 = 2u * (uint32_t)it;
    // ---- dP/dt, dS/dt ----
    float uP[R][CX], uS[R][CX];
    if (w.t.act) {
      Sums<N, CX, R> p, s;
      p.load(P, hb, pitch, c);
      s.load(S, hb, pitch, c);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const Vec<CX> oP = ldv<CX>(DP + hb + k * pitch), oS = ldv<CX>(DS + hb + k * pitch);
        auto med = [&](int i) { return w.mat(run, ME + i * en, f.mat[i], k); };
        const Vec<CX> a = med(0), b = med(1), ax = med(2), az = med(3), bx = med(4), bz = med(5),
                      la = med(6), lb = med(7);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          const float Pc = p.mid[k][j];
          float r = __fmul_rn(Pc, la[j]);
          r = __fmaf_rn(2.0f, __fmaf_rn(ax[j], p.dx[k][j], __fmul_rn(az[j], p.dz[k][j])), r);
          r = __fmaf_rn(__fmul_rn(-2.0f, Pc), lb[j], r);
          r = __fmaf_rn(2.0f, __fmaf_rn(bx[j], s.dz[k][j], -__fmul_rn(bz[j], s.dx[k][j])), r);
          r = __fmaf_rn(a[j], p.lap[k][j], r);
          float q = __fmul_rn(2.0f, __fmaf_rn(bx[j], s.dx[k][j], __fmul_rn(bz[j], s.dz[k][j])));
          q = __fmaf_rn(2.0f, __fmaf_rn(bz[j], p.dx[k][j], -__fmul_rn(bx[j], p.dz[k][j])), q);
          q = __fmaf_rn(b[j], s.lap[k][j], q);
          const bool in = w.inner(k, j);
          uP[k][j] = in ? __fmaf_rn(c.dt, r, oP[j]) : oP[j];
          uS[k][j] = in ? __fmaf_rn(c.dt, q, oS[j]) : oS[j];
        }
      }
      if (blend) {
        w.stage(U0, uP);
        w.stage(U1, uS);
      }
    }
    if (blend) w.template blend<2>(run, wt, {0, 0}, {uP, uS}, {U0, U1}, {DP, DS}, &c.hs);
    w.keep(DP, uP);
    w.keep(DS, uS);
    __syncthreads();
    words_put(tvp, nvp, l0 + part, sm, ev);
    words_get<2>(tvg, nvg, l0, sm, ev, w.live, run.err);
    __syncthreads();
    // ---- P, S, injection, recording ----
    if (w.t.act) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const int q = hb + k * pitch;
        const Vec<CX> oP = ldv<CX>(P + q), oS = ldv<CX>(S + q), vP = ldv<CX>(DP + q),
                      vS = ldv<CX>(DS + q);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          const bool in = w.inner(k, j);
          uP[k][j] = in ? __fmaf_rn(c.dt, vP[j], oP[j]) : oP[j];
          uS[k][j] = in ? __fmaf_rn(c.dt, vS[j], oS[j]) : oS[j];
        }
      }
      if (blend) {
        w.stage(U0, uP);
        w.stage(U1, uS);
      }
    }
    if (blend) w.template blend<2>(run, wt, {2, 2}, {uP, uS}, {U0, U1}, {P, S}, &c.hs);
    w.keep(P, uP);
    w.keep(S, uS);
    for (int e = w.t.e0; e < w.t.e1; ++e) {
      const int cell = run.E.key[e].y, q = hb + (cell / CX) * pitch + cell % CX;
      const int4 E = run.E.tags.ent[run.E.ent[e]];
      const float u = tag_inject(run.E.tags, E, it - 1, 0, P[q]);
      P[q] = u;
      tag_record(run.E.tags, E, it - 1, 0, u, S[q], 0.0f);
#pragma unroll
      for (int k = 0; k < R; ++k)
#pragma unroll
        for (int j = 0; j < CX; ++j)
          if (cell == k * CX + j) uP[k][j] = u;
    }
    if (run.snap_interval && it % run.snap_interval == 0) {
      w.snapshot(run, run.snaps, it, uP);
      w.snapshot(run, c.snaps_s, it, uS);
    }
    __syncthreads();
    words_put(tpp, npp, l1 + part, sm, ep2);
    words_get<3>(tpg, npg, l1, sm, ep2, w.live, run.err);
    __syncthreads();
  }
  for (int i = 0; i < 4; ++i) w.store(run, P + i * hn, f.out[i]);
}

}  // namespace

cudaError_t launch_coupled(cudaStream_t st, int N, const Plan& p, const Run& run, const Fields& f,
                           const Centered& c) {
#define FOMO_RES_F(I, CX, R, T) \
  case I: return launch_resident(st, k_res_cp<NN, CX, R, T>, p, run, f, c);
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
