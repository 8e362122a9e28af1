// resident2d_ac.cu -- acoustic2d time loop with its state on the chip
// (acoustic2d/fused_kernels.jl:27-114, kernels_det.jl:22-57, sponge.jl:30-78).
#include <type_traits>

#include "resident2d.cuh"

namespace fomo {
namespace res {
namespace {

// Shared memory (floats): vx, vz, p haloed; two arrays of pre-correction values over
// the extended tile; bx dt/dh, bz dt/dh, kappa too where R > 2 (else in registers);
// weight ramps; word tables.
template <int N, int CX, int R, int THREADS, bool SP>
__global__ void __launch_bounds__(THREADS, 1)
    k_res_ac(const __grid_constant__ Run run, const __grid_constant__ Fields f) {
  constexpr int NWIN = R + 2 * N - 1;
  constexpr bool MREG = CX * R <= kAcousticNeeds.mreg;
  extern __shared__ __align__(16) float sm[];
  const Geom& g = run.g;
  const Coef& c = run.c;
  Work<N, CX, R> w(run, SP);
  const int hn = g.rows * w.pitch, en = g.ngr * R * w.ep;
  float* VX = sm;
  float* VZ = VX + hn;
  float* P = VZ + hn;
  float* U0 = P + hn;
  float* U1 = U0 + en;
  float* ME = U1 + en;
  float* wt = ME + (MREG || g.gmat ? 0 : 3 * en);
  const long long so = (long long)w.t.shot * g.plane;
  w.load(run, P, f.in[2] ? f.in[2] + so : nullptr);
  w.load(run, VX, f.in[0] ? f.in[0] + so : nullptr);
  w.load(run, VZ, f.in[1] ? f.in[1] + so : nullptr);
  float mr[MREG ? 3 : 1][R][CX];
  if constexpr (MREG) {
#pragma unroll
    for (int i = 0; i < 3; ++i) w.load_own(run, mr[i], f.mat[i]);
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int j = 0; j < CX; ++j) {  // bx dtx, bz dtz: rounded once, as in every step
        mr[0][k][j] = __fmul_rn(mr[0][k][j], run.dtx);
        mr[1][k][j] = __fmul_rn(mr[1][k][j], run.dtz);
      }
  } else if (!g.gmat) {
    for (int i = 0; i < 3; ++i) w.load_ext(run, ME + i * en, f.mat[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < en; i += blockDim.x) {
      ME[i] = __fmul_rn(ME[i], run.dtx);
      ME[en + i] = __fmul_rn(ME[en + i], run.dtz);
    }
  }
  auto mat = [&](int i, int k) {
    if constexpr (MREG) {
      Vec<CX> v;
#pragma unroll
      for (int j = 0; j < CX; ++j) v.v[j] = mr[i][k][j];
      return v;
    } else {
      Vec<CX> v = w.mat(run, ME + i * en, f.mat[i], k);
      if (i < 2 && g.gmat) {
#pragma unroll
        for (int j = 0; j < CX; ++j) v.v[j] = __fmul_rn(v.v[j], i ? run.dtz : run.dtx);
      }
      return v;
    }
  };
  const int nwt = SP ? run.h.nbc : 3 * run.h.wstride;
  for (int i = threadIdx.x; i < nwt; i += blockDim.x) wt[i] = __ldg(run.h.wtab + i);
  // halo regions: vx is read along x (N columns left, N + 1 right) and in the ring, vz
  // along z, p along both
  const Region rv[4] = {
      {kStrip, N, N + 1, 0}, {kRows, 0, 0, 0}, {kBand, N + 1, N, 1}, {kCols, 0, 0, 1}};
  const Region rq[2] = {{kStrip, N + 1, N, 2}, {kBand, N, N + 1, 2}};
  Word* tvg = reinterpret_cast<Word*>(sm + g.words);
  const int nvg = w.get_words(run, tvg, rv, 4, hn, g.per);
  Word* tpg = tvg + nvg;
  const int npg = w.get_words(run, tpg, rq, 2, hn, g.per);
  int* tvp = reinterpret_cast<int*>(tpg + npg);
  const int nvp = w.put_words(tvp, rv, 4, hn);
  int* tpp = tvp + nvp;
  const int npp = w.put_words(tpp, rq, 2, hn);
  const bool blend = __syncthreads_or(w.cl.frame != 0);
  for (int step = 0; step < run.nsteps; ++step) {
    const int it = run.it0 + step;
    w.refresh();
    const int hb = w.hb, pitch = w.pitch;
    // this step's buffers of the two half steps, and this tile's parts
    uint64_t* l0 = run.ll + (long long)(it & 1) * 2 * gridDim.x * g.per;
    uint64_t* l1 = l0 + (long long)gridDim.x * g.per;
    const long long part = (long long)blockIdx.x * g.per;
    const uint32_t ev = 2u * (uint32_t)it - 1u, eq = 2u * (uint32_t)it;
    // ---- velocity ----
    float ux[R][CX], uz[R][CX];
    if (w.t.act) {
      Vec<CX> pw[NWIN];  // p rows z - (N - 1) ..
#pragma unroll
      for (int i = 0; i < NWIN; ++i) pw[i] = ldv<CX>(P + hb + (i - (N - 1)) * pitch);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        XWin<N, CX> xw;
        xw.load(P + hb + k * pitch);
        const Vec<CX> ox = ldv<CX>(VX + hb + k * pitch), oz = ldv<CX>(VZ + hb + k * pitch);
        const Vec<CX> bx = mat(0, k), bz = mat(1, k);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          const bool in = w.inner(k, j);
          const float dx = xw.dm(j, c), dz = zdp<N, CX>(pw, N - 1 + k, j, c);
          ux[k][j] = in ? __fmaf_rn(bx[j], dx, ox[j]) : ox[j];
          uz[k][j] = in ? __fmaf_rn(bz[j], dz, oz[j]) : oz[j];
          if constexpr (SP) {
            ux[k][j] = w.damp(run, wt, k, j, ux[k][j]);
            uz[k][j] = w.damp(run, wt, k, j, uz[k][j]);
          }
        }
      }
      if (blend) {
        w.stage(U0, ux);
        w.stage(U1, uz);
      }
    }
    if (blend) w.template blend<2>(run, wt, {0, 1}, {ux, uz}, {U0, U1}, {VX, VZ});
    w.keep(VX, ux);
    w.keep(VZ, uz);
    __syncthreads();
    words_put(tvp, nvp, l0 + part, sm, ev);
    words_get<3>(tvg, nvg, l0, sm, ev, w.live, run.err);
    __syncthreads();
    // ---- pressure, injection, recording ----
    if (w.t.act) {
      Vec<CX> vw[NWIN];  // vz rows z - N ..
#pragma unroll
      for (int i = 0; i < NWIN; ++i) vw[i] = ldv<CX>(VZ + hb + (i - N) * pitch);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        XWin<N, CX> xw;
        xw.load(VX + hb + k * pitch);
        const Vec<CX> op = ldv<CX>(P + hb + k * pitch), ka = mat(2, k);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          const float dx = xw.dp(j, c), dz = zdm<N, CX>(vw, N + k, j, c);
          const float u = __fmaf_rn(ka[j], __fmaf_rn(dx, run.dtx, __fmul_rn(dz, run.dtz)),
                                    op[j]);
          ux[k][j] = w.inner(k, j) ? u : op[j];
          if constexpr (SP) ux[k][j] = w.damp(run, wt, k, j, ux[k][j]);
        }
      }
      if (blend) w.stage(U0, ux);
    }
    if (blend) w.template blend<1>(run, wt, {2}, {ux}, {U0}, {P});
    w.keep(P, ux);
    for (int e = w.t.e0; e < w.t.e1; ++e) {
      const int cell = run.E.key[e].y, q = hb + (cell / CX) * pitch + cell % CX;
      const int4 E = run.E.tags.ent[run.E.ent[e]];
      const float u = tag_inject(run.E.tags, E, it - 1, w.t.shot, P[q]);
      P[q] = u;
      tag_record(run.E.tags, E, it - 1, w.t.shot, u, VX[q], VZ[q]);
#pragma unroll
      for (int k = 0; k < R; ++k)
#pragma unroll
        for (int j = 0; j < CX; ++j)
          if (cell == k * CX + j) ux[k][j] = u;
    }
    if (run.snap_interval && it % run.snap_interval == 0) w.snapshot(run, run.snaps, it, ux);
    __syncthreads();
    words_put(tpp, npp, l1 + part, sm, eq);
    words_get<3>(tpg, npg, l1, sm, eq, w.live, run.err);
    __syncthreads();
  }
  w.store(run, VX, f.out[0] + so);
  w.store(run, VZ, f.out[1] + so);
  w.store(run, P, f.out[2] + so);
}

}  // namespace

cudaError_t launch_acoustic(cudaStream_t st, int N, bool sponge, const Plan& p, const Run& run,
                            const Fields& f) {
#define FOMO_RES_F(I, CX, R, T)                                                          \
  case I:                                                                               \
    return sponge ? launch_resident(st, k_res_ac<NN, CX, R, T, true>, p, run, f)         \
                  : launch_resident(st, k_res_ac<NN, CX, R, T, false>, p, run, f);
  auto go = [&](auto n) -> cudaError_t {
    constexpr int NN = decltype(n)::value;
    switch (p.form) { FOMO_RES_FORMS(FOMO_RES_F) }
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
