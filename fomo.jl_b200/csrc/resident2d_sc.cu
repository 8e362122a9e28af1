// resident2d_sc.cu -- scalar2d time loop with its state on the chip
// (scalar2d/scalar2d.jl:29-84, kernels_det.jl:22-57).
#include <type_traits>

#include "resident2d.cuh"

namespace fomo {
namespace res {
namespace {

// Shared memory (floats): u^n haloed; pre-correction values over the extended tile; c2
// too where blocks are large (else in registers); weight ramps; word tables.  u^{n-1}
// is read at the cell itself only and lives in registers, the ring's too (the u^n that the
// previous step read).
template <int N, int CX, int R, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
    k_res_sc(const __grid_constant__ Run run, const __grid_constant__ Fields f,
             const __grid_constant__ Centered c) {
  constexpr bool MREG = CX * R <= kScalarNeeds.mreg;
  constexpr int NWIN = R + 2 * N;
  extern __shared__ __align__(16) float sm[];
  const Geom& g = run.g;
  Work<N, CX, R> w(run, false);
  const int hn = g.rows * w.pitch, en = g.ngr * R * w.ep;
  float* A = sm;
  float* U = A + hn;
  float* ME = U + en;
  float* wt = ME + (MREG || g.gmat ? 0 : en);
  w.load(run, A, f.in[0]);
  float mr[R][CX], u0[R][CX];
  if constexpr (MREG) w.load_own(run, mr, f.mat[0]);
  else if (!g.gmat) w.load_ext(run, ME, f.mat[0]);
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int j = 0; j < CX; ++j) u0[k][j] = 0.0f;
  if (f.in[1]) w.load_own(run, u0, f.in[1]);
  const int nwt = 3 * run.h.wstride;
  for (int i = threadIdx.x; i < nwt; i += blockDim.x) wt[i] = __ldg(run.h.wtab + i);
  const Region rg[2] = {{kStrip, N + 1, N + 1, 0}, {kBand, N + 1, N + 1, 0}};
  Word* tg = reinterpret_cast<Word*>(sm + g.words);
  const int ng = w.get_words(run, tg, rg, 2, hn, g.per);
  int* tp = reinterpret_cast<int*>(tg + ng);
  const int np = w.put_words(tp, rg, 2, hn);
  const bool blend = __syncthreads_or(w.cl.frame != 0);
  for (int step = 0; step < run.nsteps; ++step) {
    const int it = run.it0 + step;
    w.refresh();
    const int hb = w.hb, pitch = w.pitch;
    uint64_t* ll = run.ll + (long long)(it & 1) * gridDim.x * g.per;
    float u[R][CX];
    if (w.t.act) {
      Vec<CX> zw[NWIN];  // rows z - N ..
#pragma unroll
      for (int i = 0; i < NWIN; ++i) zw[i] = ldv<CX>(A + hb + (i - N) * pitch);
#pragma unroll
      for (int k = 0; k < R; ++k) {
        XWin<N, CX> xw;
        xw.load(A + hb + k * pitch);
        Vec<CX> c2;
        if constexpr (!MREG) c2 = w.mat(run, ME, f.mat[0], k);
#pragma unroll
        for (int j = 0; j < CX; ++j) {
          constexpr int L = XWin<N, CX>::L;
          const float uc = zw[N + k][j];
          float lap = __fmul_rn(c.c0, uc);
#pragma unroll
          for (int l = 1; l <= N; ++l) {
            const float nb = __fadd_rn(__fadd_rn(__fadd_rn(xw.w[L + j + l], xw.w[L + j - l]),
                                                 zw[N + k + l][j]),
                                       zw[N + k - l][j]);
            lap = __fmaf_rn(c.d2[l - 1], nb, lap);
          }
          const float v = __fmaf_rn(MREG ? mr[k][j] : c2[j], lap, __fsub_rn(__fmul_rn(2.0f, uc), u0[k][j]));
          u[k][j] = w.inner(k, j) ? v : uc;
          u0[k][j] = uc;
        }
      }
      if (blend) w.stage(U, u);
    }
    if (blend) w.template blend<1>(run, wt, {2}, {u}, {U}, {A});
    else __syncthreads();  // every block has read its windows of u^n
    w.keep(A, u);
    for (int e = w.t.e0; e < w.t.e1; ++e) {
      const int cell = run.E.key[e].y, q = hb + (cell / CX) * pitch + cell % CX;
      const int4 E = run.E.tags.ent[run.E.ent[e]];
      const float v = tag_inject(run.E.tags, E, it - 1, 0, A[q]);
      A[q] = v;
      tag_record(run.E.tags, E, it - 1, 0, v, 0.0f, 0.0f);
    }
    __syncthreads();
    words_put(tp, np, ll + (long long)blockIdx.x * g.per, sm, (uint32_t)it);
    words_get<3>(tg, ng, ll, sm, (uint32_t)it, w.live, run.err);
    __syncthreads();
  }
  // u^n from shared memory, u^{n-1} from the registers
  w.store(run, A, f.out[0]);
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int j = 0; j < CX; ++j)
      if (w.cl.own >> (k * CX + j) & 1)
        f.out[1][(long long)(w.cl.z + k) * g.ld + w.cl.x + j] = u0[k][j];
}

}  // namespace

cudaError_t launch_scalar(cudaStream_t st, int N, const Plan& p, const Run& run, const Fields& f,
                          const Centered& c) {
#define FOMO_RES_F(I, CX, R, T) \
  case I: return launch_resident(st, k_res_sc<NN, CX, R, T>, p, run, f, c);
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
