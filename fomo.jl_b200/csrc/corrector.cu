// corrector.cu -- learned per-step dispersion corrector for coarse-grid runs
// (no reference counterpart).
//
// Network: three 3x3 convolutions, bias-free, ReLU between them:
//   features (6 channels) -> 16 -> 16 -> 1, the features being
//   u^n, u^{n-1}, c2 u^n, c2^2 u^n, and at the source cells the values
//   injected in this step and in the previous one (0 elsewhere).
// Every input channel is linear in the wave's amplitude and the network has
// no bias, so the correction is positively homogeneous: it scales with the
// amplitude and needs no normalisation.  The correction is added to u^{n+1}
// after the coarse scalar step and the source injection.
//
// Tensor-core path: activations are BF16 in NHWC with 16 channels (32 bytes a
// pixel), weights BF16, accumulation FP32, via mma.sync m16n8k16 implicit
// GEMMs: a warp takes 16 consecutive pixels of a row (M), one conv tap's 16
// input channels per k-step (K = 16, 9 taps), 8 output channels per n-tile.
//   forward            Y[p, co]   = sum_tap sum_ci X[p + tap, ci] W[tap, ci, co]
//   backward (data)    dX[p, ci]  = sum_tap sum_co dY[p - tap, co] W[tap, ci, co]
//                                 = the forward kernel on flipped, transposed weights
//   backward (weights) dW[tap, ci, co] = sum_p X[p + tap, ci] dY[p, co]
//                        (M = ci, N = co, K = pixels; per-block partials reduced
//                         in block order, so gradients are deterministic)
// Parameters are FP32 masters: W1[9][6][16], W2[9][16][16], W3[9][16] (co = 1).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "fomo_internal.cuh"

namespace fomo {
namespace {

constexpr int kC = 16;                       // channel stride of every activation
constexpr int kCin = 6;                      // feature channels
constexpr int kNW1 = 9 * kCin * 16;          // 864
constexpr int kNW2 = 9 * 16 * 16;            // 2304
constexpr int kNW3 = 9 * 16;                 // 144
constexpr int kNParam = kNW1 + kNW2 + kNW3;  // 3312
// packed B fragments, [tap][ntile][lane][2] uint32 each
constexpr int kF16 = 9 * 2 * 64;  // 16 output channels (2 n-tiles)
constexpr int kF8 = 9 * 1 * 64;   // 1 output channel (1 n-tile, 7 zero columns)
constexpr int kOffF1 = 0, kOffF2 = kOffF1 + kF16, kOffF3 = kOffF2 + kF16;
constexpr int kOffT3 = kOffF3 + kF8, kOffT2 = kOffT3 + kF16;
constexpr int kNFrag = kOffT2 + kF16;

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) |
         ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16);
}
__device__ __forceinline__ float bf(uint16_t u) { return __bfloat162float(__ushort_as_bfloat16(u)); }

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// W[tap][ci][co] of a layer with ci_n x co_n channels (zero outside)
__device__ __forceinline__ float wat(const float* W, int ci_n, int co_n, int tap, int ci, int co) {
  return (ci < ci_n && co < co_n) ? W[(tap * ci_n + ci) * co_n + co] : 0.0f;
}

// B fragment of m16n8k16 (k x n): reg0 = (k = 2t, 2t+1; n = g), reg1 = (k = 2t+8, 2t+9; n = g)
// with t = lane & 3, g = lane >> 2.  Forward: B[k = ci][n = co] of tap.
// Transposed (backward data): tap' = 8 - tap, B[k = co][n = ci].
__global__ void k_pack(const float* __restrict__ P, uint32_t* __restrict__ F) {
  const float* W1 = P;
  const float* W2 = P + kNW1;
  const float* W3 = P + kNW1 + kNW2;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNFrag / 2; i += gridDim.x * blockDim.x) {
    int part, base;
    if (i < kOffF2 / 2) { part = 0; base = kOffF1 / 2; }
    else if (i < kOffF3 / 2) { part = 1; base = kOffF2 / 2; }
    else if (i < kOffT3 / 2) { part = 2; base = kOffF3 / 2; }
    else if (i < kOffT2 / 2) { part = 3; base = kOffT3 / 2; }
    else { part = 4; base = kOffT2 / 2; }
    const int nt_n = part == 2 ? 1 : 2;
    int r = i - base;
    const int lane = r & 31;
    r >>= 5;
    const int nt = r % nt_n, tap = r / nt_n;
    const int t = lane & 3, g = lane >> 2, n = nt * 8 + g;
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = 2 * t + (e & 1) + (e >> 1) * 8;
      switch (part) {
        case 0: v[e] = wat(W1, kCin, 16, tap, k, n); break;
        case 1: v[e] = wat(W2, 16, 16, tap, k, n); break;
        case 2: v[e] = wat(W3, 16, 1, tap, k, n); break;
        case 3: v[e] = wat(W3, 16, 1, 8 - tap, n, k); break;   // dY3 (1 ch) -> dH2 (16 ch)
        default: v[e] = wat(W2, 16, 16, 8 - tap, n, k); break;  // dPre2 -> dH1
      }
    }
    F[2 * i] = pack2(v[0], v[1]);
    F[2 * i + 1] = pack2(v[2], v[3]);
  }
}

// Tile storage of 32-byte pixels in shared memory: the two 16-byte channel halves of pixel
// column j change places every four pixels, so the eight rows of an ldmatrix (eight
// neighbouring pixels) fall into different banks.
__device__ __forceinline__ int tile_at(int pix, int j, int half) {
  return pix * 32 + ((half ^ ((j >> 2) & 1)) << 4);
}
template <bool TRANS>
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const char* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// Eight channels of a pixel.  Features come from the caller and may lie on any 4-byte
// boundary: vec says that they lie on a 16-byte one.
__device__ __forceinline__ uint4 ld8(const uint16_t* p, int vec) {
  if (vec) return __ldg(reinterpret_cast<const uint4*>(p));
  const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
  return make_uint4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
}

// 3x3 "same" convolution, zero padding.  A block = 4 warps of 16 pixels in R rows; its
// (R + 2) x 66 input pixels are staged once and an A fragment (16 pixels of an input row,
// one dx) feeds the output rows above, at and below it, each output's taps still in order
// 0..8.  The layers are bound by their 32 bytes a pixel through L2 and by latency: with one
// row a block, fragments were loaded nine times from global memory and the weights staged
// per 64 pixels (32 windows of 64x64: 10.5 -> 7.8 us a layer, 12.6 -> 9.7 with the mask).
// XC = 16: x has kC channels; 1: one channel a pixel, the others zero (dY of the last layer).
// MODE 0: ReLU -> bf16 (16 ch); 1: linear, channel 0 -> fp32;
// 2: multiply by (act > 0) (ReLU derivative of the layer input) -> bf16.
template <int NT, int MODE, int XC, int R>
__global__ void __launch_bounds__(128, 4) k_conv(int H, int W, const uint16_t* __restrict__ x, int vec,
                                              const uint32_t* __restrict__ frag,
                                              const uint16_t* __restrict__ act, void* out) {
  constexpr int kPW = 66;
  __shared__ __align__(16) char tile[XC == 1 ? 16 : (R + 2) * kPW * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int xb0 = blockIdx.x * 64, x0 = xb0 + warp * 16;
  const int y0 = blockIdx.y * R;
  const long long img = (long long)blockIdx.z * H * W;
  if (XC == kC) {
    for (int i = threadIdx.x; i < (R + 2) * kPW * 2; i += 128) {
      const int q = i >> 1, half = i & 1, row = q / kPW, j = q - row * kPW;
      const int yy = y0 + row - 1, xx = xb0 + j - 1;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (yy >= 0 && yy < H && xx >= 0 && xx < W)
        v = ld8(x + (img + (long long)yy * W + xx) * kC + half * 8, vec);
      *reinterpret_cast<uint4*>(tile + tile_at(q, j, half)) = v;
    }
  }
  uint2 b[9][NT];
#pragma unroll
  for (int tap = 0; tap < 9; ++tap)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      b[tap][nt] = __ldg(reinterpret_cast<const uint2*>(frag) + (tap * NT + nt) * 32 + lane);
  // the layer input whose sign masks the result, fetched with the tile
  uint32_t m[R][2][NT];
  if (MODE == 2) {
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int y = y0 + r, px = x0 + g + 8 * half;
        const uint32_t* a =
            reinterpret_cast<const uint32_t*>(act + (img + (long long)y * W + px) * kC) + t;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) m[r][half][nt] = y < H && px < W ? __ldg(a + nt * 4) : 0u;
      }
  }
  if (XC == kC) __syncthreads();
  if (x0 >= W) return;
  float acc[R][NT][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
      acc[r][nt][0] = acc[r][nt][1] = acc[r][nt][2] = acc[r][nt][3] = 0.0f;
#pragma unroll
  for (int row = 0; row < R + 2; ++row) {
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) {
      uint32_t a[4] = {0u, 0u, 0u, 0u};
      if (XC == kC) {
        const int j = warp * 16 + dx + (lane & 15);
        ldsm4<false>(a, tile + tile_at(row * kPW + j, j, lane >> 4));
      } else {
        const int yy = y0 + row - 1, xa = x0 + g + dx - 1, xb = xa + 8;
        const uint16_t* p = x + img + (long long)yy * W;
        if (t == 0 && yy >= 0 && yy < H) {
          if (xa >= 0 && xa < W) a[0] = __ldg(p + xa);
          if (xb < W) a[1] = __ldg(p + xb);
        }
      }
#pragma unroll
      for (int dy = 0; dy < 3; ++dy) {
        const int r = row - dy;
        if (r < 0 || r >= R) continue;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
          mma_bf16(acc[r][nt], a[0], a[1], a[2], a[3], b[dy * 3 + dx][nt].x, b[dy * 3 + dx][nt].y);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int y = y0 + r;
    if (y >= H) break;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int px = x0 + g + 8 * half;
      if (px >= W) continue;
      const long long pix = img + (long long)y * W + px;
      if (MODE == 1) {
        if (t == 0) reinterpret_cast<float*>(out)[pix] = acc[r][0][2 * half];
        continue;
      }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int co = nt * 8 + 2 * t;
        float v0 = acc[r][nt][2 * half], v1 = acc[r][nt][2 * half + 1];
        if (MODE == 0) {
          v0 = fmaxf(v0, 0.0f);
          v1 = fmaxf(v1, 0.0f);
        } else {
          const uint32_t a = m[r][half][nt];
          if (!(bf((uint16_t)(a & 0xffffu)) > 0.0f)) v0 = 0.0f;
          if (!(bf((uint16_t)(a >> 16)) > 0.0f)) v1 = 0.0f;
        }
        reinterpret_cast<uint32_t*>(out)[(pix * kC + co) / 2] = pack2(v0, v1);
      }
    }
  }
}

// Weight gradient partials: block b sums k-steps [b*ks_per, (b+1)*ks_per) of 16
// pixels (W % 16 == 0, so a k-step is 16 pixels of one row).
// D[m = ci][n = co] += A[ci][p] B[p][co],  A[ci][p] = X[p + tap, ci],  B = dY.
// Twelve warps: four share the k-steps, three the rows of taps.  A warp stages its 18 pixels
// of X and 16 of dY in 16-byte words, two k-steps ahead in registers, and ldmatrix.trans
// turns pixels into the K dimension (before: one warp for all nine taps, 72 two-byte loads
// a lane and k-step; 32 windows of 64x64: 32 -> 13 us a layer).
// NT = 2: dY has kC channels; 1: one channel a pixel.
template <int NT>
__global__ void __launch_bounds__(384) k_wgrad(int H, int W, long long nks, int ks_per,
                                               const uint16_t* __restrict__ x, int vec,
                                               const uint16_t* __restrict__ dy,
                                               float* __restrict__ partial) {
  constexpr int NO = 8 * NT, kStage = (18 + 16) * 32;
  constexpr int kRed = 4 * 9 * 16 * NO * 4;
  __shared__ __align__(16) char sm[kRed > 12 * kStage ? kRed : 12 * kStage];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int kg = warp / 3, ty = warp % 3;
  char* sx = sm + warp * kStage;
  char* sy = sx + 18 * 32;
  float acc[3][NT][4];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[k][nt][0] = acc[k][nt][1] = acc[k][nt][2] = acc[k][nt][3] = 0.0f;
  // k-steps fit 32 bits (at most 2^31 pixels a batch); wpr of them a row
  const unsigned wpr = W / 16, ks0 = blockIdx.x * (unsigned)ks_per;
  const unsigned ks1 = (unsigned)min(nks, (long long)ks0 + ks_per);
  struct In {
    uint4 x0, x1, d;  // halves lane and 32 + lane (lane < 4) of the 36 of X; dY
  };
  auto load = [&](unsigned ks, In& in) {
    in.x0 = in.x1 = in.d = make_uint4(0u, 0u, 0u, 0u);
    if (ks >= ks1) return;
    const unsigned row = ks / wpr;  // n*H + y
    const long long rowid = row;
    const int x0 = (int)(ks - row * wpr) * 16;
    const int yy = (int)(row % (unsigned)H) + ty - 1;
    const uint16_t* xr = x + (rowid + ty - 1) * W * kC;
    if (yy >= 0 && yy < H) {
      const int xa = x0 - 1 + (lane >> 1), xb = xa + 16;
      if (xa >= 0) in.x0 = ld8(xr + (long long)xa * kC + (lane & 1) * 8, vec);
      if (lane < 4 && xb < W) in.x1 = ld8(xr + (long long)xb * kC + (lane & 1) * 8, vec);
    }
    if (NT == 2) {
      in.d = __ldg(reinterpret_cast<const uint4*>(dy + (rowid * W + x0) * kC) + lane);
    } else {
      const uint32_t* q = reinterpret_cast<const uint32_t*>(dy + rowid * W + x0);
      in.d.x = __ldg(q + t);
      in.d.y = __ldg(q + t + 4);
    }
  };
  auto step = [&](In& in, unsigned next) {
    __syncwarp();
    *reinterpret_cast<uint4*>(sx + tile_at(lane >> 1, lane >> 1, lane & 1)) = in.x0;
    if (lane < 4)
      *reinterpret_cast<uint4*>(sx + tile_at(16 + (lane >> 1), 16 + (lane >> 1), lane & 1)) = in.x1;
    if (NT == 2) *reinterpret_cast<uint4*>(sy + tile_at(lane >> 1, lane >> 1, lane & 1)) = in.d;
    uint32_t b[4] = {g == 0 ? in.d.x : 0u, g == 0 ? in.d.y : 0u, 0u, 0u};  // (p 0-7, 8-15) of co 0-7, of co 8-15
    load(next, in);  // into the same registers: a copy would wait for the words here
    __syncwarp();
    if (NT == 2) {
      const int j = lane & 15;
      ldsm4<true>(b, sy + tile_at(j, j, lane >> 4));
    }
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) {
      uint32_t a[4];  // p 0-7 of ci 0-7, 8-15; p 8-15 of ci 0-7, 8-15
      const int j = dx + (lane >> 4) * 8 + (lane & 7);
      ldsm4<true>(a, sx + tile_at(j, j, (lane >> 3) & 1));
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        mma_bf16(acc[dx][nt], a[0], a[1], a[2], a[3], b[2 * nt], b[2 * nt + 1]);
    }
  };
  In in0, in1;
  load(ks0 + kg, in0);
  load(ks0 + kg + 4, in1);
  for (unsigned ks = ks0 + kg; ks < ks1; ks += 8) {
    step(in0, ks + 8);
    if (ks + 4 >= ks1) break;
    step(in1, ks + 12);
  }
  // D fragment: (row g / g+8 = ci, cols 2t, 2t+1 = co within the n-tile)
  __syncthreads();
  float* red = reinterpret_cast<float*>(sm);
#pragma unroll
  for (int dx = 0; dx < 3; ++dx)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int ci = g + (e >> 1) * 8, co = nt * 8 + 2 * t + (e & 1), tap = ty * 3 + dx;
        red[((kg * 9 + tap) * 16 + ci) * NO + co] = acc[dx][nt][e];
      }
  __syncthreads();
  constexpr int n = 9 * 16 * NO;
  for (int i = threadIdx.x; i < n; i += 384)
    partial[(long long)blockIdx.x * n + i] =
        ((red[i] + red[n + i]) + red[2 * n + i]) + red[3 * n + i];
}

// Sum the partials in block order into the logical gradient layout, 32 elements a block:
// 256 threads fetch 128 partials of each at once, one warp adds them in order (a thread's own
// chain of dependent loads took 16 to 28 us).  The block after the last element's, launched
// with the loss partials, sums those in order.
__global__ void __launch_bounds__(256) k_wgrad_reduce(int nblk, int NO,
                                                      const float* __restrict__ partial, int ci_n,
                                                      int co_n, float* __restrict__ grad, int nl,
                                                      const float* __restrict__ lpart, float scale,
                                                      float* __restrict__ loss) {
  constexpr int kB = 128;
  __shared__ float s[kB * 32];
  const int n = 9 * ci_n * co_n, lane = threadIdx.x & 31, wr = threadIdx.x >> 5;
  float sum = 0.0f;
  if ((int)blockIdx.x * 32 >= n) {
    for (int b0 = 0; b0 < nl; b0 += kB * 32) {
      const int m = min(kB * 32, nl - b0);
      __syncthreads();
      for (int i = threadIdx.x; i < m; i += 256) s[i] = lpart[b0 + i];
      __syncthreads();
      if (threadIdx.x == 0) {
#pragma unroll 16
        for (int i = 0; i < m; ++i) sum += s[i];
      }
    }
    if (threadIdx.x == 0) *loss = sum * scale;
    return;
  }
  const int i = min((int)blockIdx.x * 32 + lane, n - 1);
  const int co = i % co_n, ci = (i / co_n) % ci_n, tap = i / (co_n * ci_n);
  const float* p = partial + (tap * 16 + ci) * NO + co;
  for (int b0 = 0; b0 < nblk; b0 += kB) {
    const int m = min(kB, nblk - b0);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kB / 8; ++k) {
      const int b = k * 8 + wr;
      if (b < m) s[b * 32 + lane] = p[(long long)(b0 + b) * 9 * 16 * NO];
    }
    __syncthreads();
    if (wr == 0) {
#pragma unroll 16
      for (int b = 0; b < m; ++b) sum += s[b * 32 + lane];
    }
  }
  if (wr == 0 && (int)blockIdx.x * 32 + lane < n) grad[i] = sum;
}

// Masked mean-square loss: r = m (y - t); dY = 2 r / count (bf16, one channel);
// per-block partial sums of r^2 (fixed-order, deterministic).
__global__ void k_loss(long long npix, const float* __restrict__ y, const float* __restrict__ tgt,
                       const float* __restrict__ mask, float inv_count, uint16_t* __restrict__ dy,
                       float* __restrict__ part) {
  __shared__ float s[256];
  float acc = 0.0f;
  for (long long p = blockIdx.x * 256LL + threadIdx.x; p < npix; p += gridDim.x * 256LL) {
    const float r = (mask ? mask[p] : 1.0f) * (y[p] - tgt[p]);
    acc += r * r;
    dy[p] = (uint16_t)pack2(2.0f * r * inv_count, 0.0f);
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

__global__ void k_adam(int n, float* __restrict__ p, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// Window origin of image k: off[k] when an offset table is given, else k*stride.
__device__ __forceinline__ long long img_base(const long long* off, long long stride, int k) {
  return off ? off[k] : (long long)k * stride;
}

// features of the (h, w) windows of fields with row pitch ld, times scale[k]:
// (u, u_prev, c2 u, c2^2 u, s_next, s_prev) where s_* is the value injected at
// a source cell of the window in this / the previous step (n_src sources per
// window at src[2(k n_src + q)], values inj_next / inj_prev[k n_src + q]).
__global__ void k_features(int H, int W, const float* __restrict__ u, const float* __restrict__ up,
                           const float* __restrict__ c2, long long ld, const long long* u_off,
                           long long u_stride, const long long* c_off, long long c_stride,
                           const float* __restrict__ scale, int n_src, const int* __restrict__ src,
                           const float* __restrict__ inj_next, const float* __restrict__ inj_prev,
                           uint16_t* __restrict__ feat) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, k = blockIdx.z;
  if (x >= W) return;
  const long long q = img_base(u_off, u_stride, k) + (long long)y * ld + x;
  const float s = scale ? scale[k] : 1.0f;
  const float a = __fmul_rn(u[q], s), b = __fmul_rn(up[q], s);
  const float c = c2[img_base(c_off, c_stride, k) + (long long)y * ld + x];
  const float ca = __fmul_rn(c, a);
  float sn = 0.0f, sp = 0.0f;
  for (int j = 0; j < n_src; ++j) {
    const int i = k * n_src + j;
    if (src[2 * i] == x && src[2 * i + 1] == y) {
      if (inj_next) sn = __fadd_rn(sn, __fmul_rn(inj_next[i], s));
      if (inj_prev) sp = __fadd_rn(sp, __fmul_rn(inj_prev[i], s));
    }
  }
  uint32_t* f = reinterpret_cast<uint32_t*>(feat + (((long long)k * H + y) * W + x) * kC);
  f[0] = pack2(a, b);
  f[1] = pack2(ca, __fmul_rn(c, ca));
  f[2] = pack2(sn, sp);
#pragma unroll
  for (int j = 3; j < kC / 2; ++j) f[j] = 0u;
}

// Training target: the part of u^{n+1} the coarse step misses,
//   target = s * (u_next - (scalar step(u, u_prev) + injection)),
// with the scalar step's exact arithmetic (scalar2d.jl:29-53, as the solver
// kernel); mask = 1 where the stencil and the network's 7x7 receptive field
// fit the window and outside a square of half-width src_r around the source,
// else 0 (and target 0).
struct D2C {
  float two_c0;
  float d[5];
};
template <int N>
__global__ void k_target(int H, int W, D2C cf, const float* __restrict__ u,
                         const float* __restrict__ up, const float* __restrict__ un,
                         const float* __restrict__ c2, long long ld, const long long* u_off,
                         long long u_stride, const long long* c_off, long long c_stride,
                         const float* __restrict__ scale, const int* __restrict__ src,
                         const float* __restrict__ inj, int src_r, float* __restrict__ tgt,
                         float* __restrict__ mask) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, k = blockIdx.z;
  if (x >= W) return;
  const long long o = ((long long)k * H + y) * W + x;
  const int sx = src ? src[2 * k] : -1000000, sz = src ? src[2 * k + 1] : -1000000;
  const bool near_src = abs(x - sx) <= src_r && abs(y - sz) <= src_r;
  constexpr int E = N > 3 ? N : 3;  // the stencil and the network's receptive field fit
  if (x < E || x >= W - E || y < E || y >= H - E || near_src) {
    tgt[o] = 0.0f;
    if (mask) mask[o] = 0.0f;
    return;
  }
  const long long q = img_base(u_off, u_stride, k) + (long long)y * ld + x;
  const float uc = u[q];
  float lap = __fmul_rn(cf.two_c0, uc);
#pragma unroll
  for (int l = 1; l <= N; ++l) {
    const float nb = __fadd_rn(__fadd_rn(__fadd_rn(u[q + l], u[q - l]), u[q + l * ld]), u[q - l * ld]);
    lap = __fmaf_rn(cf.d[l - 1], nb, lap);
  }
  const float c = c2[img_base(c_off, c_stride, k) + (long long)y * ld + x];
  float nxt = __fmaf_rn(c, lap, __fsub_rn(__fmul_rn(2.0f, uc), up[q]));
  if (x == sx && y == sz && inj) nxt = __fadd_rn(nxt, inj[k]);
  const float s = scale ? scale[k] : 1.0f;
  tgt[o] = __fmul_rn(__fsub_rn(un[q], nxt), s);
  if (mask) mask[o] = 1.0f;
}

struct Bufs {
  uint32_t* frag;
  uint16_t *h1, *h2, *d3, *dh2, *dh1;
  float *y, *part, *lpart;
};

int plan_bufs(fomo_ctx* ctx, long long npix, int nblk, int nlb, Bufs& b) {
  Arena ar;
  const size_t o_f = ar.take<uint32_t>(kNFrag);
  const size_t o_h1 = ar.take<uint16_t>(npix * kC), o_h2 = ar.take<uint16_t>(npix * kC);
  const size_t o_d3 = ar.take<uint16_t>(npix), o_dh2 = ar.take<uint16_t>(npix * kC);
  const size_t o_dh1 = ar.take<uint16_t>(npix * kC);
  const size_t o_y = ar.take<float>(npix);
  const size_t o_p = ar.take<float>((size_t)std::max(nblk, 1) * 9 * 16 * 16);
  const size_t o_l = ar.take<float>(std::max(nlb, 1));
  if (int rc = ensure_workspace(ctx, ar.off)) return rc;
  b.frag = ws_ptr<uint32_t>(ctx, o_f);
  b.h1 = ws_ptr<uint16_t>(ctx, o_h1);
  b.h2 = ws_ptr<uint16_t>(ctx, o_h2);
  b.d3 = ws_ptr<uint16_t>(ctx, o_d3);
  b.dh2 = ws_ptr<uint16_t>(ctx, o_dh2);
  b.dh1 = ws_ptr<uint16_t>(ctx, o_dh1);
  b.y = ws_ptr<float>(ctx, o_y);
  b.part = ws_ptr<float>(ctx, o_p);
  b.lpart = ws_ptr<float>(ctx, o_l);
  return FOMO_OK;
}

int aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Rows per block of a layer: four where that still gives every SM two blocks, else one
// (a single 120x100 image: 240 blocks of one row, 60 of four).
template <int NT, int MODE, int XC>
void conv(cudaStream_t st, int n, int h, int w, const uint16_t* x, const uint32_t* frag,
          const uint16_t* act, void* out) {
  const int vec = aligned16(x), wide = (w + 63) / 64, tall = (h + 3) / 4;
  if ((long long)wide * tall * n >= 296)
    k_conv<NT, MODE, XC, 4><<<dim3(wide, tall, n), 128, 0, st>>>(h, w, x, vec, frag, act, out);
  else
    k_conv<NT, MODE, XC, 1><<<dim3(wide, h, n), 128, 0, st>>>(h, w, x, vec, frag, act, out);
}

cudaError_t forward(cudaStream_t st, int n, int h, int w, const uint16_t* feat, const float* params,
                    const Bufs& b, float* y, bool pack = true) {
  if (pack) k_pack<<<(kNFrag / 2 + 255) / 256, 256, 0, st>>>(params, b.frag);
  conv<2, 0, kC>(st, n, h, w, feat, b.frag + kOffF1, nullptr, b.h1);
  conv<2, 0, kC>(st, n, h, w, b.h1, b.frag + kOffF2, nullptr, b.h2);
  conv<1, 1, kC>(st, n, h, w, b.h2, b.frag + kOffF3, nullptr, y);
  return cudaGetLastError();
}

int check_dims(fomo_ctx* ctx, int n, int h, int w, bool grad) {
  if (n < 1 || h < 1 || w < 1) return fail(ctx, FOMO_EARG, "corrector: empty batch");
  if (grad && (w % 16)) return fail(ctx, FOMO_EARG, "corrector gradients need width % 16 == 0");
  if ((long long)n * h * w > (1LL << 31)) return fail(ctx, FOMO_EARG, "corrector batch too large");
  return FOMO_OK;
}

}  // namespace

// Device-side helpers used by the corrected coarse solver.
cudaError_t corr_forward_device(cudaStream_t st, int h, int w, const float* u, const float* up,
                                const float* c2, long long ld, int n_src, const int* src,
                                const float* inj_next, const float* inj_prev,
                                const float* params, void* scratch, float* y, bool pack);
size_t corr_scratch_bytes(long long npix);

size_t corr_scratch_bytes(long long npix) {
  return 4 * (size_t)kNFrag + 3 * (size_t)npix * kC * 2 + 64 * 4;
}

cudaError_t corr_forward_device(cudaStream_t st, int h, int w, const float* u, const float* up,
                                const float* c2, long long ld, int n_src, const int* src,
                                const float* inj_next, const float* inj_prev,
                                const float* params, void* scratch, float* y, bool pack) {
  const long long npix = (long long)h * w;
  Bufs b{};
  char* s = static_cast<char*>(scratch);
  b.frag = reinterpret_cast<uint32_t*>(s);
  uint16_t* feat = reinterpret_cast<uint16_t*>(s + 4 * (size_t)kNFrag);
  b.h1 = feat + npix * kC;
  b.h2 = b.h1 + npix * kC;
  k_features<<<dim3((w + 127) / 128, h, 1), 128, 0, st>>>(
      h, w, u, up, c2, ld, nullptr, 0, nullptr, 0, nullptr, n_src, src, inj_next, inj_prev, feat);
  return forward(st, 1, h, w, feat, params, b, y, pack);
}

}  // namespace fomo

using namespace fomo;

extern "C" {

int fomo_corr_param_count(void) { return kNParam; }

int fomo_corr_features(fomo_ctx* ctx, int32_t n, int32_t h, int32_t w, const float* u,
                       const float* u_prev, const float* c2, int64_t ld, const int64_t* u_off,
                       int64_t u_stride, const int64_t* c2_off, int64_t c2_stride,
                       const float* scale, int32_t n_src, const int32_t* src,
                       const float* inj_next, const float* inj_prev, uint16_t* feat) {
  if (!ctx) return FOMO_EARG;
  if (int rc = check_dims(ctx, n, h, w, false)) return rc;
  if (!u || !u_prev || !c2 || !feat || ld < w || n_src < 0 || (n_src > 0 && !src))
    return fail(ctx, FOMO_EARG, "corrector features: bad arguments");
  k_features<<<dim3((w + 127) / 128, h, n), 128, 0, ctx->stream>>>(
      h, w, u, u_prev, c2, ld, reinterpret_cast<const long long*>(u_off), u_stride,
      reinterpret_cast<const long long*>(c2_off), c2_stride, scale, n_src, src, inj_next,
      inj_prev, feat);
  FOMO_CU(ctx, cudaGetLastError());
  return FOMO_OK;
}

int fomo_corr_target(fomo_ctx* ctx, int32_t n, int32_t h, int32_t w, int32_t fd_order,
                     const float* u, const float* u_prev, const float* u_next, const float* c2,
                     int64_t ld, const int64_t* u_off, int64_t u_stride, const int64_t* c2_off,
                     int64_t c2_stride, const float* scale, const int32_t* src, const float* inj,
                     int32_t src_r, float* target, float* mask) {
  if (!ctx) return FOMO_EARG;
  if (int rc = check_dims(ctx, n, h, w, false)) return rc;
  const int N = order_to_N(fd_order);
  if (N < 0) return fail(ctx, FOMO_EARG, "Unsupported FD order: " + std::to_string(fd_order));
  if (!u || !u_prev || !u_next || !c2 || !target || ld < w)
    return fail(ctx, FOMO_EARG, "corrector target: bad arguments");
  D2C cf;
  cf.two_c0 = 2.0f * kD2C0[N];
  for (int l = 0; l < 5; ++l) cf.d[l] = kD2[N][l];
  const dim3 grid((w + 127) / 128, h, n);
  const long long* uo = reinterpret_cast<const long long*>(u_off);
  const long long* co = reinterpret_cast<const long long*>(c2_off);
#define FOMO_TGT(NN)                                                                          \
  case NN:                                                                                    \
    k_target<NN><<<grid, 128, 0, ctx->stream>>>(h, w, cf, u, u_prev, u_next, c2, ld, uo,       \
                                                u_stride, co, c2_stride, scale, src, inj, src_r, \
                                                target, mask);                                 \
    break;
  switch (N) { FOMO_TGT(1) FOMO_TGT(2) FOMO_TGT(3) FOMO_TGT(4) FOMO_TGT(5) }
#undef FOMO_TGT
  FOMO_CU(ctx, cudaGetLastError());
  return FOMO_OK;
}

int fomo_corr_forward(fomo_ctx* ctx, int32_t n, int32_t h, int32_t w, const uint16_t* feat,
                      const float* params, float* y) {
  if (!ctx) return FOMO_EARG;
  if (int rc = check_dims(ctx, n, h, w, false)) return rc;
  if (!feat || !params || !y) return fail(ctx, FOMO_EARG, "corrector forward: null pointer");
  Bufs b{};
  if (int rc = plan_bufs(ctx, (long long)n * h * w, 1, 1, b)) return rc;
  FOMO_CU(ctx, forward(ctx->stream, n, h, w, feat, params, b, y));
  return FOMO_OK;
}

int fomo_corr_gradients(fomo_ctx* ctx, int32_t n, int32_t h, int32_t w, const uint16_t* feat,
                        const float* target, const float* mask, const float* params, float* grad,
                        float* loss, float* y_out) {
  if (!ctx) return FOMO_EARG;
  if (int rc = check_dims(ctx, n, h, w, true)) return rc;
  if (!feat || !target || !params || !grad || !loss)
    return fail(ctx, FOMO_EARG, "corrector gradients: null pointer");
  cudaStream_t st = ctx->stream;
  const long long npix = (long long)n * h * w, nks = npix / 16;
  const int ks_per = 64;
  const int nblk = (int)((nks + ks_per - 1) / ks_per);
  const int nlb = (int)std::min<long long>(1024, (npix + 255) / 256);
  Bufs b{};
  if (int rc = plan_bufs(ctx, npix, nblk, nlb, b)) return rc;
  float* y = y_out ? y_out : b.y;
  FOMO_CU(ctx, forward(st, n, h, w, feat, params, b, y));
  // loss and dY3
  const float count = (float)npix;  // the loss is a mean over every pixel (mask zeros included)
  k_loss<<<nlb, 256, 0, st>>>(npix, y, target, mask, 1.0f / count, b.d3, b.lpart);
  // layer 3: dW3 = sum h2[p+tap] dY3[p];  dH2 = conv_t(dY3, W3) * (h2 > 0)
  k_wgrad<1><<<nblk, 384, 0, st>>>(h, w, nks, ks_per, b.h2, 1, b.d3, b.part);
  k_wgrad_reduce<<<(kNW3 + 31) / 32 + 1, 256, 0, st>>>(nblk, 8, b.part, 16, 1, grad + kNW1 + kNW2,
                                                       nlb, b.lpart, 1.0f / count, loss);
  conv<2, 2, 1>(st, n, h, w, b.d3, b.frag + kOffT3, b.h2, b.dh2);
  // layer 2: dW2 = sum h1[p+tap] dPre2[p];  dH1 = conv_t(dPre2, W2) * (h1 > 0)
  k_wgrad<2><<<nblk, 384, 0, st>>>(h, w, nks, ks_per, b.h1, 1, b.dh2, b.part);
  k_wgrad_reduce<<<kNW2 / 32, 256, 0, st>>>(nblk, 16, b.part, 16, 16, grad + kNW1, 0, nullptr, 0.0f,
                                            nullptr);
  conv<2, 2, kC>(st, n, h, w, b.dh2, b.frag + kOffT2, b.h1, b.dh1);
  // layer 1: dW1 = sum feat[p+tap] dPre1[p]
  k_wgrad<2><<<nblk, 384, 0, st>>>(h, w, nks, ks_per, feat, aligned16(feat), b.dh1, b.part);
  k_wgrad_reduce<<<kNW1 / 32, 256, 0, st>>>(nblk, 16, b.part, kCin, 16, grad, 0, nullptr, 0.0f,
                                            nullptr);
  FOMO_CU(ctx, cudaGetLastError());
  return FOMO_OK;
}

int fomo_corr_adam(fomo_ctx* ctx, int32_t count, float* params, const float* grad, float* m,
                   float* v, float lr, float beta1, float beta2, float eps, int32_t step) {
  if (!ctx) return FOMO_EARG;
  if (count < 1 || !params || !grad || !m || !v || step < 1)
    return fail(ctx, FOMO_EARG, "corrector adam: bad arguments");
  const float c1 = 1.0f - std::pow(beta1, (float)step), c2 = 1.0f - std::pow(beta2, (float)step);
  k_adam<<<(count + 255) / 256, 256, 0, ctx->stream>>>(count, params, grad, m, v, lr, beta1, beta2,
                                                      eps, c1, c2);
  FOMO_CU(ctx, cudaGetLastError());
  return FOMO_OK;
}

}  // extern "C"
