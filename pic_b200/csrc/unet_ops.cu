// unet_ops.cu -- the learned preconditioner's network kernels other than the
// tensor-core convolutions: input features, pooling, upsample + concat, ReLU
// backward, the 1x1 head, loss, output scaling, the weight gradient of the
// 3x3 convolutions, and Adam.  NHWC BF16 activations are moved 8 channels
// (16 bytes) per thread; parameters and gradients are FP32.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/picunet.h"

namespace {

using bf16 = __nv_bfloat16;

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
inline unsigned capped(int64_t n, int t, unsigned cap) {
  unsigned b = nblk(n, t);
  return b < cap ? (b ? b : 1u) : cap;
}

int launched() { return cudaPeekAtLastError() == cudaSuccess ? UNET_OK : UNET_ERR_CUDA; }

// 8 BF16 channels as one 16-byte word
struct V8 {
  uint4 u;
};

__device__ __forceinline__ void v8_to_f(const V8 &v, float f[8]) {
  const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v.u);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float2 t = __bfloat1622float2(h[q]);
    f[2 * q] = t.x;
    f[2 * q + 1] = t.y;
  }
}

__device__ __forceinline__ V8 f_to_v8(const float f[8]) {
  V8 v;
  __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&v.u);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
  return v;
}

__device__ __forceinline__ V8 ld8(const bf16 *p) { V8 v; v.u = *reinterpret_cast<const uint4 *>(p); return v; }
__device__ __forceinline__ void st8(bf16 *p, const V8 &v) { *reinterpret_cast<uint4 *>(p) = v.u; }

// ---- residual scale -------------------------------------------------------
// s = sqrt(sum over unknown nodes of r^2 / count): per-block partials in a
// fixed order; the last block to finish sums them in block order
// (deterministic), writes scale[0] = s, scale[1] = 1/s (0 when r = 0) and
// re-arms the ticket.
constexpr int RMS_THREADS = 256;

__global__ void __launch_bounds__(RMS_THREADS) k_rms(int64_t npix, const double *__restrict__ r,
                                                     const int32_t *__restrict__ mask, double *__restrict__ part,
                                                     unsigned int *ticket, double *__restrict__ scale) {
  __shared__ double ss[RMS_THREADS];
  __shared__ double sc[RMS_THREADS];
  __shared__ bool last;
  double s = 0.0, c = 0.0;
  for (int64_t p = (int64_t)blockIdx.x * RMS_THREADS + threadIdx.x; p < npix; p += (int64_t)gridDim.x * RMS_THREADS)
    if (mask[p] > 0) {
      s += r[p] * r[p];
      c += 1.0;
    }
  ss[threadIdx.x] = s;
  sc[threadIdx.x] = c;
  __syncthreads();
  for (int o = RMS_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      ss[threadIdx.x] += ss[threadIdx.x + o];
      sc[threadIdx.x] += sc[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = ss[0];
    part[2 * blockIdx.x + 1] = sc[0];
    __threadfence();
    last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  double ts = 0.0, tc = 0.0;
  for (unsigned b = 0; b < gridDim.x; ++b) {
    ts += *(volatile double *)&part[2 * b];
    tc += *(volatile double *)&part[2 * b + 1];
  }
  const double v = (tc > 0.0) ? sqrt(ts / tc) : 0.0;
  scale[0] = v;
  scale[1] = (v > 0.0) ? 1.0 / v : 0.0;
  *ticket = 0u;
}

__global__ void k_features(int64_t npix, const double *__restrict__ r, const double *__restrict__ scale,
                           const float *__restrict__ fs, bf16 *__restrict__ x) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npix) return;
  const float f[8] = {(float)(r[p] * scale[1]), fs[3 * p], fs[3 * p + 1], fs[3 * p + 2], 0.f, 0.f, 0.f, 0.f};
  st8(x + 8 * p, f_to_v8(f));
}

// ---- pooling / upsampling (g = channel group of 8) --------------------------
__global__ void k_pool(int n, int h, int w, int c, const bf16 *__restrict__ x, bf16 *__restrict__ y) {
  const int h2 = (h + 1) / 2, w2 = (w + 1) / 2, G = c / 8;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * h2 * w2 * G) return;
  const int g = (int)(idx % G);
  const int64_t q = idx / G;
  const int j2 = (int)(q % w2), i2 = (int)((q / w2) % h2), b = (int)(q / ((int64_t)w2 * h2));
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  int cnt = 0;
  for (int di = 0; di < 2; ++di)
    for (int dj = 0; dj < 2; ++dj) {
      const int i = 2 * i2 + di, j = 2 * j2 + dj;
      if (i < h && j < w) {
        float f[8];
        v8_to_f(ld8(x + (((int64_t)b * h + i) * w + j) * c + 8 * g), f);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += f[e];
        ++cnt;
      }
    }
  const float inv = 1.0f / (float)cnt;
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] *= inv;
  st8(y + idx * 8, f_to_v8(s));
}

__global__ void k_pool_bwd(int n, int h, int w, int c, const bf16 *__restrict__ dy, bf16 *__restrict__ dx,
                           int acc) {
  const int h2 = (h + 1) / 2, w2 = (w + 1) / 2, G = c / 8;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * h * w * G) return;
  const int g = (int)(idx % G);
  const int64_t q = idx / G;
  const int j = (int)(q % w), i = (int)((q / w) % h), b = (int)(q / ((int64_t)w * h));
  const int i2 = i / 2, j2 = j / 2;
  const float inv = 1.0f / (float)((min(2 * i2 + 2, h) - 2 * i2) * (min(2 * j2 + 2, w) - 2 * j2));
  float f[8];
  v8_to_f(ld8(dy + (((int64_t)b * h2 + i2) * w2 + j2) * c + 8 * g), f);
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] *= inv;
  if (acc) {
    float a[8];
    v8_to_f(ld8(dx + idx * 8), a);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] += a[e];
  }
  st8(dx + idx * 8, f_to_v8(f));
}

__global__ void k_upcat(int n, int h, int w, int c1, int c2, const bf16 *__restrict__ lo,
                        const bf16 *__restrict__ skip, bf16 *__restrict__ y) {
  const int h2 = (h + 1) / 2, w2 = (w + 1) / 2, G1 = c1 / 8, G = (c1 + c2) / 8;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * h * w * G) return;
  const int g = (int)(idx % G);
  const int64_t q = idx / G;
  const int j = (int)(q % w), i = (int)((q / w) % h), b = (int)(q / ((int64_t)w * h));
  const bf16 *src = (g < G1) ? lo + (((int64_t)b * h2 + i / 2) * w2 + j / 2) * c1 + 8 * g
                             : skip + q * c2 + 8 * (g - G1);
  st8(y + idx * 8, ld8(src));
}

__global__ void k_upcat_bwd_lo(int n, int h, int w, int c1, int c2, const bf16 *__restrict__ dy,
                               bf16 *__restrict__ dlo) {
  const int h2 = (h + 1) / 2, w2 = (w + 1) / 2, G1 = c1 / 8, ct = c1 + c2;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)n * h2 * w2 * G1) return;
  const int g = (int)(idx % G1);
  const int64_t q = idx / G1;
  const int j2 = (int)(q % w2), i2 = (int)((q / w2) % h2), b = (int)(q / ((int64_t)w2 * h2));
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int di = 0; di < 2; ++di)
    for (int dj = 0; dj < 2; ++dj) {
      const int i = 2 * i2 + di, j = 2 * j2 + dj;
      if (i < h && j < w) {
        float f[8];
        v8_to_f(ld8(dy + (((int64_t)b * h + i) * w + j) * ct + 8 * g), f);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += f[e];
      }
    }
  st8(dlo + idx * 8, f_to_v8(s));
}

__global__ void k_upcat_bwd_skip(int64_t npix, int c1, int c2, const bf16 *__restrict__ dy,
                                 bf16 *__restrict__ dskip, int acc) {
  const int G2 = c2 / 8, ct = c1 + c2;
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= npix * G2) return;
  const int g = (int)(idx % G2);
  const int64_t p = idx / G2;
  V8 v = ld8(dy + p * ct + c1 + 8 * g);
  if (acc) {
    float f[8], a[8];
    v8_to_f(v, f);
    v8_to_f(ld8(dskip + idx * 8), a);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] += a[e];
    v = f_to_v8(f);
  }
  st8(dskip + idx * 8, v);
}

// ---- ReLU backward + bias gradient ------------------------------------------
// Block of G * floor(256/G) threads (G = c/8 channel groups): each thread keeps
// one channel group for the whole grid-stride loop and sums its 8 bias
// gradients in registers.
__global__ void k_relu_bwd(int64_t npix, int c, const bf16 *__restrict__ y, bf16 *__restrict__ dy,
                           float *__restrict__ db) {
  extern __shared__ float sdb[];
  const int G = c / 8;
  for (int k = threadIdx.x; k < c; k += blockDim.x) sdb[k] = 0.0f;
  __syncthreads();
  const int g = threadIdx.x % G;
  float a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const int64_t tot = npix * G;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < tot;
       idx += (int64_t)gridDim.x * blockDim.x) {
    float fy[8], fd[8];
    v8_to_f(ld8(y + idx * 8), fy);
    v8_to_f(ld8(dy + idx * 8), fd);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      fd[e] = (fy[e] > 0.0f) ? fd[e] : 0.0f;
      a[e] += fd[e];
    }
    st8(dy + idx * 8, f_to_v8(fd));
  }
  if (32 % G == 0) {
    // lanes g, g + G, ... hold the same channels: one shared-memory add a
    // warp and channel instead of 32/G colliding ones (9.2 -> 5 us at 65,536
    // pixels of 32 channels); blockDim.x is then a multiple of 32
    for (int o = 16; o >= G; o >>= 1)
#pragma unroll
      for (int e = 0; e < 8; ++e) a[e] += __shfl_xor_sync(0xffffffffu, a[e], o);
    if ((threadIdx.x & 31) < G)
#pragma unroll
      for (int e = 0; e < 8; ++e) atomicAdd(&sdb[8 * g + e], a[e]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) atomicAdd(&sdb[8 * g + e], a[e]);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < c; k += blockDim.x) atomicAdd(db + k, sdb[k]);
}

// ---- 1x1 head (c = 32) --------------------------------------------------------
__global__ void k_head(int64_t npix, const bf16 *__restrict__ y, const float *__restrict__ w,
                       const float *__restrict__ b, float *__restrict__ z) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npix) return;
  float s = b[0];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    float f[8];
    v8_to_f(ld8(y + p * 32 + 8 * g), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(w[8 * g + e], f[e], s);
  }
  z[p] = s;
}

// Four threads a pixel, eight channels each (a warp reads and writes 512
// consecutive bytes); the channel sums meet by shuffles, then one shared add a
// warp and channel.  93 -> 6 us at 65,536 pixels against a thread a pixel with
// 33 colliding shared adds a thread.  The bias gradient is one number, a sum
// of terms of both signs over all pixels: a few CTAs form it besides, in FP64,
// so that it is rounded 16 times in all (592 rounded adds into a running sum
// were 1e-6 off where that sum cancels).
constexpr int kHeadBiasCtas = 16;

__global__ void __launch_bounds__(256) k_head_bwd(int64_t npix, const bf16 *__restrict__ y,
                                                  const float *__restrict__ w, const float *__restrict__ gz,
                                                  bf16 *__restrict__ dy, float *__restrict__ dw,
                                                  float *__restrict__ db) {
  __shared__ float s[32];
  __shared__ double sb[8];
  if (threadIdx.x < 32) s[threadIdx.x] = 0.0f;
  __syncthreads();
  const int g = threadIdx.x & 3;
  float a[8], ww[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    a[e] = 0.0f;
    ww[e] = w[8 * g + e];
  }
  for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < 4 * npix; q += (int64_t)gridDim.x * blockDim.x) {
    const float gp = gz[q >> 2];
    float f[8], o[8];
    v8_to_f(ld8(y + q * 8), f);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      o[e] = gp * ww[e];
      a[e] = fmaf(gp, f[e], a[e]);
    }
    st8(dy + q * 8, f_to_v8(o));
  }
  const int nb = min(kHeadBiasCtas, (int)gridDim.x);
  if ((int)blockIdx.x < nb) {
    const int64_t p1 = npix * (blockIdx.x + 1) / nb;
    double ab = 0.0;
#pragma unroll 8
    for (int64_t p = npix * blockIdx.x / nb + threadIdx.x; p < p1; p += 256) ab += (double)gz[p];
    for (int o = 16; o > 0; o >>= 1) ab += __shfl_xor_sync(0xffffffffu, ab, o);
    if ((threadIdx.x & 31) == 0) sb[threadIdx.x >> 5] = ab;
  }
  for (int o = 16; o >= 4; o >>= 1) {
#pragma unroll
    for (int e = 0; e < 8; ++e) a[e] += __shfl_xor_sync(0xffffffffu, a[e], o);
  }
  if ((threadIdx.x & 31) < 4) {
#pragma unroll
    for (int e = 0; e < 8; ++e) atomicAdd(&s[8 * g + e], a[e]);
  }
  __syncthreads();
  if (threadIdx.x < 32) atomicAdd(dw + threadIdx.x, s[threadIdx.x]);
  if (threadIdx.x == 32 && (int)blockIdx.x < nb) {
    double ab = 0.0;
    for (int q = 0; q < 8; ++q) ab += sb[q];
    atomicAdd(db, (float)ab);
  }
}

__global__ void k_loss(int64_t npix, const float *__restrict__ z, const double *__restrict__ t,
                       const double *__restrict__ scale, const int32_t *__restrict__ mask, float *__restrict__ gz,
                       double *__restrict__ acc) {
  __shared__ double sd[2];
  if (threadIdx.x < 2) sd[threadIdx.x] = 0.0;
  __syncthreads();
  const double inv_scale = scale[1];
  double a0 = 0.0, a1 = 0.0;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += (int64_t)gridDim.x * blockDim.x) {
    if (mask[p] > 0) {
      const double tt = t[p] * inv_scale;
      const double d = (double)z[p] - tt;
      gz[p] = (float)(2.0 * d);
      a0 += d * d;
      a1 += tt * tt;
    } else {
      gz[p] = 0.0f;
    }
  }
  // a shared FP64 add a warp, not a thread (18.5 -> 4 us at 16,384 pixels)
  for (int o = 16; o > 0; o >>= 1) {
    a0 += __shfl_xor_sync(0xffffffffu, a0, o);
    a1 += __shfl_xor_sync(0xffffffffu, a1, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(&sd[0], a0);
    atomicAdd(&sd[1], a1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(acc, sd[0]);
    atomicAdd(acc + 1, sd[1]);
  }
}

__global__ void k_output(int64_t npix, const float *__restrict__ z, const double *__restrict__ scale,
                         const int32_t *__restrict__ mask, double *__restrict__ out) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npix) return;
  out[p] = (mask[p] > 0) ? scale[0] * (double)z[p] : 0.0;
}

__global__ void k_adam(int64_t n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, bf16 *__restrict__ pb, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  if (pb) pb[i] = __float2bfloat16(pi);
}

// Weight gradient of a 3x3 'same' convolution on the CUDA cores, for channel
// counts that are no multiple of 8.  CTA =
// (32 output channels x 32 input channels) x a strided set of 32-pixel tiles;
// each thread accumulates 9 taps x 4 input channels of one output channel in
// registers, from tiles of dy and of the 9 shifted x staged in shared memory.
__global__ void __launch_bounds__(256) k_wgrad(int n, int h, int w, int c, int k, const bf16 *__restrict__ x,
                                               const bf16 *__restrict__ dy, float *__restrict__ dw) {
  __shared__ float sdy[32][33];
  __shared__ float sx[9][32][33];
  const int ncb = (c + 31) / 32;
  const int kb = blockIdx.x / ncb, cb = blockIdx.x % ncb;
  const int t = threadIdx.x;
  const int kk = t >> 3, cq = (t & 7) * 4;
  const int64_t np = (int64_t)n * h * w;
  float acc[9][4];
#pragma unroll
  for (int a = 0; a < 9; ++a)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[a][q] = 0.0f;
  for (int64_t p0 = (int64_t)blockIdx.y * 32; p0 < np; p0 += (int64_t)gridDim.y * 32) {
    for (int e = t; e < 32 * 32; e += 256) {
      const int pp = e >> 5, kc = e & 31;
      const int64_t p = p0 + pp;
      const int kx = kb * 32 + kc;
      sdy[pp][kc] = (p < np && kx < k) ? __bfloat162float(dy[p * k + kx]) : 0.0f;
    }
    for (int e = t; e < 9 * 32 * 32; e += 256) {
      const int tap = e >> 10, pp = (e >> 5) & 31, cc = e & 31;
      const int64_t p = p0 + pp;
      const int cx = cb * 32 + cc;
      float v = 0.0f;
      if (p < np && cx < c) {
        const int j = (int)(p % w), i = (int)((p / w) % h);
        const int64_t b = p / ((int64_t)w * h);
        const int ii = i + tap / 3 - 1, jj = j + tap % 3 - 1;
        if (ii >= 0 && ii < h && jj >= 0 && jj < w) v = __bfloat162float(x[((b * h + ii) * w + jj) * c + cx]);
      }
      sx[tap][pp][cc] = v;
    }
    __syncthreads();
#pragma unroll 4
    for (int pp = 0; pp < 32; ++pp) {
      const float d = sdy[pp][kk];
#pragma unroll
      for (int tap = 0; tap < 9; ++tap)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[tap][q] = fmaf(d, sx[tap][pp][cq + q], acc[tap][q]);
    }
    __syncthreads();
  }
  const int kx = kb * 32 + kk;
  if (kx >= k) return;
#pragma unroll
  for (int tap = 0; tap < 9; ++tap)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int cx = cb * 32 + cq + q;
      if (cx < c && acc[tap][q] != 0.0f) atomicAdd(dw + ((int64_t)kx * 9 + tap) * c + cx, acc[tap][q]);
    }
}

// The same on the tensor cores, for channel counts that are multiples of 8
// (16-byte rows): dW = sum over pixels of dy^T x, a GEMM whose K is the pixels.
// CTA = (16 MT output channels x 32 input channels) x a strided set of tiles
// of 4 image rows x 32 pixels.  The tile's dy and its x with a one-pixel rim
// are staged once (cp.async, two stages, zeros outside the image) and serve
// all nine taps: warp t owns tap t and reads x at its shift.  Pixels run along
// the rows of both operands in shared memory, so both are read transposed
// (ldmatrix.trans); rows are padded by 16 bytes, which spreads the eight rows
// of a matrix over all banks.  BF16 products, FP32 accumulation; partial sums
// of the CTAs meet in dw by atomicAdd as before.
// mma.sync and not tcgen05: the widest layer needs 2.8 GMAC a call (a few
// microseconds at either rate) and the call is bound by staging and latency;
// M is 32..64, half the smallest full-rate tcgen05 tile.
// At 4 x 128^2: 306 -> 12 us a call (mean over the network's ten layers).
constexpr int WG_ROWS = 4, WG_PIX = 32, WG_THREADS = 9 * 32;
constexpr int WG_XS = 40;  // x row in shared memory: 32 channels + 8 of padding

template <int MT>
struct WgTile {
  static constexpr int DS = 16 * MT + 8;
  bf16 x[(WG_ROWS + 2) * (WG_PIX + 2)][WG_XS];
  bf16 dy[WG_ROWS * WG_PIX][DS];
};

__device__ __forceinline__ void wg_cp16(bf16 *dst, const bf16 *src, bool valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = valid ? 16 : 0;  // 0: the 16 bytes are zero-filled, src is not read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void wg_ldsm4t(unsigned (&r)[4], const bf16 *p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

__device__ __forceinline__ void wg_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int MT>
__device__ __forceinline__ void wg_stage(WgTile<MT> &T, int tile, int ti, int tj, int h, int w, int c, int k, int kb,
                                         int cb, const bf16 *__restrict__ x, const bf16 *__restrict__ dy) {
  const int b = tile / (ti * tj), i0 = tile / tj % ti * WG_ROWS, j0 = tile % tj * WG_PIX;
  for (int e = threadIdx.x; e < (WG_ROWS + 2) * (WG_PIX + 2) * 4; e += WG_THREADS) {
    const int g = e & 3, px = e >> 2;
    const int i = i0 + px / (WG_PIX + 2) - 1, j = j0 + px % (WG_PIX + 2) - 1, ch = cb * 32 + 8 * g;
    const bool in = i >= 0 && i < h && j >= 0 && j < w && ch < c;
    wg_cp16(&T.x[px][8 * g], in ? x + (((int64_t)b * h + i) * w + j) * c + ch : x, in);
  }
  for (int e = threadIdx.x; e < WG_ROWS * WG_PIX * 2 * MT; e += WG_THREADS) {
    const int g = e % (2 * MT), px = e / (2 * MT);
    const int i = i0 + px / WG_PIX, j = j0 + px % WG_PIX, ch = kb * 16 * MT + 8 * g;
    const bool in = i < h && j < w && ch < k;
    wg_cp16(&T.dy[px][8 * g], in ? dy + (((int64_t)b * h + i) * w + j) * k + ch : dy, in);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// RAGGED: tiles may reach past the image (its tests: 2% of a training step)
template <int MT, bool RAGGED>
__global__ void __launch_bounds__(WG_THREADS) k_wgrad_mma(int n, int h, int w, int c, int k, const bf16 *__restrict__ x,
                                                          const bf16 *__restrict__ dy, float *__restrict__ dw) {
  extern __shared__ __align__(128) unsigned char wg_smem[];
  WgTile<MT> *T = reinterpret_cast<WgTile<MT> *>(wg_smem);
  const int ncb = (c + 31) / 32, kb = blockIdx.x / ncb, cb = blockIdx.x % ncb;
  const int ti = (h + WG_ROWS - 1) / WG_ROWS, tj = (w + WG_PIX - 1) / WG_PIX;
  // up to 2^31 - 1 tiles (images of one pixel): the step past the last one still fits
  const unsigned tiles = (unsigned)(n * ti * tj);
  const int lane = threadIdx.x & 31, tap = threadIdx.x >> 5, tr = tap / 3, ts = tap % 3;
  float acc[MT][4][4];
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[a][q][e] = 0.0f;
  const int apix = (lane & 7) + ((lane >> 4) & 1) * 8, ach = ((lane >> 3) & 1) * 8;
  const int bpix = (lane & 7) + ((lane >> 3) & 1) * 8, bch = ((lane >> 4) & 1) * 8;
  int stage = 0;
  if (blockIdx.y < tiles) wg_stage<MT>(T[0], (int)blockIdx.y, ti, tj, h, w, c, k, kb, cb, x, dy);
  for (unsigned at = blockIdx.y; at < tiles; at += gridDim.y, stage ^= 1) {
    const int tile = (int)at;
    const unsigned next = at + gridDim.y;
    if (next < tiles) {
      wg_stage<MT>(T[stage ^ 1], (int)next, ti, tj, h, w, c, k, kb, cb, x, dy);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const WgTile<MT> &S = T[stage];
    // Past the image's last row and column dy is zero-filled, and taps that reach
    // back inside would multiply real activations by those zeros (an infinite
    // one to NaN): rows past the end are left out, and so is the one column
    // that reaches back, at the first column's taps
    const int rows = RAGGED ? min(WG_ROWS, h - tile / tj % ti * WG_ROWS) : WG_ROWS;
    const int past = RAGGED && ts == 0 ? w - tile % tj * WG_PIX : WG_PIX;  // WG_PIX or more: none
    for (int row = 0; row < rows; ++row) {
      unsigned A[2][MT][4], B[2][2][4];
#pragma unroll
      for (int s = 0; s < 2; ++s) {  // 16 pixels of the row each
#pragma unroll
        for (int a = 0; a < MT; ++a) wg_ldsm4t(A[s][a], &S.dy[row * WG_PIX + 16 * s + apix][16 * a + ach]);
#pragma unroll
        for (int q = 0; q < 2; ++q)
          wg_ldsm4t(B[s][q], &S.x[(row + tr) * (WG_PIX + 2) + 16 * s + ts + bpix][16 * q + bch]);
      }
      if (past < WG_PIX && (past & 7) >> 1 == (lane & 3)) {  // a lane holds two pixels of every eight
        const unsigned keep = past & 1 ? 0x0000ffffu : 0xffff0000u;
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (past >> 3 == 2 * s + (e & 1)) B[s][q][e] &= keep;
      }
#pragma unroll
      for (int a = 0; a < MT; ++a)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          // the row's sum from zero, then a rounded add: the tensor cores
          // truncate what they add to, so a long chain in them drifts
          float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
          for (int s = 0; s < 2; ++s) wg_mma(t, A[s][a], B[s][q >> 1][2 * (q & 1)], B[s][q >> 1][2 * (q & 1) + 1]);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[a][q][e] += t[e];
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int kx = kb * 16 * MT + 16 * a + (lane >> 2) + 8 * (e >> 1);
        const int cx = cb * 32 + 8 * q + 2 * (lane & 3) + (e & 1);
        if (kx < k && cx < c && acc[a][q][e] != 0.0f) atomicAdd(dw + ((int64_t)kx * 9 + tap) * c + cx, acc[a][q][e]);
      }
}

// Grid: the CTAs of a (k, c) block share its tiles; two CTAs per SM in all,
// each CTA taking at least two tiles while there are enough (fewer atomics).
template <int MT>
int run_wgrad_mma(int n, int h, int w, int c, int k, const bf16 *x, const bf16 *dy, float *dw, cudaStream_t st) {
  const size_t smem = 2 * sizeof(WgTile<MT>);
  const auto fn = h % WG_ROWS || w % WG_PIX ? k_wgrad_mma<MT, true> : k_wgrad_mma<MT, false>;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return UNET_ERR_CUDA;
  const unsigned gx = (unsigned)(((k + 16 * MT - 1) / (16 * MT)) * ((c + 31) / 32));
  const int64_t tiles = (int64_t)n * ((h + WG_ROWS - 1) / WG_ROWS) * ((w + WG_PIX - 1) / WG_PIX);
  int64_t gy = (2 * 148 + gx - 1) / gx;
  if (gy > (tiles + 1) / 2) gy = (tiles + 1) / 2;
  fn<<<dim3(gx, (unsigned)gy), WG_THREADS, smem, st>>>(n, h, w, c, k, x, dy, dw);
  return launched();
}

// 3x3 'same' convolution of 8 input channels with bias and ReLU (the
// network's first layer).  Eight channels are one 16-byte row, too thin for
// the im2col loads of the tensor-core kernels (343 us at 1025^2 x 32 outputs,
// whatever the tile); the work is 4.8 GMAC and the bytes a read of 17 MB and a
// write of 67.  A warp takes 16 consecutive pixels: a tap's operand is 16 rows
// of 16 bytes straight from L1, the whole filter sits in registers (9 taps x 4
// blocks of 8 outputs), mma.sync m16n8k8 adds a tap's eight products at a
// time, in the tap order of the implicit GEMM (the same bits).  343 -> 52 us.
template <int NT>  // blocks of 8 outputs held by a warp
__global__ void __launch_bounds__(256) k_conv8(int n, int h, int w, int k, const bf16 *__restrict__ x,
                                               const bf16 *__restrict__ wt, const bf16 *__restrict__ bias,
                                               bf16 *__restrict__ y) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int k0 = blockIdx.y * 8 * NT;
  unsigned B[9][NT];
  float b0[NT], b1[NT];
#pragma unroll
  for (int q = 0; q < NT; ++q) {
    const int ko = k0 + 8 * q;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
      B[tap][q] = ko < k ? *reinterpret_cast<const unsigned *>(wt + ((int64_t)(ko + g) * 9 + tap) * 8 + 2 * t) : 0u;
    b0[q] = ko < k ? __bfloat162float(bias[ko + 2 * t]) : 0.0f;
    b1[q] = ko < k ? __bfloat162float(bias[ko + 2 * t + 1]) : 0.0f;
  }
  const int np = n * h * w, segs = (np + 15) / 16;  // < 2^31 - 16, checked by the caller
  const int step = gridDim.x * (blockDim.x / 32);
  for (int sg = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); sg < segs; sg += step) {
    const int p0 = sg * 16 + g, p1 = p0 + 8;
    unsigned A[9][2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int p = e ? p1 : p0;
      const int row = p / w, j = p - row * w, i = row % h;
      const bool up = p < np && i > 0, mid = p < np, down = p < np && i + 1 < h;
      const unsigned *xp = reinterpret_cast<const unsigned *>(x + (int64_t)p * 8 + 2 * t);  // 4 words a pixel
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        const int di = tap / 3 - 1, dj = tap % 3 - 1;
        const bool in = (di < 0 ? up : di > 0 ? down : mid) && (dj < 0 ? j > 0 : dj > 0 ? j + 1 < w : true);
        A[tap][e] = in ? __ldg(xp + ((int64_t)di * w + dj) * 4) : 0u;
      }
    }
    float acc[NT][4];
#pragma unroll
    for (int q = 0; q < NT; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[q][e] = 0.0f;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
      for (int q = 0; q < NT; ++q)
        asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
                     : "+f"(acc[q][0]), "+f"(acc[q][1]), "+f"(acc[q][2]), "+f"(acc[q][3])
                     : "r"(A[tap][0]), "r"(A[tap][1]), "r"(B[tap][q]));
#pragma unroll
    for (int q = 0; q < NT; ++q) {
      const int ko = k0 + 8 * q;
      if (ko >= k) break;
      auto relu = [](float v) { return v < 0.0f ? 0.0f : v; };
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int p = e ? p1 : p0;
        if (p >= np) continue;
        const __nv_bfloat162 o = __floats2bfloat162_rn(relu(acc[q][2 * e] + b0[q]), relu(acc[q][2 * e + 1] + b1[q]));
        *reinterpret_cast<__nv_bfloat162 *>(y + (int64_t)p * k + ko + 2 * t) = o;
      }
    }
  }
}

__global__ void k_fill(int64_t n, float *p, float v) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

__global__ void k_tobf16(int64_t n, const float *s, bf16 *d) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = __float2bfloat16(s[i]);
}

}  // namespace

// the first layer's convolution (c = 8), for unet_conv; shapes checked there
int unet_conv8(int n, int h, int w, int k, const void *x, const void *wt, const void *bias, void *y, void *stream) {
  const int64_t segs = ((int64_t)n * h * w + 15) / 16;
  const dim3 grid((unsigned)((segs + 7) / 8 < 148 * 4 ? (segs + 7) / 8 : 148 * 4), (unsigned)((k + 31) / 32));
  k_conv8<4><<<grid, 256, 0, (cudaStream_t)stream>>>(n, h, w, k, (const bf16 *)x, (const bf16 *)wt, (const bf16 *)bias,
                                                     (bf16 *)y);
  return launched();
}

extern "C" {

int unet_rms(int64_t npix, const double *r, const int32_t *mask, double *scratch, double *scale, void *stream) {
  if (npix <= 0 || !r || !mask || !scratch || !scale) return UNET_ERR_SHAPE;
  const unsigned g = capped(npix, RMS_THREADS, UNET_RMS_BLOCKS);
  unsigned int *ticket = (unsigned int *)(scratch + 2 * UNET_RMS_BLOCKS);
  k_rms<<<g, RMS_THREADS, 0, (cudaStream_t)stream>>>(npix, r, mask, scratch, ticket, scale);
  return launched();
}

int unet_features(int32_t h, int32_t w, const double *r, const double *scale, const float *feat_static,
                  void *x_out, void *stream) {
  const int64_t np = (int64_t)h * w;
  if (np <= 0) return UNET_ERR_SHAPE;
  k_features<<<nblk(np, 256), 256, 0, (cudaStream_t)stream>>>(np, r, scale, feat_static, (bf16 *)x_out);
  return launched();
}

int unet_pool(int32_t n, int32_t h, int32_t w, int32_t c, const void *x, void *y, void *stream) {
  if (n < 1 || h < 1 || w < 1 || c < 8 || c % 8) return UNET_ERR_SHAPE;
  const int64_t tot = (int64_t)n * ((h + 1) / 2) * ((w + 1) / 2) * (c / 8);
  k_pool<<<nblk(tot, 256), 256, 0, (cudaStream_t)stream>>>(n, h, w, c, (const bf16 *)x, (bf16 *)y);
  return launched();
}

int unet_pool_bwd(int32_t n, int32_t h, int32_t w, int32_t c, const void *dy, void *dx, int32_t accumulate,
                  void *stream) {
  if (n < 1 || h < 1 || w < 1 || c < 8 || c % 8) return UNET_ERR_SHAPE;
  const int64_t tot = (int64_t)n * h * w * (c / 8);
  k_pool_bwd<<<nblk(tot, 256), 256, 0, (cudaStream_t)stream>>>(n, h, w, c, (const bf16 *)dy, (bf16 *)dx,
                                                                accumulate);
  return launched();
}

int unet_upcat(int32_t n, int32_t h, int32_t w, int32_t c1, int32_t c2, const void *lo, const void *skip,
               void *y, void *stream) {
  if (n < 1 || h < 1 || w < 1 || c1 < 8 || c2 < 8 || c1 % 8 || c2 % 8) return UNET_ERR_SHAPE;
  const int64_t tot = (int64_t)n * h * w * ((c1 + c2) / 8);
  k_upcat<<<nblk(tot, 256), 256, 0, (cudaStream_t)stream>>>(n, h, w, c1, c2, (const bf16 *)lo,
                                                             (const bf16 *)skip, (bf16 *)y);
  return launched();
}

int unet_upcat_bwd(int32_t n, int32_t h, int32_t w, int32_t c1, int32_t c2, const void *dy, void *dlo,
                   void *dskip, int32_t accumulate_skip, void *stream) {
  if (n < 1 || h < 1 || w < 1 || c1 < 8 || c2 < 8 || c1 % 8 || c2 % 8) return UNET_ERR_SHAPE;
  const int64_t tlo = (int64_t)n * ((h + 1) / 2) * ((w + 1) / 2) * (c1 / 8);
  k_upcat_bwd_lo<<<nblk(tlo, 256), 256, 0, (cudaStream_t)stream>>>(n, h, w, c1, c2, (const bf16 *)dy,
                                                                    (bf16 *)dlo);
  const int64_t npix = (int64_t)n * h * w;
  k_upcat_bwd_skip<<<nblk(npix * (c2 / 8), 256), 256, 0, (cudaStream_t)stream>>>(
      npix, c1, c2, (const bf16 *)dy, (bf16 *)dskip, accumulate_skip);
  return launched();
}

int unet_relu_bwd(int64_t npix, int32_t c, const void *y, void *dy, float *db, void *stream) {
  if (npix < 1 || c < 8 || c % 8 || c > 1024) return UNET_ERR_SHAPE;
  const int G = c / 8;
  const int threads = G * (256 / G > 0 ? 256 / G : 1);
  const unsigned g = capped(npix * G, threads, 148u * 4u);
  k_relu_bwd<<<g, threads, c * sizeof(float), (cudaStream_t)stream>>>(npix, c, (const bf16 *)y, (bf16 *)dy, db);
  return launched();
}

int unet_head(int64_t npix, int32_t c, const void *y, const float *w, const float *b, float *z, void *stream) {
  if (npix < 1 || c != 32) return UNET_ERR_SHAPE;
  k_head<<<nblk(npix, 256), 256, 0, (cudaStream_t)stream>>>(npix, (const bf16 *)y, w, b, z);
  return launched();
}

int unet_head_bwd(int64_t npix, int32_t c, const void *y, const float *w, const float *gz, void *dy, float *dw,
                  float *db, void *stream) {
  if (npix < 1 || c != 32) return UNET_ERR_SHAPE;
  k_head_bwd<<<capped(4 * npix, 256, 148u * 4u), 256, 0, (cudaStream_t)stream>>>(npix, (const bf16 *)y, w, gz,
                                                                              (bf16 *)dy, dw, db);
  return launched();
}

int unet_loss(int64_t npix, const float *z, const double *target, const double *scale, const int32_t *mask,
              float *gz, double *loss2, void *stream) {
  if (npix < 1) return UNET_ERR_SHAPE;
  k_loss<<<capped(npix, 256, 148u * 8u), 256, 0, (cudaStream_t)stream>>>(npix, z, target, scale, mask, gz, loss2);
  return launched();
}

int unet_output(int64_t npix, const float *z, const double *scale, const int32_t *mask, double *out,
                void *stream) {
  if (npix < 1) return UNET_ERR_SHAPE;
  k_output<<<nblk(npix, 256), 256, 0, (cudaStream_t)stream>>>(npix, z, scale, mask, out);
  return launched();
}

int unet_adam(int64_t n, float *p, const float *g, float *m, float *v, void *p_bf16, float lr, float beta1,
              float beta2, float eps, int32_t t, void *stream) {
  if (n < 1 || t < 1) return UNET_ERR_SHAPE;
  const float c1 = 1.0f - powf(beta1, (float)t), c2 = 1.0f - powf(beta2, (float)t);
  k_adam<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(n, p, g, m, v, (bf16 *)p_bf16, lr, beta1, beta2, eps,
                                                          c1, c2);
  return launched();
}

int unet_wgrad(int32_t n, int32_t h, int32_t w, int32_t c, int32_t k, const void *x, const void *dy, float *dw,
               void *stream) {
  if (n < 1 || h < 1 || w < 1 || c < 1 || k < 1) return UNET_ERR_SHAPE;
  const int64_t np = (int64_t)n * h * w;
  // the tensor-core form wants 16-byte channel groups (and indexes tiles in
  // 32 bits); other shapes and alignments take the CUDA cores, and so do images
  // that leave nearly all of a tile empty, one pixel wide or of two in all
  // (100,000 pixels of 32 -> 32 channels, CUDA cores and tensor cores, us: 1x1
  // 273, 671; 2x1 282, 411; 1x2 284, 339; 6x1 282, 385; 16x1 280, 292)
  if (c % 8 == 0 && k % 8 == 0 && (((uintptr_t)x | (uintptr_t)dy) & 15) == 0 && np < ((int64_t)1 << 31) && w > 1 &&
      (int64_t)h * w > 2) {
    if (k > 32) return run_wgrad_mma<4>(n, h, w, c, k, (const bf16 *)x, (const bf16 *)dy, dw, (cudaStream_t)stream);
    return run_wgrad_mma<2>(n, h, w, c, k, (const bf16 *)x, (const bf16 *)dy, dw, (cudaStream_t)stream);
  }
  const unsigned gx = (unsigned)(((k + 31) / 32) * ((c + 31) / 32));
  unsigned gy = (unsigned)((np + 31) / 32);
  const unsigned cap = (148u * 8u + gx - 1) / gx;
  if (gy > cap) gy = cap;
  k_wgrad<<<dim3(gx, gy), 256, 0, (cudaStream_t)stream>>>(n, h, w, c, k, (const bf16 *)x, (const bf16 *)dy, dw);
  return launched();
}

int unet_fill_f32(int64_t n, float *p, float v, void *stream) {
  if (n < 1) return UNET_ERR_SHAPE;
  k_fill<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(n, p, v);
  return launched();
}

int unet_f32_to_bf16(int64_t n, const float *src, void *dst, void *stream) {
  if (n < 1) return UNET_ERR_SHAPE;
  k_tobf16<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(n, src, (bf16 *)dst);
  return launched();
}

}  // extern "C"
