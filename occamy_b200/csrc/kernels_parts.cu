// fp32 on the tensor cores: a value is carried as three bf16 parts, hi + mid + lo, which together hold
// its 24 mantissa bits (conv_tc_split.cu multiplies them).  A tensor is three NHWC planes one after the
// other, all hi parts first.  Convolutions write and read that form directly; the kernels here make it
// from fp32, bring it back, and pool it.  All are bound by memory: a thread moves 16 bytes of each plane.
#include "kernels.h"
#include "runtime.h"

namespace occ {

static inline int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)rt().num_sms * 64;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

__device__ __forceinline__ void split3(float v, uint16_t &hi, uint16_t &mid, uint16_t &lo) {
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  const float hf = __bfloat162float(h);
  const float r1 = fabsf(hf) < INFINITY ? v - hf : 0.0f;   // exact: the part bf16 dropped
  const __nv_bfloat16 m = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(m);
  hi = __bfloat16_as_ushort(h);
  mid = __bfloat16_as_ushort(m);
  lo = __bfloat16_as_ushort(__float2bfloat16_rn(r2));
}
__device__ __forceinline__ float join3(uint16_t hi, uint16_t mid, uint16_t lo) {
  return (__uint_as_float((uint32_t)hi << 16) + __uint_as_float((uint32_t)mid << 16)) +
         __uint_as_float((uint32_t)lo << 16);
}
// eight values of consecutive channels; x points at the hi parts, `plane` elements from plane to plane
__device__ __forceinline__ void load8(const uint16_t *x, int64_t plane, float *f) {
  uint4 u[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) u[j] = *reinterpret_cast<const uint4 *>(x + j * plane);
  const uint32_t *h = &u[0].x, *m = &u[1].x, *l = &u[2].x;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    f[2 * k] = join3(h[k] & 0xffff, m[k] & 0xffff, l[k] & 0xffff);
    f[2 * k + 1] = join3(h[k] >> 16, m[k] >> 16, l[k] >> 16);
  }
}
__device__ __forceinline__ void store8(uint16_t *y, int64_t plane, const float *f) {
  uint32_t o[3][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    uint16_t a[3], b[3];
    split3(f[2 * k], a[0], a[1], a[2]);
    split3(f[2 * k + 1], b[0], b[1], b[2]);
#pragma unroll
    for (int j = 0; j < 3; ++j) o[j][k] = a[j] | ((uint32_t)b[j] << 16);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
    *reinterpret_cast<uint4 *>(y + j * plane) = make_uint4(o[j][0], o[j][1], o[j][2], o[j][3]);
}

// x fp32 [N][C][HW] -> three planes [N][HW][Cp] (channels C..Cp-1 zero), through a 32 x 32 tile like the
// plain layout conversion.
__global__ void split3_nchw_kernel(const float *__restrict__ x, uint16_t *__restrict__ y, int C, int Cp,
                                   int HW, int64_t plane) {
  chain_begin();
  __shared__ float tile[32][33];
  const int n = blockIdx.z;
  const int c0 = blockIdx.y * 32, p0 = blockIdx.x * 32;
  const float *xn = x + (int64_t)n * C * HW;
  uint16_t *yn = y + (int64_t)n * Cp * HW;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, p = p0 + threadIdx.x;
    tile[i][threadIdx.x] = (c < C && p < HW) ? xn[(int64_t)c * HW + p] : 0.0f;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int p = p0 + i, c = c0 + threadIdx.x;
    if (p < HW && c < Cp) {
      uint16_t h, m, l;
      split3(tile[threadIdx.x][i], h, m, l);
      const int64_t at = (int64_t)p * Cp + c;
      yn[at] = h;
      yn[at + plane] = m;
      yn[at + 2 * plane] = l;
    }
  }
}

void launch_split3_nchw(const float *x, bf16 *y, int N, int C, int Cp, int H, int W, cudaStream_t s) {
  const int HW = H * W;
  if ((int64_t)N * C * HW == 0) return;
  dim3 grid((HW + 31) / 32, (Cp + 31) / 32, N), block(32, 8);
  launch_chained(split3_nchw_kernel, grid, block, 0, s, x, (uint16_t *)y, C, Cp, HW, (int64_t)N * HW * Cp);
  count(CNT_LAUNCHES);
}

// ... and back, C channels
__global__ void join3_nchw_kernel(const uint16_t *__restrict__ x, float *__restrict__ y, int C, int HW,
                                  int64_t plane) {
  chain_begin();
  __shared__ float tile[32][33];
  const int n = blockIdx.z;
  const int c0 = blockIdx.y * 32, p0 = blockIdx.x * 32;
  const uint16_t *xn = x + (int64_t)n * C * HW;
  float *yn = y + (int64_t)n * C * HW;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int p = p0 + i, c = c0 + threadIdx.x;
    const int64_t at = (int64_t)p * C + c;
    tile[i][threadIdx.x] = (p < HW && c < C) ? join3(xn[at], xn[at + plane], xn[at + 2 * plane]) : 0.0f;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, p = p0 + threadIdx.x;
    if (c < C && p < HW) yn[(int64_t)c * HW + p] = tile[threadIdx.x][i];
  }
}

void launch_join3_nchw(const bf16 *x, float *y, int N, int C, int H, int W, cudaStream_t s) {
  const int HW = H * W;
  if ((int64_t)N * C * HW == 0) return;
  dim3 grid((HW + 31) / 32, (C + 31) / 32, N), block(32, 8);
  launch_chained(join3_nchw_kernel, grid, block, 0, s, (const uint16_t *)x, y, C, HW, (int64_t)N * C * HW);
  count(CNT_LAUNCHES);
}

// x fp32 [M][K] (row length ld) -> three planes [M][Kp]
__global__ void split3_rows_kernel(const float *__restrict__ x, uint16_t *__restrict__ y, int K, int Kp,
                                   int ld, int64_t total, int64_t plane) {
  chain_begin();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int k = (int)(i % Kp);
    const int64_t m = i / Kp;
    uint16_t h, md, l;
    split3(k < K ? x[m * ld + k] : 0.0f, h, md, l);
    y[i] = h;
    y[i + plane] = md;
    y[i + 2 * plane] = l;
  }
}

void launch_split3_rows(const float *x, bf16 *y, int M, int K, int Kp, int ld, cudaStream_t s) {
  const int64_t total = (int64_t)M * Kp;
  if (total == 0) return;
  launch_chained(split3_rows_kernel, grid_for(total, 256), 256, 0, s, x, (uint16_t *)y, K, Kp, ld, total, total);
  count(CNT_LAUNCHES);
}

// Few-channel inputs: x fp32 [N][C][H][W] -> three planes [N][H][Wp][Cp], the image shifted right by pad_w
// pixels, zeros elsewhere (launch_pad_input_bf16 explains the form).  One thread per eight values.
__global__ void split3_pad_kernel(const float *__restrict__ x, uint16_t *__restrict__ y, int C, int H, int W, int Wp,
                                  int Cp, int pad_w, int64_t pieces, int64_t plane) {
  chain_begin();
  const int row = Wp * Cp / 8;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < pieces;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t nh = i / row;
    const int pc = (int)(i - nh * row);
    const int64_t n = nh / H;
    const int h = (int)(nh - n * H);
    float f[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = pc * 8 + u, w = e / Cp - pad_w, c = e % Cp;
      f[u] = c < C && w >= 0 && w < W ? x[((n * C + c) * H + h) * (int64_t)W + w] : 0.0f;
    }
    store8(y + i * 8, plane, f);
  }
}

void launch_split3_pad(const float *x, bf16 *y, int N, int C, int H, int W, int Wp, int Cp, int pad_w,
                       cudaStream_t s) {
  const int64_t plane = (int64_t)N * H * Wp * Cp;
  if (plane == 0) return;
  launch_chained(split3_pad_kernel, grid_for(plane / 8, 256), 256, 0, s, x, (uint16_t *)y, C, H, W, Wp, Cp, pad_w,
                 plane / 8, plane);
  count(CNT_LAUNCHES);
}

// Pooling, one thread per (n, p, q, 8 channels); ties and NaN as in the fp32 kernel.
__global__ void __launch_bounds__(256) pool3_kernel(const uint16_t *__restrict__ x, uint16_t *__restrict__ y, int C8,
                                                    int H, int W, int P, int Q, int kh, int kw, int pad_h, int pad_w,
                                                    int sh, int sw, bool avg, int64_t total, int64_t plane_in) {
  chain_begin();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int c8 = (int)(i % C8);
    int64_t rest = i / C8;
    const int q = (int)(rest % Q);
    rest /= Q;
    const int p = (int)(rest % P);
    const int64_t n = rest / P;
    const int h0 = max(p * sh - pad_h, 0), h1 = min(p * sh - pad_h + kh, H);
    const int w0 = max(q * sw - pad_w, 0), w1 = min(q * sw - pad_w + kw, W);
    float m[8], sum[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      m[k] = -INFINITY;
      sum[k] = 0.0f;
    }
    for (int h = h0; h < h1; ++h)
#pragma unroll 3
      for (int w = w0; w < w1; ++w) {
        float f[8];
        load8(x + (((n * H + h) * W + w) * C8 + c8) * 8, plane_in, f);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (f[k] > m[k] || f[k] != f[k]) m[k] = f[k];
          sum[k] += f[k];
        }
      }
    if (avg)
#pragma unroll
      for (int k = 0; k < 8; ++k) m[k] = sum[k] / (float)(kh * kw);
    store8(y + i * 8, total * 8, m);
  }
}

void launch_pool3(const bf16 *x, bf16 *y, int N, int C, int H, int W, int P, int Q, int kh, int kw, int pad_h,
                  int pad_w, int sh, int sw, bool avg, cudaStream_t s) {
  const int64_t total = (int64_t)N * P * Q * (C / 8);
  if (total == 0) return;
  launch_chained(pool3_kernel, grid_for(total, 256), 256, 0, s, (const uint16_t *)x, (uint16_t *)y, C / 8, H, W, P, Q,
                 kh, kw, pad_h, pad_w, sh, sw, avg, total, (int64_t)N * C * H * W);
  count(CNT_LAUNCHES);
}

// Global average pool: planes [N][HW][C] -> fp32 [N][C].  One CTA per (image, 64 channels); 16 rows of
// threads split the pixels, the partial sums meet in shared memory.
constexpr int GAP3_ROWS = 16;
__global__ void __launch_bounds__(8 * GAP3_ROWS) gap3_kernel(const uint16_t *__restrict__ x, float *__restrict__ y,
                                                            int HW, int C8, int64_t plane) {
  chain_begin();
  __shared__ float part[GAP3_ROWS][8][8];
  const int lane8 = threadIdx.x & 7, prow = threadIdx.x >> 3;
  const int c8 = blockIdx.x * 8 + lane8;
  const int64_t n = blockIdx.y;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (c8 < C8)
    for (int p = prow; p < HW; p += GAP3_ROWS) {
      float f[8];
      load8(x + ((n * HW + p) * C8 + c8) * 8, plane, f);
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] += f[k];
    }
#pragma unroll
  for (int k = 0; k < 8; ++k) part[prow][lane8][k] = acc[k];
  __syncthreads();
  if (threadIdx.x < 64) {
    const int l = threadIdx.x >> 3, k = threadIdx.x & 7;
    float sum = 0.0f;
#pragma unroll
    for (int r = 0; r < GAP3_ROWS; ++r) sum += part[r][l][k];
    if (blockIdx.x * 8 + l < C8) y[n * C8 * 8 + (blockIdx.x * 8 + l) * 8 + k] = sum / (float)HW;
  }
}

void launch_gap3(const bf16 *x, float *y, int N, int HW, int C, cudaStream_t s) {
  if ((int64_t)N * C == 0) return;
  const dim3 grid((unsigned)((C / 8 + 7) / 8), (unsigned)N);
  launch_chained(gap3_kernel, grid, 8 * GAP3_ROWS, 0, s, (const uint16_t *)x, y, HW, C / 8, (int64_t)N * HW * C);
  count(CNT_LAUNCHES);
}

// Filters, once per constant: [K][C][R][S] fp32 -> [R*S/f][3][K][Cf].  The S width taps of a few-channel
// filter are folded into its channels (f = S, Cf = Sp * Cp); otherwise f = 1 and Cf = Cp.
__global__ void pack_split3_kernel(const float *__restrict__ w, uint16_t *__restrict__ out, int K, int C, int R,
                                   int S, int Sp, int Cp, int64_t total) {
  const int Cf = Sp ? Sp * Cp : Cp;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int cf = (int)(i % Cf);
    const int k = (int)((i / Cf) % K);
    const int64_t t = i / ((int64_t)Cf * K);
    const int c = cf % Cp;
    const int r = (int)(Sp ? t : t / S), s2 = Sp ? cf / Cp : (int)(t % S);
    float v = 0.0f;
    if (c < C && s2 < S) v = w[(((int64_t)k * C + c) * R + r) * S + s2];
    uint16_t part[3];
    split3(v, part[0], part[1], part[2]);
#pragma unroll
    for (int j = 0; j < 3; ++j) out[((t * 3 + j) * K + k) * Cf + cf] = part[j];
  }
}

void launch_pack_split3(const float *w, bf16 *out, int K, int C, int R, int S, int Sp, int Cp, cudaStream_t s) {
  const int64_t total = (int64_t)K * R * (Sp ? Sp : S) * Cp;
  if (total == 0) return;
  launch_apart(pack_split3_kernel, grid_for(total, 256), 256, s, w, (uint16_t *)out, K, C, R, S, Sp, Cp, total);
  count(CNT_LAUNCHES);
}

}  // namespace occ
