// A whole inverted-residual block as one kernel: 1x1 convolution (C -> E channels), 3x3 depthwise
// convolution on the E channels (stride 1 or 2, pad 1), 1x1 convolution (E -> K), each with bias and clamp,
// and the shortcut.
//
// The block's two wide tensors (E is six times C in a MobileNetV2) are what the separate kernels spend
// their time on: at batch 128 they move 3.3 GB, against 0.5 GB of narrow tensors.  Here a CTA owns a tile
// of output pixels and walks the E channels in chunks of EC:
//     GEMM 1    the tile's input pixels with their halo, times the chunk's filters, into TMEM
//     drain     bias, clamp, 16-bit values into shared memory (zero outside the image: the depthwise
//               convolution's padding)
//     depthwise on the CUDA cores, shared memory to shared memory
//     GEMM 2    the chunk's contribution to the tile's K output channels, accumulated in TMEM
// The first bias rides on GEMM 1 as three parts that add up to its fp32 value, times a column of ones for
// the pixels inside the image.  Every value is rounded where the separate kernels round it.  The GEMMs of one chunk run while the CUDA
// cores work on the next phase, two CTAs share an SM, each walks its tiles without a gap between them, and
// the next filters and pixels travel meanwhile.  Few tiles: the chunks of a tile are shared by a cluster of
// up to eight CTAs, whose sums meet as in conv_tc_split.cu.  What bounds it is the depthwise stage (the
// half-rate multiply-add pipe and its chains) and the rate TMEM is read at; the figures are at the dispatch
// rule (ir_supported).  Two output rows at a time per thread were no faster: the registers spill.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <unordered_map>

#include "conv_tc_dev.cuh"

#include "kernels.h"
#include "runtime.h"

namespace occ {

constexpr int IR_WORKERS = 256;         // drain, depthwise, finish
constexpr int IR_THREADS = IR_WORKERS + 32;   // and a warp that loads and issues MMAs
constexpr int IR_MAX_E = 1024;
constexpr int IR_MAX_SPLITS = 8;
constexpr int IR_MAX_BLOCKS = 4;       // 128-pixel blocks of a tile's input

struct alignas(64) IrParams {
  CUtensorMap tmX, tmW1, tmB1, tmW2;
  const void *w2, *b2;                 // depthwise filter, [9][E], and bias (or null): fp16, in the bf16 mode fp32
  const float *b3;                     // or null
  const void *residual;                // like y, or null
  void *y;
  int H, W, P, Q, C, E, K, Kp;         // Kp: K padded to the MMA's 16
  int bk, kcs;                         // channels of an input tile in shared memory, such tiles
  int chunks, splits;
  int tw, th, iw, ih, segs, seg_rows;  // output tile, input tile, row segments of a column and their length
  int tiles_w, tiles_h, tiles;
  int rows_owner;                      // output pixels each CTA of a cluster finishes
  TcFastDiv div_iw, div_tw, div_w, div_h, div_g8;
  uint32_t x_bytes, ex_bytes;          // one input tile; the chunk's expanded pixels
  float floor3, lo3, hi3;              // tc_act()
  uint32_t lo1, hi1, lo2, hi2;         // bounds after the first two stages, as 16-bit pairs
  int clip1;                           // the first ones are a clip's (else hi1 is none)
  int zero_inside;                     // zero is within the first one
  int consts_ready;
  int *err;
};

namespace {

__device__ __forceinline__ void ir_cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void ir_cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void ir_st_async(uint32_t addr, uint32_t bar, const uint32_t *r) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ir_sts128(uint32_t addr, const uint32_t *r) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void ir_sts64(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ uint2 ir_lds64(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}
// Pairs of 16-bit values.  Rounding is monotonic, so clamping rounded values to rounded bounds is
// rounding the clamped value.  A clip makes a bound of NaN, as the ABI's does ...
template <bool F16>
__device__ __forceinline__ uint32_t ir_clip(uint32_t v, uint32_t lo, uint32_t hi) {
  if constexpr (F16) {
    asm("max.f16x2 %0, %0, %1;" : "+r"(v) : "r"(lo));
    asm("min.f16x2 %0, %0, %1;" : "+r"(v) : "r"(hi));
  } else {
    asm("max.bf16x2 %0, %0, %1;" : "+r"(v) : "r"(lo));
    asm("min.bf16x2 %0, %0, %1;" : "+r"(v) : "r"(hi));
  }
  return v;
}
// ... ReLU (lo 0) and no activation (lo -inf) keep it,
template <bool F16>
__device__ __forceinline__ uint32_t ir_floor(uint32_t v, uint32_t lo) {
  if constexpr (F16) asm("max.NaN.f16x2 %0, %0, %1;" : "+r"(v) : "r"(lo));
  else asm("max.NaN.bf16x2 %0, %0, %1;" : "+r"(v) : "r"(lo));
  return v;
}
// and so does any bound on the depthwise sums, where fp16 sums that overflow can make one.
template <bool F16>
__device__ __forceinline__ uint32_t ir_clamp(uint32_t v, uint32_t lo, uint32_t hi) {
  v = ir_floor<F16>(v, lo);
  if constexpr (F16) asm("min.NaN.f16x2 %0, %0, %1;" : "+r"(v) : "r"(hi));
  else asm("min.NaN.bf16x2 %0, %0, %1;" : "+r"(v) : "r"(hi));
  return v;
}
template <bool F16>
__device__ __forceinline__ uint32_t ir_cvt(float a, float b) {
  uint32_t r;
  if constexpr (F16) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
  return r;
}
__device__ __forceinline__ uint32_t ir_hfma2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ uint64_t ir_ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// The depthwise stage's arithmetic on two channels: packed fp16 in the fp16 mode, like that mode's
// depthwise kernel, packed fp32 in the bf16 mode.
template <bool F16>
struct IrPair;
template <>
struct IrPair<true> {
  typedef uint32_t T;
  static __device__ __forceinline__ void filter(uint32_t addr, T *w) {   // of four channels
    const uint2 v = ir_lds64(addr);
    w[0] = v.x;
    w[1] = v.y;
  }
  static __device__ __forceinline__ T load(uint32_t w) { return w; }
  static __device__ __forceinline__ T fma(T a, T b, T c) { return ir_hfma2(a, b, c); }
  static __device__ __forceinline__ uint32_t out(T a) { return a; }
};
template <>
struct IrPair<false> {
  typedef uint64_t T;
  static __device__ __forceinline__ void filter(uint32_t addr, T *w) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(w[0]), "=l"(w[1]) : "r"(addr));
  }
  static __device__ __forceinline__ T load(uint32_t w) { return pair16_to_f2<false>(w); }
  static __device__ __forceinline__ T fma(T a, T b, T c) { return ir_ffma2(a, b, c); }
  static __device__ __forceinline__ uint32_t out(T a) { return f2_to_bf16x2<false>(a); }
};

}  // namespace

//   EC   E channels of a chunk, 64 or 32 (whichever leaves less of the last chunk empty)
//   ST   stride of the depthwise convolution
//   CL   a tile has more than one CTA
template <int EC, int ST, bool F16, bool CL>
__global__ void __launch_bounds__(IR_THREADS, 2) ir_kernel(const __grid_constant__ IrParams p) {
  constexpr uint32_t IDESC0 = (1u << 4) | (F16 ? 0u : ((1u << 7) | (1u << 10))) | ((uint32_t)(128 >> 4) << 24);
  constexpr uint32_t PITCH = EC * 2;             // bytes of a pixel's chunk
  constexpr int QUADS = EC / 4;                  // depthwise: four channels to a lane ...
  constexpr int COLS = 32 / QUADS;               // ... and this many columns to a warp
  constexpr uint32_t DW_BYTES = 128 * PITCH;
  constexpr uint32_t WD_ROW = EC * (F16 ? 2 : 4), WD_STAGE = 10 * WD_ROW;   // depthwise filter and bias of a chunk
  constexpr uint32_t ONE_ROW = 32;               // bytes of a row of the bias step's operands
  typedef IrPair<F16> V;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t s0 = smem_u32(smem_raw);
  if ((s0 & 1023u) != 0u) {
    if (threadIdx.x == 0) atomicExch(p.err, 1007);
    return;
  }
  const int splits = CL ? p.splits : 1;
  const int pin = p.iw * p.ih, blocks = (pin + 127) >> 7, pout = p.tw * p.th;
  const uint32_t w1_tile = EC * (uint32_t)p.bk * 2u, w1_bytes = (uint32_t)p.kcs * w1_tile + EC * ONE_ROW;
  const uint32_t w2_bytes = (uint32_t)p.Kp * PITCH;
  const uint32_t w1_stage = (w1_bytes + 1023u) & ~1023u, w2_stage = (w2_bytes + 1023u) & ~1023u;
  const uint32_t sX = s0, sOne = sX + (uint32_t)p.kcs * p.x_bytes, sW1 = sOne + (uint32_t)blocks * 128u * ONE_ROW;
  const uint32_t sW2 = sW1 + 2u * w1_stage, sDW = sW2 + 2u * w2_stage, sEX = sDW + DW_BYTES;
  // the K sums of the tile's pixels, pushed here by the cluster's CTAs
  const uint32_t sS = sEX + p.ex_bytes, sums_pitch = (uint32_t)p.Kp * 4u;
  uint8_t *misc = smem_raw + (sS + (CL ? (uint32_t)(splits * p.rows_owner) * sums_pitch : 0u) - s0);
  uint64_t *bars = reinterpret_cast<uint64_t *>(misc);
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t x_bar = bar0, w1_bar = bar0 + 8, w2_bar = bar0 + 24, g1_bar = bar0 + 40, g2_bar = bar0 + 48,
                 sums_bar = bar0 + 56, drained_bar = bar0 + 64, dwdone_bar = bar0 + 72;
  volatile uint32_t *tmem_holder = reinterpret_cast<volatile uint32_t *>(bars + 10);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 10) + 1;
  const uint32_t sWD = bar0 + 96;                       // two stages
  float *b3_s = reinterpret_cast<float *>(misc + 96 + 2 * WD_STAGE);   // Kp floats

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int quad = warp & 3, part = warp >> 2;
  const int rank = CL ? (int)cluster_ctarank() : 0;
  const int total_tiles = p.tiles, first_tile = (int)blockIdx.x / splits;
  const int step_tiles = CL ? total_tiles : (int)gridDim.x;
  const uint32_t d2_col = (uint32_t)blocks * EC, need = d2_col + (uint32_t)p.Kp;
  const uint32_t cols = need <= 64u ? 64u : need <= 128u ? 128u : need <= 256u ? 256u : 512u;
  int err_code = 0;
  struct Tile {
    int q0, p0, n;
  };
  auto tile_of = [&](int t) {
    const uint32_t r = tc_fdiv((uint32_t)t, p.div_w);
    Tile o;
    o.q0 = (t - (int)r * p.tiles_w) * p.tw;
    o.n = (int)tc_fdiv(r, p.div_h);
    o.p0 = ((int)r - o.n * p.tiles_h) * p.th;
    return o;
  };

  if (threadIdx.x == 0) {
    tma_prefetch_map(&p.tmX);
    tma_prefetch_map(&p.tmW1);
    tma_prefetch_map(&p.tmB1);
    tma_prefetch_map(&p.tmW2);
#pragma unroll
    for (int i = 0; i < 8; ++i) mbar_init(bar0 + 8u * i, 1);
    mbar_init(drained_bar, IR_WORKERS / 32);
    mbar_init(dwdone_bar, IR_WORKERS / 32);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if constexpr (CL) {
      const int m = min(p.rows_owner, pout - rank * p.rows_owner);
      mbar_expect_tx(sums_bar, m > 0 ? (uint32_t)(splits * m) * sums_pitch : 0u);
    }
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void *)tmem_holder)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CL) ir_cluster_arrive();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  const uint32_t d1 = tmem, d2 = tmem + d2_col;

  // Chunks are numbered through the CTA's tiles: chunk g is number g % mine of tile g / mine and uses filter
  // stages g & 1.
  const int mine = (p.chunks - rank + splits - 1) / splits;
  const int chunks_all = mine * ((total_tiles - first_tile + step_tiles - 1) / step_tiles);
  auto chunk_e0 = [&](int c) { return (rank + c * splits) * EC; };

  if (warp == IR_WORKERS / 32) {
    // Loads and products, in a warp of their own: done by one of the workers they kept all of them waiting
    // at the next barrier for a third of a chunk's time.
    auto load_w1 = [&](int g, int c) {
      const uint32_t st = (uint32_t)(g & 1), bar = w1_bar + 8u * st, dst = sW1 + st * w1_stage;
      expect_tx_warp(bar, w1_bytes);
      for (int k = 0; k < p.kcs; ++k)
        load_3d_warp(dst + (uint32_t)k * w1_tile, &p.tmW1, bar, k * p.bk, chunk_e0(c), 0);
      load_3d_warp(dst + (uint32_t)p.kcs * w1_tile, &p.tmB1, bar, 0, chunk_e0(c), 0);
    };
    auto load_w2 = [&](int g, int c) {
      const uint32_t st = (uint32_t)(g & 1), bar = w2_bar + 8u * st;
      const int e0 = chunk_e0(c), n = min(EC, p.E - e0) * (F16 ? 2 : 4);
      const int rows = p.b2 ? 10 : 9;
      expect_tx_warp(bar, w2_bytes + (uint32_t)(rows * n));
      load_3d_warp(sW2 + st * w2_stage, &p.tmW2, bar, e0, 0, 0);
      for (int t = 0; t < rows; ++t)
        bulk_load_warp(sWD + st * WD_STAGE + (uint32_t)t * WD_ROW,
                     reinterpret_cast<const uint8_t *>(t < 9 ? p.w2 : p.b2) + ((int64_t)(t % 9) * p.E + e0) * (F16 ? 2 : 4),
                     (uint32_t)n, bar);
    };
    auto load_x = [&](int t) {
      const Tile o = tile_of(t);
      expect_tx_warp(x_bar, (uint32_t)(p.kcs * pin * p.bk) * 2u);
      for (int k = 0; k < p.kcs; ++k)
        load_4d_warp(sX + (uint32_t)k * p.x_bytes, &p.tmX, x_bar, k * p.bk, o.q0 * ST - 1, o.p0 * ST - 1, o.n);
    };
    auto gemm1 = [&](int g) {
      const uint32_t w = sW1 + (uint32_t)(g & 1) * w1_stage;
      const uint64_t a0 = make_smem_desc(sX, p.bk), b0 = make_smem_desc(w, p.bk);
      const uint64_t a1 = make_smem_desc(sOne, 16), b1 = make_smem_desc(w + (uint32_t)p.kcs * w1_tile, 16);
      const uint32_t a_hi = (uint32_t)(a0 >> 32), b_hi = (uint32_t)(b0 >> 32);
      const uint32_t a_block = (128u * p.bk * 2u) >> 4, x_step = p.x_bytes >> 4, w_step = w1_tile >> 4;
      const int kks = p.bk / 16;
#pragma unroll 1
      for (int b = 0; b < blocks; ++b) {
        const uint32_t d = d1 + (uint32_t)(b * EC);
        // the bias: a column of ones per part of it, zero for pixels outside the image
        mma_warp(d, (uint32_t)a1 + (uint32_t)b * ((128u * ONE_ROW) >> 4), (uint32_t)(a1 >> 32), (uint32_t)b1,
                 (uint32_t)(b1 >> 32), IDESC0 | ((uint32_t)(EC >> 3) << 17), 0u);
#pragma unroll 1
        for (int k = 0; k < p.kcs; ++k)
#pragma unroll 4
          for (int kk = 0; kk < kks; ++kk)
            mma_warp(d, (uint32_t)a0 + (uint32_t)k * x_step + (uint32_t)b * a_block + 2u * kk, a_hi,
                     (uint32_t)b0 + (uint32_t)k * w_step + 2u * kk, b_hi, IDESC0 | ((uint32_t)(EC >> 3) << 17), 1u);
      }
      commit_warp(g1_bar);
    };
    auto gemm2 = [&](int g, int c) {
      const uint64_t a0 = make_smem_desc(sDW, EC), b0 = make_smem_desc(sW2 + (uint32_t)(g & 1) * w2_stage, EC);
#pragma unroll
      for (int kk = 0; kk < EC / 16; ++kk)
        mma_warp(d2, (uint32_t)a0 + 2u * kk, (uint32_t)(a0 >> 32), (uint32_t)b0 + 2u * kk, (uint32_t)(b0 >> 32),
                 IDESC0 | ((uint32_t)(p.Kp >> 3) << 17), (c | kk) ? 1u : 0u);
      commit_warp(g2_bar);
    };
    auto first_filters = [&]() {
      load_w1(0, 0);
      load_w2(0, 0);
      if (chunks_all > 1) load_w2(1, mine > 1 ? 1 : 0);
    };
    if (p.consts_ready) first_filters();
    pdl_launch_dependents();
    pdl_wait();
    if (!p.consts_ready) first_filters();
    int c = 0, t = first_tile, xs = 0;   // chunk g is number c of tile t, the CTA's xs-th
#pragma unroll 1
    for (int g = 0; g <= chunks_all; ++g) {
      const int before = c == 0 ? mine - 1 : c - 1, after = c + 1 == mine ? 0 : c + 1;
      if (g < chunks_all) {
        // the last chunk has been drained, this tile's ones are there
        if (!mbar_wait_warp(drained_bar, g & 1, abort_flag)) err_code = 1;
        if (err_code) break;
        tc_fence_after();
        if (c == 0) load_x(t);
        if (g + 1 < chunks_all) load_w1(g + 1, after);
        if (!mbar_wait_warp(w1_bar + 8u * (g & 1), (g >> 1) & 1, abort_flag)) err_code = 2;
        if (c == 0 && !mbar_wait_warp(x_bar, xs & 1, abort_flag)) err_code = 3;
        if (err_code) break;
        tc_fence_after();
        gemm1(g);
        if (g >= 2) {   // these filters replace those of chunk g - 2
          if (!mbar_wait_warp(g2_bar, g & 1, abort_flag)) err_code = 4;
          if (err_code) break;
          load_w2(g, c);
        }
      }
      if (g >= 1) {
        const int h = g - 1;
        if (!mbar_wait_warp(dwdone_bar, h & 1, abort_flag)) err_code = 5;
        if (!mbar_wait_warp(w2_bar + 8u * (h & 1), (h >> 1) & 1, abort_flag)) err_code = 6;
        if (err_code) break;
        tc_fence_after();
        gemm2(h, before);
      }
      c = after;
      if (c == 0) {
        t += step_tiles;
        ++xs;
      }
    }
    if (err_code) *abort_flag = 1;
  }

  if (warp < 8) {
    auto final_bias = [&]() {
      for (int i = threadIdx.x; i < p.Kp; i += IR_WORKERS) b3_s[i] = p.b3 && i < p.K ? p.b3[i] : 0.0f;
    };
    // ones of a tile's input pixels, three to a row, for the bias parts
    auto ones = [&](const Tile &o) {
      for (int px = threadIdx.x; px < blocks * 128; px += IR_WORKERS) {
        const int y = (int)tc_fdiv((uint32_t)px, p.div_iw), x = px - y * p.iw;
        const bool in = px < pin && (unsigned)(o.p0 * ST - 1 + y) < (unsigned)p.H && (unsigned)(o.q0 * ST - 1 + x) < (unsigned)p.W;
        const uint32_t one = F16 ? 0x3c00u : 0x3f80u;
        const uint32_t v[4] = {in ? one | (one << 16) : 0u, in ? one : 0u, 0u, 0u}, z[4] = {0u, 0u, 0u, 0u};
        const uint32_t row = sOne + (uint32_t)px * ONE_ROW, sw = (((uint32_t)px >> 2) & 1u) << 4;   // 32-byte swizzle
        ir_sts128(row + sw, v);
        ir_sts128(row + (16u ^ sw), z);
      }
    };
    Tile o = tile_of(first_tile);
    ones(o);
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(drained_bar);
    if (p.consts_ready) final_bias();
    pdl_launch_dependents();
    pdl_wait();
    if (!p.consts_ready) final_bias();

    const int dq = lane % QUADS, dsub = lane / QUADS;   // depthwise: channels 4 * dq .. + 3, column within the warp's
    const int row0 = rank * p.rows_owner, g8 = p.K / 8, items = min(p.rows_owner, pout - row0) * g8;
    // a column of a row segment: where its window is in the expanded pixels, where its results go
    struct Unit {
      uint32_t col[3], dst;
      int rows;
    };
    const uint32_t down = (uint32_t)p.iw * PITCH, dst_down = (uint32_t)p.tw * PITCH;
    auto unit = [&](int u) {
      const int seg = (int)tc_fdiv((uint32_t)u, p.div_tw), q = u - seg * p.tw, r0 = seg * p.seg_rows;
      Unit w;
      w.rows = min(p.seg_rows, p.th - r0);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const uint32_t x = (uint32_t)(q * ST + j), key = EC == 64 ? x & 7u : (x >> 1) & 3u;
        w.col[j] = sEX + ((uint32_t)(r0 * ST * p.iw) + x) * PITCH + ((((uint32_t)dq >> 1) ^ key) << 4) + (dq & 1) * 8u;
      }
      // tw is a multiple of eight: every row of the tile has this column's swizzle
      const uint32_t m = (uint32_t)(r0 * p.tw + q), sw = EC == 64 ? m & 7u : (m >> 1) & 3u;
      w.dst = sDW + m * PITCH + ((((uint32_t)dq >> 1) ^ sw) << 4) + (dq & 1) * 8u;
      return w;
    };
    const Unit first_unit = unit(warp * COLS + dsub);
    int c = 0, t = first_tile;
#pragma unroll 1
    for (int g = 0; g < chunks_all; ++g) {
      const bool last = c + 1 == mine;
      if (!mbar_wait(g1_bar, g & 1, abort_flag)) err_code = 7;
      tc_fence_after();
      // drain: this thread's pixel of each block, half of the chunk's channels
#pragma unroll 1
      for (int b = 0; b < blocks; ++b) {
        if (b * 128 + quad * 32 >= pin) break;   // the same for the whole warp
        const int px = b * 128 + quad * 32 + lane;
        uint32_t r[EC / 2];
        tc_ld<EC / 2>(d1 + ((uint32_t)(quad * 32) << 16) + (uint32_t)(b * EC + part * (EC / 2)), r);
        const int y = (int)tc_fdiv((uint32_t)px, p.div_iw), x = px - y * p.iw;
        const uint32_t row = sEX + (uint32_t)px * PITCH;
        const uint32_t key = EC == 64 ? (uint32_t)x & 7u : ((uint32_t)x >> 1) & 3u;
        uint32_t lo = p.lo1, hi = p.hi1;
        if (!p.zero_inside) {   // the clamp would lift the padding's zeros
          const bool in = (unsigned)(o.p0 * ST - 1 + y) < (unsigned)p.H && (unsigned)(o.q0 * ST - 1 + x) < (unsigned)p.W;
          lo = in ? lo : 0u;
          hi = in ? hi : 0u;
        }
        tc_ld_wait();
#pragma unroll
        for (int k = 0; k < EC / 16; ++k) {
          uint32_t v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            v[j] = ir_cvt<F16>(__uint_as_float(r[k * 8 + 2 * j]), __uint_as_float(r[k * 8 + 2 * j + 1]));
          if (p.clip1) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = ir_clip<F16>(v[j], lo, hi);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = ir_floor<F16>(v[j], lo);
          }
          if (px < pin) ir_sts128(row + (((uint32_t)(part * (EC / 16) + k) ^ key) << 4), v);
        }
      }
      Tile nx = o;
      if (last && t + step_tiles < total_tiles) {
        nx = tile_of(t + step_tiles);
        ones(nx);
        fence_async_smem();
      }
      tc_fence_before();
      epi_bar();
      if (lane == 0 && g + 1 < chunks_all) mbar_arrive(drained_bar);
      // the depthwise results of the chunk before have been multiplied; this chunk's filter is there
      if (g >= 1 && !mbar_wait(g2_bar, (g - 1) & 1, abort_flag)) err_code = 8;
      if (!mbar_wait(w2_bar + 8u * (g & 1), (g >> 1) & 1, abort_flag)) err_code = 9;
      {
        typename V::T wt[9][2], bt[2];
        const uint32_t wd = sWD + (uint32_t)(g & 1) * WD_STAGE + (uint32_t)dq * (F16 ? 8u : 16u);
#pragma unroll
        for (int k = 0; k < 9; ++k) V::filter(wd + (uint32_t)k * WD_ROW, wt[k]);
        if (p.b2) V::filter(wd + 9u * WD_ROW, bt);
        else bt[0] = bt[1] = 0;
        const int units = p.tw * p.segs;
        // The last chunk may reach past the E channels (E is a multiple of 16: a thread's four are all in or all
        // out).  No filter was loaded for those, and their results meet the zeros that fill up the second
        // filter: they have to be zero, not whatever the sums make of it.
        const bool beyond = chunk_e0(c) + 4 * dq >= p.E;
#pragma unroll 1
        for (int u = warp * COLS + dsub; u < units; u += 8 * COLS) {   // (tw is a multiple of eight: no warp is split)
          Unit w = u < 8 * COLS ? first_unit : unit(u);
          if (beyond) {
            for (; w.rows > 0; --w.rows, w.dst += dst_down) ir_sts64(w.dst, 0u, 0u);
            continue;
          }
          typename V::T win[3][3][2];   // [input row % 3][column][channel pair]
          auto load = [&](int slot) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const uint2 v = ir_lds64(w.col[j]);
              win[slot][j][0] = V::load(v.x);
              win[slot][j][1] = V::load(v.y);
              w.col[j] += down;
            }
          };
          auto output = [&](int a, int b, int d) {   // window slots of the three filter rows
            typename V::T s[2] = {bt[0], bt[1]};
#pragma unroll
            for (int j = 0; j < 9; ++j)   // row by row, like the kernel for this stage alone
#pragma unroll
              for (int h = 0; h < 2; ++h)
                s[h] = V::fma(win[j < 3 ? a : j < 6 ? b : d][j % 3][h], wt[j][h], s[h]);
            ir_sts64(w.dst, ir_clamp<F16>(V::out(s[0]), p.lo2, p.hi2), ir_clamp<F16>(V::out(s[1]), p.lo2, p.hi2));
            w.dst += dst_down;
          };
          if (ST == 1) {
            load(0);
            load(1);
#pragma unroll 1
            while (true) {
              load(2);
              output(0, 1, 2);
              if (--w.rows <= 0) break;
              load(0);
              output(1, 2, 0);
              if (--w.rows <= 0) break;
              load(1);
              output(2, 0, 1);
              if (--w.rows <= 0) break;
            }
          } else {
            load(0);
#pragma unroll 1
            while (true) {
              load(1);
              load(2);
              output(0, 1, 2);
              if (--w.rows <= 0) break;
              load(1);
              load(0);
              output(2, 1, 0);
              if (--w.rows <= 0) break;
            }
          }
        }
      }
      fence_async_smem();
      epi_bar();
      if (lane == 0) mbar_arrive(dwdone_bar);
      c = last ? 0 : c + 1;
      if (!last) continue;

      if constexpr (!CL) {
        // This thread's pixel, sixteen channels at a time, every second sixteen; nothing of it passes through
        // shared memory, so that no warp waits for another.
        const int row = quad * 32 + lane, y = (int)tc_fdiv((uint32_t)row, p.div_tw), x = row - y * p.tw;
        const bool on = row < pout && o.p0 + y < p.P && o.q0 + x < p.Q;
        const int64_t at = (((int64_t)o.n * p.P + o.p0 + y) * p.Q + o.q0 + x) * p.K;
        constexpr int AHEAD = 2;   // sixteens whose shortcut values are fetched while the last products are made
        uint4 early[AHEAD][2];
        auto shortcut = [&](int k, uint4 *v) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
            if (on && k * 16 + h * 8 < p.K)
              v[h] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p.residual) + at + k * 16 + h * 8);
        };
        if (p.residual)
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) shortcut(part + 2 * u, early[u]);
        __syncwarp();
        if (!mbar_wait(g2_bar, g & 1, abort_flag)) err_code = 10;
        tc_fence_after();
        auto finish = [&](int k, const uint4 *rs) {
          uint32_t r[16];
          tc_ld<16>(d2 + ((uint32_t)(quad * 32) << 16) + (uint32_t)(k * 16), r);
          tc_ld_wait();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t w[4] = {rs[h].x, rs[h].y, rs[h].z, rs[h].w};
            uint32_t out[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float a = 0.f, b = 0.f;
              if (p.residual) f2_unpack(pair16_to_f2<F16>(w[j]), a, b);
              const float2 bias = *reinterpret_cast<const float2 *>(b3_s + k * 16 + h * 8 + 2 * j);
              a += __uint_as_float(r[h * 8 + 2 * j]) + bias.x;
              b += __uint_as_float(r[h * 8 + 2 * j + 1]) + bias.y;
              out[j] = f2_to_bf16x2<F16>(f2_pack(tc_act(a, p.floor3, p.lo3, p.hi3), tc_act(b, p.floor3, p.lo3, p.hi3)));
            }
            if (on && k * 16 + h * 8 < p.K && !err_code)
              *reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(p.y) + at + k * 16 + h * 8) =
                  make_uint4(out[0], out[1], out[2], out[3]);
          }
          __syncwarp();
        };
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
          if (part + 2 * u < p.Kp / 16) finish(part + 2 * u, early[u]);
#pragma unroll 1
        for (int k = part + 2 * AHEAD; k < p.Kp / 16; k += 2) {
          uint4 v[2];
          if (p.residual) shortcut(k, v);
          __syncwarp();
          finish(k, v);
        }
        tc_fence_before();
      } else {
      // What this thread finishes first: its shortcut values are fetched while the last products are made.
      auto item_at = [&](int it, int &m, int &ch) -> int64_t {   // pixel and channel of an item, its place in y; -1: none
        const int r = (int)tc_fdiv((uint32_t)it, p.div_g8);
        m = row0 + r;
        ch = (it - r * g8) * 8;
        const int y = (int)tc_fdiv((uint32_t)m, p.div_tw), x = m - y * p.tw;
        if (it >= items || o.p0 + y >= p.P || o.q0 + x >= p.Q) return -1;
        return (((int64_t)o.n * p.P + o.p0 + y) * p.Q + o.q0 + x) * p.K + ch;
      };
      constexpr int AHEAD = 2;
      uint4 early[AHEAD];
      if (p.residual)
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          int m, ch;
          const int64_t at = item_at((int)threadIdx.x + u * IR_WORKERS, m, ch);
          if (at >= 0) early[u] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p.residual) + at);
        }
      __syncwarp();
      if (!mbar_wait(g2_bar, g & 1, abort_flag)) err_code = 10;
      tc_fence_after();
      ir_cluster_wait();   // every CTA of the cluster has started
      // sums of this thread's pixel to the CTA that finishes it, sixteen channels at a time
      {
        const int row = quad * 32 + lane;
        uint32_t to = 0, to_bar = 0;
        const int owner = row / p.rows_owner;
        if (row < pout) {
          to = cluster_map(sS, (uint32_t)owner) + (uint32_t)(rank * p.rows_owner + row - owner * p.rows_owner) * sums_pitch;
          to_bar = cluster_map(sums_bar, (uint32_t)owner);
        }
        const bool on = row < pout && !err_code;
        for (int k = part; k < p.Kp / 16; k += 2) {
          uint32_t r[16];
          tc_ld<16>(d2 + ((uint32_t)(quad * 32) << 16) + (uint32_t)(k * 16), r);
          tc_ld_wait();
          if (on)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t at = to + (((uint32_t)(k * 4 + j)) ^ ((uint32_t)row & 3u)) * 16u;
              ir_st_async(at, to_bar, r + 4 * j);
            }
          __syncwarp();
        }
      }
      if (!err_code && !mbar_wait(sums_bar, 0, abort_flag)) err_code = 11;
      // finish: eight channels of a pixel to a thread, neighbouring threads on neighbouring channels
      auto finish = [&](int it, const uint4 *early) {
        int m, ch;
        const int64_t at = item_at(it, m, ch);
        if (at < 0 || err_code) return;
        const int r = m - row0;
        uint4 rs = make_uint4(0, 0, 0, 0);
        if (p.residual) rs = early ? *early : *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p.residual) + at);
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = b3_s[ch + j];
        for (int k = 0; k < splits; ++k) {
          const uint8_t *b = smem_raw + (sS - s0) + (size_t)(k * p.rows_owner + r) * sums_pitch;
          const float4 x = *reinterpret_cast<const float4 *>(b + (((uint32_t)(ch / 4)) ^ ((uint32_t)m & 3u)) * 16u);
          const float4 y = *reinterpret_cast<const float4 *>(b + (((uint32_t)(ch / 4 + 1)) ^ ((uint32_t)m & 3u)) * 16u);
          v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
          v[4] += y.x; v[5] += y.y; v[6] += y.z; v[7] += y.w;
        }
        const uint32_t w[4] = {rs.x, rs.y, rs.z, rs.w};
        uint32_t out[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float a = 0.f, b = 0.f;
          if (p.residual) f2_unpack(pair16_to_f2<F16>(w[j]), a, b);
          out[j] = f2_to_bf16x2<F16>(f2_pack(tc_act(v[2 * j] + a, p.floor3, p.lo3, p.hi3), tc_act(v[2 * j + 1] + b, p.floor3, p.lo3, p.hi3)));
        }
        *reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(p.y) + at) = make_uint4(out[0], out[1], out[2], out[3]);
      };
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) finish((int)threadIdx.x + u * IR_WORKERS, early + u);
      for (int it = (int)threadIdx.x + AHEAD * IR_WORKERS; it < items; it += IR_WORKERS) finish(it, nullptr);
      }
      o = nx;
      t += step_tiles;
    }
  }
  __syncwarp();
  if constexpr (CL) {
    if (warp >= 8) ir_cluster_wait();
  }
  if (err_code) {
    atomicExch(p.err, 1100 + err_code);
    *abort_flag = 1;
    for (int i = 0; i < 50; ++i) __nanosleep(20000);   // copies in flight land before memory goes
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CL) {
    // one that gave up stays until the others have gone (each of their waits is bounded)
    if (*abort_flag) {
      ir_cluster_arrive();
      ir_cluster_wait();
    }
  }
  if (warp == 3)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
}

template <bool F16>
__global__ void pack_bias3_kernel(const float *__restrict__ b, uint16_t *__restrict__ out, int E) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  float v = b[e];
  for (int j = 0; j < 16; ++j) {
    uint16_t bits = 0;
    if (j < 3) {
      // (a value beyond fp16's range is spread over the parts)
      const float part = F16 ? fminf(fmaxf(v, -65504.0f), 65504.0f) : v;
      const uint32_t w = ir_cvt<F16>(part, 0.0f) & 0xffffu;
      float back, zero;
      f2_unpack(pair16_to_f2<F16>(w), back, zero);
      bits = (uint16_t)w;
      v -= back;
    }
    out[e * 16 + j] = bits;
  }
}
void launch_pack_bias3(const float *b, bf16 *out, int E, bool f16, cudaStream_t s) {
  if (f16) launch_apart(pack_bias3_kernel<true>, (E + 127) / 128, 128, s, b, (uint16_t *)out, E);
  else launch_apart(pack_bias3_kernel<false>, (E + 127) / 128, 128, s, b, (uint16_t *)out, E);
  count(CNT_LAUNCHES);
}

// fp32 [E][T] -> fp16 [T][E]: the depthwise filter (T = 9) or its bias (T = 1) in the fp16 mode
__global__ void pack_ir_half_kernel(const float *__restrict__ w, uint16_t *__restrict__ out, int E, int T) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T * E) return;
  const int t = i / E, e = i - t * E;
  out[i] = (uint16_t)(ir_cvt<true>(w[e * T + t], 0.0f) & 0xffffu);
}
void launch_pack_ir_half(const float *w, void *out, int E, int T, cudaStream_t s) {
  launch_apart(pack_ir_half_kernel, (T * E + 255) / 256, 256, s, w, (uint16_t *)out, E, T);
  count(CNT_LAUNCHES);
}

// ---- host side ----------------------------------------------------------------------
namespace {

struct IrChoice {
  int ec, tw, th, segs, seg_rows, splits;
  size_t smem;
  double us;   // modelled; < 0: not possible
};

size_t ir_smem(int ec, int kcs, int bk, int pin, int pout, int Kp, int splits, bool f16,
               uint32_t *x_bytes, uint32_t *ex_bytes) {
  auto up = [](size_t v) { return (v + 1023) / 1024 * 1024; };
  const size_t x = up((size_t)pin * bk * 2), ex = up((size_t)pin * ec * 2);
  if (x_bytes) *x_bytes = (uint32_t)x;
  if (ex_bytes) *ex_bytes = (uint32_t)ex;
  const int blocks = (pin + 127) / 128, owner = (pout + splits - 1) / splits;
  const size_t front = kcs * x + (size_t)blocks * 128 * 32 + 2 * up((size_t)ec * (kcs * bk * 2 + 32)) + 2 * up((size_t)Kp * ec * 2);
  const size_t pixels = 128 * ec * 2 + ex, sums = (size_t)splits * owner * Kp * 4;
  const size_t body = front + pixels + (splits > 1 ? sums : 0);
  // the MMA reads whole 128-pixel blocks of the last input tile
  const size_t reach = (size_t)(kcs - 1) * x + (size_t)blocks * 128 * bk * 2;
  return (body > reach ? body : reach) + 96 + (size_t)20 * ec * (f16 ? 2 : 4) + (size_t)Kp * 4;
}

// Tile, chunk width and cluster size with the lowest modelled time.  The model is a fit to clock readings
// inside the kernel, per chunk and with one or two CTAs on an SM: 9.6 cycles and channel to drain 32 pixels of
// a TMEM quadrant (16 bytes a cycle), 210 or 295 cycles per row of the depthwise stage, and what a chunk
// spends at its barriers.
IrChoice ir_choose(int N, int C, int E, int K, int P, int Q, int stride, bool f16, int nsm) {
  IrChoice best{0, 0, 0, 0, 0, 0, 0, -1.0};
  const int Cp = (C + 15) / 16 * 16, bk = Cp <= 16 ? 16 : Cp <= 32 ? 32 : 64, kcs = (Cp + bk - 1) / bk;
  const int Kp = (K + 15) / 16 * 16;
  for (int ec = 64; ec >= 32; ec -= 32) {
    const int chunks = (E + ec - 1) / ec, slots = 8 * 128 / ec;
    for (int tw = 8; tw <= Q + 7 && tw <= 32; tw += 8)
      for (int th = 2; th <= P + 1 && tw * th <= 128; ++th) {
        const int iw = (tw - 1) * stride + 3, ih = (th - 1) * stride + 3, pin = iw * ih;
        const int blocks = (pin + 127) / 128;
        if (blocks > IR_MAX_BLOCKS || blocks * ec + Kp > 512) continue;
        const int groups = ((pin + 31) / 32 + 3) / 4;   // 32-pixel groups of the fullest TMEM quadrant
        int segs = 1, rows = 0;                          // rows: that a warp computes
        for (int g = 1; g <= 8 && g <= th; ++g) {
          const int r = (th + g - 1) / g, n = r * ((tw * g + slots - 1) / slots);
          if ((g - 1) * r < th && (rows == 0 || n < rows)) rows = n, segs = g;
        }
        const long tiles = (long)((Q + tw - 1) / tw) * ((P + th - 1) / th) * N;
        for (int s = 1; s <= IR_MAX_SPLITS && s <= chunks; ++s) {
          const size_t smem = ir_smem(ec, kcs, bk, pin, tw * th, Kp, s, f16, nullptr, nullptr);
          if (smem > TC_SMEM_LIMIT) break;
          const int res = smem <= TC_SMEM_DUO && blocks * ec + Kp <= 256 ? 2 : 1;
          const long ctas = tiles * s;
          if (s > 1 && ctas > (long)(nsm - nsm / 9) * res) break;
          const int r = ctas > nsm ? res : 1;
          const double waves = (double)((ctas + (long)nsm * r - 1) / ((long)nsm * r));
          const double row = (f16 ? 1.0 : 1.6) * (stride == 2 ? 1.3 : 1.0) * (r == 2 ? 295 : 210);
          const double chunk = groups * (ec * 9.6 + 40) + rows * row + (r == 2 ? 2300 : 1700);
          const double us = (waves * (((chunks + s - 1) / s) * chunk + 3300) + 5000 + (s > 1 ? 1500 : 0)) / 1850.0;
          if (best.us < 0 || us < best.us) best = IrChoice{ec, tw, th, segs, (th + segs - 1) / segs, s, smem, us};
        }
      }
  }
  return best;
}

struct IrKey {
  IrArgs a;
  bool operator==(const IrKey &o) const { return memcmp(&a, &o.a, sizeof(a)) == 0; }
};
struct IrKeyHash {
  size_t operator()(const IrKey &k) const {
    const unsigned char *b = (const unsigned char *)&k.a;
    uint64_t h = 1469598103934665603ull;
    for (size_t i = 0; i < sizeof(k.a); ++i) h = (h ^ b[i]) * 1099511628211ull;
    return (size_t)h;
  }
};
struct IrPlan {
  IrParams p;
  IrChoice c;
  int grid;
  bool ok;
};

template <int EC, int ST, bool F16, bool CL>
void ir_launch_one(const IrPlan &pl, cudaStream_t s) {
  auto kernel = ir_kernel<EC, ST, F16, CL>;
  static unsigned char attr_done[TC_MAX_DEVICES] = {};
  if (tc_first_use_on_device(attr_done)) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT);
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  }
  tc_launch_pdl(kernel, pl.grid, IR_THREADS, pl.c.smem, s, pl.p, pl.p.splits);
  went_forwards();
}
template <int EC, int ST>
void ir_launch_es(const IrPlan &pl, bool f16, cudaStream_t s) {
  const bool cl = pl.p.splits > 1;
  if (f16 && cl) ir_launch_one<EC, ST, true, true>(pl, s);
  else if (f16) ir_launch_one<EC, ST, true, false>(pl, s);
  else if (cl) ir_launch_one<EC, ST, false, true>(pl, s);
  else ir_launch_one<EC, ST, false, false>(pl, s);
}

uint32_t pair_bits(float v, bool f16) {
  uint16_t b;
  if (f16) {
    const __half h = __float2half_rn(v);
    memcpy(&b, &h, 2);
  } else {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    memcpy(&b, &h, 2);
  }
  return b | ((uint32_t)b << 16);
}

IrPlan ir_build(const IrArgs &a) {
  Runtime &r = rt();
  IrPlan pl;
  memset(&pl, 0, sizeof(pl));
  pl.c = ir_choose(a.form_n, a.C, a.E, a.K, a.P, a.Q, a.stride, a.f16 != 0, r.num_sms);
  if (pl.c.us < 0) return pl;
  const IrChoice &c = pl.c;
  IrParams &p = pl.p;
  const int Cp = (a.C + 15) / 16 * 16;
  p.bk = Cp <= 16 ? 16 : Cp <= 32 ? 32 : 64;
  p.kcs = (Cp + p.bk - 1) / p.bk;
  p.w2 = a.w2; p.b2 = a.b2; p.b3 = a.b3;
  p.residual = a.residual;
  p.y = a.y;
  p.H = a.H; p.W = a.W; p.P = a.P; p.Q = a.Q; p.C = a.C; p.E = a.E; p.K = a.K;
  p.Kp = (a.K + 15) / 16 * 16;
  p.chunks = (a.E + c.ec - 1) / c.ec;
  p.splits = c.splits;
  p.tw = c.tw; p.th = c.th;
  p.iw = (c.tw - 1) * a.stride + 3;
  p.ih = (c.th - 1) * a.stride + 3;
  p.segs = c.segs; p.seg_rows = c.seg_rows;
  p.tiles_w = (a.Q + c.tw - 1) / c.tw;
  p.tiles_h = (a.P + c.th - 1) / c.th;
  p.rows_owner = (c.tw * c.th + c.splits - 1) / c.splits;
  p.div_iw = make_fastdiv(p.iw);
  p.div_tw = make_fastdiv(p.tw);
  p.div_w = make_fastdiv(p.tiles_w);
  p.div_h = make_fastdiv(p.tiles_h);
  p.div_g8 = make_fastdiv(a.K / 8);
  p.tiles = p.tiles_w * p.tiles_h * a.N;
  pl.c.smem = ir_smem(c.ec, p.kcs, p.bk, p.iw * p.ih, c.tw * c.th, p.Kp, c.splits, a.f16 != 0, &p.x_bytes, &p.ex_bytes);
  p.clip1 = a.lo[0] == a.lo[0];
  p.lo1 = pair_bits(p.clip1 ? a.lo[0] : a.floor[0], a.f16);
  p.hi1 = pair_bits(p.clip1 ? a.hi[0] : INFINITY, a.f16);
  p.lo2 = pair_bits(a.lo[1] == a.lo[1] ? a.lo[1] : a.floor[1], a.f16);
  p.hi2 = pair_bits(a.hi[1] == a.hi[1] ? a.hi[1] : INFINITY, a.f16);
  p.zero_inside = !(a.lo[0] > 0.0f || a.hi[0] < 0.0f);
  p.floor3 = a.floor[2]; p.lo3 = a.lo[2]; p.hi3 = a.hi[2];
  p.consts_ready = a.consts_ready;
  p.err = r.dev_err;
  bool ok = true;
  {
    const uint64_t dims[4] = {(uint64_t)a.C, (uint64_t)a.W, (uint64_t)a.H, (uint64_t)a.N};
    const uint64_t st[3] = {(uint64_t)a.C * 2, (uint64_t)a.W * a.C * 2, (uint64_t)a.H * a.W * a.C * 2};
    const uint32_t box[4] = {(uint32_t)p.bk, (uint32_t)p.iw, (uint32_t)p.ih, 1};
    ok &= make_map(&p.tmX, a.x, 4, dims, st, box, p.bk * 2, true);
  }
  {
    const uint64_t dims[3] = {(uint64_t)Cp, (uint64_t)a.E, 1};
    const uint64_t st[2] = {(uint64_t)Cp * 2, (uint64_t)a.E * Cp * 2};
    const uint32_t box[3] = {(uint32_t)p.bk, (uint32_t)c.ec, 1};
    ok &= make_map(&p.tmW1, a.w1, 3, dims, st, box, p.bk * 2, true);
  }
  {
    const uint64_t dims[3] = {16, (uint64_t)a.E, 1};
    const uint64_t st[2] = {32, (uint64_t)a.E * 32};
    const uint32_t box[3] = {16, (uint32_t)c.ec, 1};
    ok &= make_map(&p.tmB1, a.b1, 3, dims, st, box, 32, true);
  }
  {
    const uint64_t dims[3] = {(uint64_t)a.E, (uint64_t)a.K, 1};
    const uint64_t st[2] = {(uint64_t)a.E * 2, (uint64_t)a.K * a.E * 2};
    const uint32_t box[3] = {(uint32_t)c.ec, (uint32_t)p.Kp, 1};
    ok &= make_map(&p.tmW2, a.w3, 3, dims, st, box, c.ec * 2, true);
  }
  const int res = pl.c.smem <= TC_SMEM_DUO && (p.iw * p.ih + 127) / 128 * c.ec + p.Kp <= 256 ? 2 : 1;
  pl.grid = c.splits > 1 || p.tiles < r.num_sms * res ? p.tiles * c.splits : r.num_sms * res;
  pl.ok = ok;
#ifdef OCCAMY_TUNING
  if (getenv("OCCAMY_TC_PLAN_LOG"))
    fprintf(stderr, "[irplan] N %d C %d E %d K %d in %dx%d s%d: ec %d tile %dx%d (in %d) segs %d splits %d grid %d smem %zu us %.1f\n",
            a.N, a.C, a.E, a.K, a.W, a.H, a.stride, c.ec, c.tw, c.th, p.iw * p.ih, c.segs, c.splits, pl.grid, pl.c.smem, c.us);
#endif
  return pl;
}

}  // namespace

bool ir_supported(int N, int C, int E, int K, int H, int W, int P, int Q, int stride, bool f16) {
#ifdef OCCAMY_TUNING
  if (const char *f = getenv("OCCAMY_IR")) if (!strcmp(f, "0")) return false;
#endif
  if (N < 1 || C < 16 || C % 8 || E % 16 || E > IR_MAX_E || K % 8 || K > 160 || H < 2 || W < 2) return false;
  if (stride != 1 && stride != 2) return false;
  if (P != (H - 1) / stride + 1 || Q != (W - 1) / stride + 1) return false;
  if ((int64_t)N * P * Q >= (1ll << 31)) return false;
  const IrChoice c = ir_choose(N, C, E, K, P, Q, stride, f16, rt().num_sms);
  // Worth it where the separate kernels (3.3 us each, 4.6 TB/s of their tensors) take longer.  MobileNetV2's
  // blocks, fp16: at batch 1 all of them (10.5 -> 5.5 us each), at batch 128 those at 112x112 and 56x56 (197 ->
  // 117, 150 -> 121, 125 -> 61 us) and some later ones.
  // The last factor is for the model's error: a block is fused where the gain is plain.  The model was fitted to a kernel
  // that loaded and issued by one lane, and has not been since; as a whole warp it takes 0.77 to 0.95 of the time, where no
  // cluster shares the chunks: fused and
  // apart now 112 and 118 us (24 -> 144 -> 24 at 56x56, batch 128; 61 and 70 at 64), 37 and 46 (32 -> 192 -> 32 at 28x28),
  // 24 and 29 (96 -> 576 -> 160, stride 2), 24 and 31 (96 -> 576 -> 96 at 14x14, batch 64), 47 and 47 (there at 128, 1.18
  // by the model).  In clusters 35 against 25 (96 -> 576 -> 160 at 64, 1.06 by the model).  With fp32 sums in the depthwise
  // stage it is slower again, and the lower factor stays: MobileNetV2 in bf16 with factors of 0.9, 1.0, 1.1 and 1.2 takes
  // 203, 203, 203 and 203 us (4 images), 314, 314, 315, 315 (16), 574, 577, 590, 604 (64), 966, 964, 956, 976 (128).
  double bytes = 2.0 * N * ((double)H * W * (C + 2.0 * E) + (double)P * Q * (2.0 * E + K + (C == K ? K : 0)));
  if (C % 16) bytes += 5.0 * N * H * W * (C + 16);   // the separate kernels' input is padded in a pass of its own
  const double margin = f16 && c.splits == 1 ? 1.1 : 0.9;
  return c.us >= 0 && c.us < margin * (9.9 + bytes / 4.6e6);
}

bool launch_ir(const IrArgs &a, cudaStream_t s) {
  static std::unordered_map<IrKey, IrPlan, IrKeyHash> plans;
  IrKey key;
  memcpy(&key.a, &a, sizeof(a));
  auto it = plans.find(key);
  if (it == plans.end()) {
    if (plans.size() > 1024) plans.clear();
    it = plans.emplace(key, ir_build(a)).first;
  }
  const IrPlan &pl = it->second;
  if (!pl.ok) return false;
  if (pl.c.ec == 64 && a.stride == 1) ir_launch_es<64, 1>(pl, a.f16 != 0, s);
  else if (pl.c.ec == 64) ir_launch_es<64, 2>(pl, a.f16 != 0, s);
  else if (a.stride == 1) ir_launch_es<32, 1>(pl, a.f16 != 0, s);
  else ir_launch_es<32, 2>(pl, a.f16 != 0, s);
  OCC_CUDA(cudaGetLastError());
  count(CNT_LAUNCHES);
  count(CNT_TC_LAUNCHES);
  count(CNT_INVERTED_RESIDUAL);
  return true;
}

}  // namespace occ
