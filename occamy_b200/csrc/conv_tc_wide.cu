// 3x3 / stride 1 / pad 1 convolutions with at most 128 output channels: weights on the M side of the MMA, pixels on
// the N side, and every pixel in shared memory once.
//
// What bounds such a layer is shared memory, which delivers 128 bytes a cycle to the tensor core and takes in the
// next operands meanwhile.  With pixels on the M side an MMA of 128 channels reads 8 KB in its 64 cycles, all there
// is; with weights there and 256 pixels on the N side (tc_conv_pn_kernel) it reads 12 KB in 128, but each k-step's
// 48 KB come in anew: 188 bytes a cycle.  Here a tile's input block (its rows plus one above and below, its columns
// plus one on either side, 64 channels) comes in once and the nine taps are windows of it, shifted by whole pixels: a
// swizzled operand may start at any multiple of 128 bytes.  The N index runs through the block's rows, so two of its
// columns are junk (an eighth of 14-column strips), which the epilogue leaves out.
// Before (tc_conv_pn_kernel, pool by itself) and now: 128 -> 128 at 28x28, 256 images, 59.6 -> 46.0 us, 32 images
// 17.7 -> 13.3; 64 -> 128 at 112x112, 64 images, 159 -> 103; 128 -> 128 there with its pool 193 + 36 -> 152.  The last is
// 1560 TFLOP/s of the layer's own operations, 0.94 of the burst rate; what the junk columns take comes on top.
//
// One persistent CTA per SM, roles by warp:
//   (warps 0, 1 and 10: whole warps that elect a lane for each instruction)
//   warp 0      input blocks, two buffers of 64 channels each
//   warp 1      MMA issuer: three taps, 12 MMAs, per barrier -- a poll and what goes with it cost as much as two MMAs; two accumulators of up to 256 pixels
//   warps 2-9   epilogue: a thread owns a channel; bias and clamp, 16-bit values into the staged slabs (64 channels of
//               all the tile's pixels), two bytes at a time, the 32 lanes of a warp next to one another
//   warp 10     weights: six tiles of one tap and 64 channels, handed back one by one
//   warp 11     slab store (one lane)
// POOL: a 2x2 / stride 2 max pool behind the layer.  A thread has all the pixels of its channel.
// Every wait is bounded; one that runs out records a code and the kernel drains.
#include "conv_tc_dev.cuh"
#include "kernels.h"

namespace occ {

namespace {

constexpr int WD_TAPS = 6;                       // weight tiles in shared memory: two filter rows
constexpr uint32_t WD_W_BYTES = 128u * 64u * 2u;  // of one of them
constexpr int WD_X = 2;                          // input blocks

// one pixel's value of this thread's channel into a slab whose rows are 128 bytes
__device__ __forceinline__ void wd_put(uint32_t slab, int row, uint32_t chunk, uint32_t low, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(slab + (uint32_t)row * 128u + ((chunk ^ ((uint32_t)row & 7u)) << 4) + low),
               "h"((uint16_t)v)
               : "memory");
}

template <bool CLAMP, bool POOL>
__global__ void __launch_bounds__(WD_THREADS, 1) tc_conv_wide_kernel(const __grid_constant__ TcParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) atomicExch(p.err, 1007);
    return;
  }
  const uint32_t base = smem_u32(smem_raw);
  const uint32_t x_bytes = (uint32_t)p.halo_a_bytes;
  const uint32_t sX = base, sW = sX + WD_X * x_bytes, sD = sW + WD_TAPS * WD_W_BYTES;
  const int nslab = (p.K + 63) / 64;
  const uint32_t slab_bytes = (uint32_t)p.wide_slab_bytes;
  const uint32_t bar0 = sD + nslab * slab_bytes;
  auto x_full = [&](int s) { return bar0 + 8u * s; };
  auto x_empty = [&](int s) { return bar0 + 8u * (WD_X + s); };
  auto w_full = [&](int g) { return bar0 + 8u * (2 * WD_X + g); };              // three taps
  auto w_empty = [&](int s) { return bar0 + 8u * (2 * WD_X + 2 + s); };
  auto t_full = [&](int s) { return bar0 + 8u * (2 * WD_X + 2 + WD_TAPS + s); };
  auto t_empty = [&](int s) { return bar0 + 8u * (2 * WD_X + 4 + WD_TAPS + s); };
  auto d_full = [&](int s) { return bar0 + 8u * (2 * WD_X + 6 + WD_TAPS + s); };
  auto d_empty = [&](int s) { return bar0 + 8u * (2 * WD_X + 8 + WD_TAPS + s); };
  constexpr int NBARS = 2 * WD_X + 10 + WD_TAPS;
  static_assert(8 * NBARS + 16 <= WD_MISC_BYTES, "barriers, the TMEM address and the flag");
  uint8_t *misc = smem_raw + (bar0 - base) + 8 * NBARS;
  volatile uint32_t *tmem_holder = reinterpret_cast<volatile uint32_t *>(misc);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(misc + 8);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_map(&p.tmA[0]);
    tma_prefetch_map(&p.tmB);
    tma_prefetch_map(&p.tmD);
    for (int s = 0; s < WD_X; ++s) {
      mbar_init(x_full(s), 1);
      mbar_init(x_empty(s), 1);
    }
    for (int s = 0; s < WD_TAPS; ++s) mbar_init(w_empty(s), 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(w_full(s), 3);
      mbar_init(t_full(s), 1);
      mbar_init(t_empty(s), 8);
      mbar_init(d_full(s), 4);
      mbar_init(d_empty(s), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void *)tmem_holder)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  int err_code = 0;
  pdl_launch_dependents();
  // (resident weights may be fetched while the kernel before this one is still running)
  if (!(warp == 10 && p.consts_ready)) pdl_wait();

  if (warp == 0) {
    // ------------------------------------------------------------ input blocks
    {
      const uint32_t bytes = (uint32_t)((p.th + 2) * p.halo_wp) * 128u;
      int s = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        const TcTile tl = tc_decode<128>(p, tile);
        for (int cb = 0; cb < p.cblocks; ++cb) {
          if (!mbar_wait_warp(x_empty(s), phase ^ 1u, abort_flag)) {
            err_code = 1;
            break;
          }
          expect_tx_warp(x_full(s), bytes);
          // what lies outside the image arrives as zeros: the padding
          load_4d_warp(sX + s * x_bytes, &p.tmA[0], x_full(s), cb * 64, tl.q0 - 1, tl.p0 - 1, tl.n0);
          if (++s == WD_X) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------ weights
    {
      int s = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x)
        for (int cb = 0; cb < p.cblocks && !err_code; ++cb)
          for (int t = 0; t < 9; ++t) {
            if (!mbar_wait_warp(w_empty(s), phase ^ 1u, abort_flag)) {
              err_code = 1;
              break;
            }
            expect_tx_warp(w_full(s / 3), WD_W_BYTES);
            load_3d_warp(sW + s * WD_W_BYTES, &p.tmB, w_full(s / 3), cb * 64, 0, t);
            if (++s == WD_TAPS) {
              s = 0;
              phase ^= 1u;
            }
          }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.n_mma >> 3) << 17) |
                             ((uint32_t)(128 >> 4) << 24);
      const uint64_t w0 = make_smem_desc(sW, 64), x0 = make_smem_desc(sX, 64);
      const uint32_t hi = (uint32_t)(w0 >> 32), w_lo0 = (uint32_t)w0, x_lo0 = (uint32_t)x0;
      const uint32_t wp8 = (uint32_t)p.halo_wp * 8u;   // one block row in descriptor units
      int xs = 0, acc = 0, g = 0;
      uint32_t x_phase = 0, acc_phase = 0, w_phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        if (!mbar_wait_warp(t_empty(acc), acc_phase ^ 1u, abort_flag)) {
          err_code = 2;
          break;
        }
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * 256);
        for (int cb = 0; cb < p.cblocks && !err_code; ++cb) {
          if (!mbar_wait_warp(x_full(xs), x_phase, abort_flag)) {
            err_code = 3;
            break;
          }
          uint32_t x_lo = x_lo0 + (uint32_t)xs * (x_bytes >> 4);
#pragma unroll 1
          for (int r = 0; r < 3; ++r) {
            if (!mbar_wait_warp(w_full(g), w_phase, abort_flag)) {
              err_code = 4;
              break;
            }
            tc_fence_after();
            const uint32_t w_lo = w_lo0 + (uint32_t)(g * 3) * (WD_W_BYTES >> 4);
            const uint32_t more = (uint32_t)((cb | r) != 0);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                mma_warp(d_tmem, w_lo + (uint32_t)c * (WD_W_BYTES >> 4) + 2u * kk, hi, x_lo + 8u * c + 2u * kk, hi, idesc,
                         (c | kk) ? 1u : more);
              commit_warp(w_empty(g * 3 + c));
            }
            x_lo += wp8;
            g ^= 1;
            if (g == 0) w_phase ^= 1u;
          }
          commit_warp(x_empty(xs));
          if (++xs == WD_X) {
            xs = 0;
            x_phase ^= 1u;
          }
        }
        commit_warp(t_full(acc));
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else if (warp == 11) {
    // ------------------------------------------------------------ slab store
    // (as a whole warp, polling, it takes issue slots from the epilogue: 64 -> 128 at 112x112 103 us this way, 122 that way)
    if (lane == 0) {
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x, phase ^= 1u) {
        const TcTile tl = tc_decode<128>(p, tile);
        for (int sl = 0; sl < nslab; ++sl) {
          if (!mbar_wait(d_full(sl), phase, abort_flag)) {
            err_code = 6;
            break;
          }
          tma_store_4d(&p.tmD, sD + sl * slab_bytes, sl * 64, POOL ? tl.q0 >> 1 : tl.q0, POOL ? tl.p0 >> 1 : tl.p0, tl.n0);
          tma_store_commit();
        }
        if (err_code) break;
        if (nslab == 2) {
          tma_store_wait_read<1>();
          mbar_arrive(d_empty(0));
        }
        tma_store_wait_read<0>();
        mbar_arrive(d_empty(nslab - 1));
      }
      tma_store_wait_read<0>();
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int quad = warp & 3;                 // TMEM lane quadrant = 32 output channels
    const int half = (warp - 2) >> 2;          // which of the tile's rows
    const int ch = quad * 32 + lane, sl = quad >> 1;
    const uint32_t chunk = (uint32_t)(ch & 63) >> 3, low = (uint32_t)(ch & 7) * 2u;
    const float bias = (p.bias && ch < p.K) ? p.bias[ch] : 0.0f;
    const float lo = p.lo, hi = p.hi;
    const uint64_t bias2 = f2_pack(bias, bias);
    const uint32_t slab = sD + sl * slab_bytes;
    const bool active = sl < nslab;            // warp-uniform
    constexpr int STEP = POOL ? 2 : 1;         // rows taken together
    const int groups = (p.th + STEP - 1) / STEP, h0 = half ? (groups + 1) / 2 * STEP : 0,
              h1 = half ? p.th : (groups + 1) / 2 * STEP;
    const int tw = p.tw, wp = p.halo_wp, cols = (tw + 15) / 16;
    int acc = 0;
    uint32_t acc_phase = 0, d_phase = 0;
    auto pair16 = [&](uint32_t a, uint32_t b) {   // two pixels
      const uint64_t v = f2_add(f2_pack(__uint_as_float(a), __uint_as_float(b)), bias2);
      if constexpr (CLAMP) {
        float x, y;
        f2_unpack(v, x, y);
        return f2_to_bf16x2(f2_pack(tc_clip(x, lo, hi), tc_clip(y, lo, hi)));
      } else {
        return f2_to_bf16x2_relu(v);
      }
    };
    for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
      if (!mbar_wait(t_full(acc), acc_phase, abort_flag)) {
        err_code = 5;
        break;
      }
      tc_fence_after();
      if (active && !mbar_wait(d_empty(sl), d_phase ^ 1u, abort_flag)) {
        err_code = 7;
        break;
      }
      d_phase ^= 1u;
      const uint32_t t_ch = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * 256);
      if (active && h0 < h1) {
        // sixteen columns of a row (of two rows) at a time, the next ones on their way
        uint32_t ra[STEP][16], rb[STEP][16];
        auto request = [&](int h, int c, uint32_t (*r)[16]) {
#pragma unroll
          for (int k = 0; k < STEP; ++k) tc_ld16(t_ch + (uint32_t)((h + k) * wp + c * 16), r[k]);
        };
        int h = h0, c = 0;
        auto step = [&](uint32_t (*r)[16], uint32_t (*next)[16]) -> bool {
          tc_ld_wait();
          const int row = h, col = c * 16;
          if (++c == cols) {
            c = 0;
            h += STEP;
          }
          const bool more = h < h1;
          if (more) request(h, c, next);
          const int left = tw - col;
          if constexpr (POOL) {
            const int at = (row >> 1) * (tw >> 1) + (col >> 1);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t v = tc_max2<false>(pair16(r[0][2 * j], r[0][2 * j + 1]), pair16(r[1][2 * j], r[1][2 * j + 1]));
              v = tc_max2<false>(v, v >> 16);
              if (2 * j < left) wd_put(slab, at + j, chunk, low, v);
            }
          } else {
            const int at = row * tw + col;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint32_t v = pair16(r[0][2 * j], r[0][2 * j + 1]);
              if (2 * j < left) wd_put(slab, at + 2 * j, chunk, low, v);
              if (2 * j + 1 < left) wd_put(slab, at + 2 * j + 1, chunk, low, v >> 16);
            }
          }
          return more;
        };
        request(h, c, ra);
#pragma unroll 1
        while (step(ra, rb) && step(rb, ra)) {
        }
      }
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(t_empty(acc));
        if (active) mbar_arrive(d_full(sl));
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  if (err_code) {
    atomicExch(p.err, 1000 + err_code);
    *abort_flag = 1;
    for (int i = 0; i < 50; ++i) __nanosleep(20000);   // copies in flight land before memory goes
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

template <bool CLAMP, bool POOL>
void wide_launch_one(const TcParams &p, int grid, size_t smem, cudaStream_t s) {
  static unsigned char attr_done[TC_MAX_DEVICES] = {};
  if (tc_first_use_on_device(attr_done))
    cudaFuncSetAttribute(tc_conv_wide_kernel<CLAMP, POOL>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT);
  tc_launch_pdl(tc_conv_wide_kernel<CLAMP, POOL>, grid, WD_THREADS, smem, s, p);
}

}  // namespace

size_t tc_wide_smem(int x_bytes, int slabs, int slab_bytes) {
  return (size_t)WD_X * x_bytes + WD_TAPS * WD_W_BYTES + (size_t)slabs * slab_bytes + WD_MISC_BYTES;
}

void tc_launch_wide(const TcParams &p, bool clamp, bool pool, int grid, size_t smem, cudaStream_t s) {
  if (pool) {
    if (clamp) wide_launch_one<true, true>(p, grid, smem, s);
    else wide_launch_one<false, true>(p, grid, smem, s);
  } else {
    if (clamp) wide_launch_one<true, false>(p, grid, smem, s);
    else wide_launch_one<false, false>(p, grid, smem, s);
  }
}

}  // namespace occ
