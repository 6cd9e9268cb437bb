// Two layers in one kernel: the convolution that ends a block, y = relu(sum), and the 1x1 convolution that begins the
// next, t = relu(y * W + b).  (Both outputs are written: y is the next block's shortcut.)
//
// What bounds these layers where images are large is HBM: y is the widest tensor of a network (411 MB for 256 images of
// 256 channels at 56x56), and the second layer reads all of it.  Here the staged slab of y that TMA stores is an operand
// of the second product as it lies in shared memory: 64 channels of 128 pixels, K-major in the 128-byte swizzle.
// 256 images (ncu), the two layers apart and together: 64 -> 256 with shortcut -> 64 at 56x56 217 -> 157 us (1.03 GB, the
// copy rate), with a projection of 64 channels in its place 178 -> 121 (0.72 GB); 128 -> 512 with shortcut -> 128 at
// 28x28 120 -> 88.  ResNet-50 at 256 images 3001 -> 2746 us.  One issuer for both products: 159, 165 and 97.  Not taken,
// for being slower: 256 -> 1024 -> 256 at 14x14 (75 against 67 apart: a megabyte of weights per tile), and 128 + 256 ->
// 512 -> 128 at 28x28 (163 against 133: six blocks of x leave no room for the next tile's).
//
// A CTA works through tiles of 128 pixels, y in chunks of 128 channels:
//   product 1   D1[c & 1] = x * W1[chunk] (+ x2 * W1b[chunk]), the tile's x resident for all chunks
//   epilogue 1  + bias (+ shortcut tensor, fetched into the slab ahead of time), ReLU, 16 bits -> two slabs
//   product 2   D2 += slab * W2[all of t's channels][64 of y's], as soon as a slab is written
//   epilogue 2  behind the next tile's first chunk, so that nobody waits for the last products
// The tensor core works on one chunk's product 1 and another one's product 2 while the epilogue works on a third.
//
//   (all but the epilogue: whole warps that elect a lane for each instruction)
//   warp 0      x
//   warps 1, 14 MMA issuers of product 1 and product 2: an issuer's polls of barriers, some 200 cycles
//               each, are its time, and the two products share none
//   warps 2-9   epilogue, two per TMEM lane quadrant
//   warps 10, 15 weights of product 1 and product 2, a ring of tiles each
//   warps 11-12 slabs of y (alternate slabs): handed out empty or with the shortcut's values, stored;
//               a slab is free again when the store has read it and product 2 is done
//   warp 13     slabs of t
// Every wait is bounded; one that runs out records a code and the kernel drains.
#include "conv_pair.h"

namespace occ {

namespace {

constexpr int PR_THREADS = 512;
constexpr uint32_t PR_BLOCK = 128u * 128u;   // 128 rows of 64 channels: an x block, a slab of y, a weight tile
constexpr uint32_t PR_T = 128u * 64u;        // a slab of t: 32 channels
constexpr int PR_MAX_A = 6, PR_MAX_W = 4, PR_MAX_S = 8;

template <bool F16, bool RES>
__global__ void __launch_bounds__(PR_THREADS, 1) tc_pair_kernel(const __grid_constant__ PairParams p) {
  constexpr uint32_t FORMAT = (1u << 4) | (F16 ? 0u : ((1u << 7) | (1u << 10))) | ((uint32_t)(128 >> 4) << 24);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) atomicExch(p.err, 1007);
    return;
  }
  const int nA = p.a_blocks, nW = p.w1_tiles, nV = p.w2_tiles, nS = p.slabs;
  const uint32_t sA = smem_u32(smem_raw), sW = sA + nA * PR_BLOCK, sV = sW + nW * PR_BLOCK, sS = sV + nV * PR_BLOCK, sT = sS + nS * PR_BLOCK;
  const uint32_t misc = sT + 2 * PR_T;
  float *bias1 = reinterpret_cast<float *>(smem_raw + (misc - sA));     // K1 floats, then K2
  float *bias2 = bias1 + p.K1;
  const uint32_t bar0 = misc + (uint32_t)(p.K1 + p.K2) * 4u;
  auto a_full = [&](int s) { return bar0 + 8u * s; };
  auto a_empty = [&](int s) { return bar0 + 8u * (PR_MAX_A + s); };
  auto w_full = [&](int s) { return bar0 + 8u * (2 * PR_MAX_A + s); };
  auto w_empty = [&](int s) { return bar0 + 8u * (2 * PR_MAX_A + PR_MAX_W + s); };
  auto v_full = [&](int s) { return bar0 + 8u * (2 * (PR_MAX_A + PR_MAX_W) + s); };
  auto v_empty = [&](int s) { return bar0 + 8u * (2 * (PR_MAX_A + PR_MAX_W) + PR_MAX_W + s); };
  constexpr int B1 = 2 * (PR_MAX_A + 2 * PR_MAX_W);
  auto s_ready = [&](int s) { return bar0 + 8u * (B1 + s); };               // free, or holds the shortcut's values
  auto s_full = [&](int s) { return bar0 + 8u * (B1 + PR_MAX_S + s); };     // written by the epilogue
  auto s_read = [&](int s) { return bar0 + 8u * (B1 + 2 * PR_MAX_S + s); }; // product 2 is done with it
  constexpr int B2 = B1 + 3 * PR_MAX_S;
  auto d1_full = [&](int s) { return bar0 + 8u * (B2 + s); };
  auto d1_empty = [&](int s) { return bar0 + 8u * (B2 + 2 + s); };
  auto t_full = [&](int s) { return bar0 + 8u * (B2 + 4 + s); };
  auto t_empty = [&](int s) { return bar0 + 8u * (B2 + 6 + s); };
  const uint32_t d2_full = bar0 + 8u * (B2 + 8), d2_empty = bar0 + 8u * (B2 + 9);
  constexpr int NBARS = B2 + 10;
  static_assert(NBARS * 8 + 16 <= PR_MISC_BYTES, "barriers, the TMEM address and the flag");
  uint8_t *tail = smem_raw + (bar0 - sA) + 8 * NBARS;
  volatile uint32_t *tmem_holder = reinterpret_cast<volatile uint32_t *>(tail);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tail + 8);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    tma_prefetch_map(&p.tmA[0]);
    tma_prefetch_map(&p.tmB1[0]);
    tma_prefetch_map(&p.tmB2);
    tma_prefetch_map(&p.tmY);
    for (int s = 0; s < nA; ++s) {
      mbar_init(a_full(s), 1);
      mbar_init(a_empty(s), 1);
    }
    for (int s = 0; s < nW; ++s) {
      mbar_init(w_full(s), 1);
      mbar_init(w_empty(s), 1);
    }
    for (int s = 0; s < nV; ++s) {
      mbar_init(v_full(s), 1);
      mbar_init(v_empty(s), 1);
    }
    for (int s = 0; s < nS; ++s) {
      mbar_init(s_ready(s), 1);
      mbar_init(s_full(s), 8);
      mbar_init(s_read(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(d1_full(s), 1);
      mbar_init(d1_empty(s), 8);
      mbar_init(t_full(s), 8);
      mbar_init(t_empty(s), 1);
    }
    mbar_init(d2_full, 1);
    mbar_init(d2_empty, 8);
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
  const uint32_t tmem = *tmem_holder, tmem2 = tmem + 256u;
  const int chunks = p.K1 / 128, k1 = p.blocks1 + p.blocks2;
  int err_code = 0;
  pdl_launch_dependents();
  // (resident weights may be fetched while the kernel before this one is still running)
  if (!((warp == 10 || warp == 15) && p.consts_ready)) pdl_wait();

  auto pixels = [&](int tile) {
    if (p.descending) tile = p.total_tiles - 1 - tile;
    const uint32_t s2 = tc_fdiv((uint32_t)tile, p.div_w), nn = tc_fdiv(s2, p.div_h);
    TcTile t;
    t.k0 = 0;
    t.q0 = (tile - (int)s2 * p.tiles_w) * p.tw;
    t.p0 = (int)(s2 - nn * (uint32_t)p.tiles_h) * p.th;
    t.n0 = (int)nn * p.tn;
    return t;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ x
    {
      int s = 0;
      uint32_t phase = 0;
      const uint32_t bytes = (uint32_t)p.rows * 128u;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        const TcTile tl = pixels(tile);
        for (int k = 0; k < k1; ++k) {
          if (!mbar_wait_warp(a_empty(s), phase ^ 1u, abort_flag)) {
            err_code = 1;
            break;
          }
          const bool second = k >= p.blocks1;
          expect_tx_warp(a_full(s), bytes);
          load_4d_warp(sA + s * PR_BLOCK, &p.tmA[second], a_full(s), (second ? k - p.blocks1 : k) * 64, tl.q0, tl.p0, tl.n0);
          if (++s == nA) {
            s = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 10) {
    // ------------------------------------------------------------ weights of product 1
    {
      int s = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x)
        for (int c = 0; c < chunks && !err_code; ++c)
          for (int k = 0; k < k1; ++k) {
            if (!mbar_wait_warp(w_empty(s), phase ^ 1u, abort_flag)) {
              err_code = 1;
              break;
            }
            const bool second = k >= p.blocks1;
            expect_tx_warp(w_full(s), PR_BLOCK);
            load_3d_warp(sW + s * PR_BLOCK, &p.tmB1[second], w_full(s), (second ? k - p.blocks1 : k) * 64, c * 128, 0);
            if (++s == nW) {
              s = 0;
              phase ^= 1u;
            }
          }
    }
  } else if (warp == 15) {
    // ------------------------------------------------------------ weights of product 2
    {
      int s = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x)
        for (int c = 0; c < p.K1; c += 64) {
          if (!mbar_wait_warp(v_empty(s), phase ^ 1u, abort_flag)) {
            err_code = 1;
            break;
          }
          expect_tx_warp(v_full(s), (uint32_t)p.K2 * 128u);
          load_3d_warp(sV + s * PR_BLOCK, &p.tmB2, v_full(s), c, 0, 0);
          if (++s == nV) {
            s = 0;
            phase ^= 1u;
          }
        }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ product 1
    {
      const uint32_t idesc = FORMAT | ((uint32_t)(128 >> 3) << 17);
      const uint64_t d0 = make_smem_desc(sA, 64);
      const uint32_t hi = (uint32_t)(d0 >> 32), a_lo0 = (uint32_t)d0, w_lo0 = (uint32_t)make_smem_desc(sW, 64);
      constexpr uint32_t STEP = PR_BLOCK >> 4;
      int ws = 0, a_base = 0, a_next = 0, d1 = 0;
      uint32_t w_phase = 0, a_phase = 0, d1_phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        a_base = a_next;
        for (int c = 0; c < chunks && !err_code; ++c) {
          if (!mbar_wait_warp(d1_empty(d1), d1_phase ^ 1u, abort_flag)) {
            err_code = 2;
            break;
          }
          int as = a_base;
#pragma unroll 1
          for (int k = 0; k < k1; ++k) {
            if ((c == 0 && !mbar_wait_warp(a_full(as), a_phase, abort_flag)) ||
                !mbar_wait_warp(w_full(ws), w_phase, abort_flag)) {
              err_code = 3;
              break;
            }
            tc_fence_after();
            const uint32_t a_lo = a_lo0 + (uint32_t)as * STEP, b_lo = w_lo0 + (uint32_t)ws * STEP;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_warp(tmem + (uint32_t)(d1 * 128), a_lo + 2u * kk, hi, b_lo + 2u * kk, hi, idesc, kk ? 1u : (uint32_t)(k != 0));
            commit_warp(w_empty(ws));
            if (c == chunks - 1) commit_warp(a_empty(as));
            if (++ws == nW) {
              ws = 0;
              w_phase ^= 1u;
            }
            if (++as == nA) {
              as = 0;
              if (c == 0) a_phase ^= 1u;
            }
          }
          if (err_code) break;
          a_next = as;
          commit_warp(d1_full(d1));
          d1 ^= 1;
          if (d1 == 0) d1_phase ^= 1u;
        }
      }
    }
  } else if (warp == 14) {
    // ------------------------------------------------------------ product 2
    {
      const uint32_t idesc = FORMAT | ((uint32_t)(p.K2 >> 3) << 17);
      const uint64_t d0 = make_smem_desc(sS, 64);
      const uint32_t hi = (uint32_t)(d0 >> 32), s_lo0 = (uint32_t)d0, v_lo0 = (uint32_t)make_smem_desc(sV, 64);
      constexpr uint32_t STEP = PR_BLOCK >> 4;
      int vs = 0, ss = 0;
      uint32_t v_phase = 0, s_phase = 0, d2_phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        if (!mbar_wait_warp(d2_empty, d2_phase ^ 1u, abort_flag)) {
          err_code = 2;
          break;
        }
        d2_phase ^= 1u;
#pragma unroll 1
        for (int c = 0; c < p.K1; c += 64) {
          if (!mbar_wait_warp(v_full(vs), v_phase, abort_flag) || !mbar_wait_warp(s_full(ss), s_phase, abort_flag)) {
            err_code = 3;
            break;
          }
          tc_fence_after();
          const uint32_t a_lo = s_lo0 + (uint32_t)ss * STEP, b_lo = v_lo0 + (uint32_t)vs * STEP;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk)
            mma_warp(tmem2, a_lo + 2u * kk, hi, b_lo + 2u * kk, hi, idesc, kk ? 1u : (uint32_t)(c != 0));
          commit_warp(v_empty(vs));
          commit_warp(s_read(ss));
          if (++vs == nV) {
            vs = 0;
            v_phase ^= 1u;
          }
          if (++ss == nS) {
            ss = 0;
            s_phase ^= 1u;
          }
        }
        if (!err_code) commit_warp(d2_full);
      }
    }
  } else if (warp == 11 || warp == 12) {
    // ------------------------------------------------------------ slabs of y
    {
      const int me = warp - 11, per_tile = 2 * chunks;
      // hand-outs: slab number `r` of this CTA is slab r_sl of tile r_tile, in buffer r_buf
      int r_tile = blockIdx.x, r_sl = me, r_buf = me;
      auto hand_out = [&]() {
        if (r_tile >= p.total_tiles) return;
        if constexpr (RES) {
          const TcTile tl = pixels(r_tile);
          expect_tx_warp(s_ready(r_buf), (uint32_t)p.rows * 128u);
          load_4d_warp(sS + r_buf * PR_BLOCK, &p.tmR, s_ready(r_buf), r_sl * 64, tl.q0, tl.p0, tl.n0);
        } else {
          arrive_warp(s_ready(r_buf));
        }
        r_buf += 2;
        if (r_buf >= nS) r_buf -= nS;
        r_sl += 2;
        if (r_sl >= per_tile) {
          r_sl -= per_tile;
          r_tile += gridDim.x;
        }
      };
      for (int i = 0; i < nS / 2; ++i) hand_out();
      int buf = me, last = -1;
      uint32_t phase = 0, last_phase = 0;
      // the slab stored before the newest is free when product 2 has been made with it
      auto give_back = [&]() {
        if (last < 0) return true;
        if (!mbar_wait_warp(s_read(last), last_phase, abort_flag)) {
          err_code = 6;
          return false;
        }
        hand_out();
        return true;
      };
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        const TcTile tl = pixels(tile);
        for (int sl = me; sl < per_tile; sl += 2) {
          if (!mbar_wait_warp(s_full(buf), phase, abort_flag)) {
            err_code = 6;
            break;
          }
          store_4d_warp(&p.tmY, sS + buf * PR_BLOCK, sl * 64, tl.q0, tl.p0, tl.n0);
          tma_store_commit();
          tma_store_wait_read<1>();
          if (!give_back()) break;
          last = buf;
          last_phase = phase;
          buf += 2;
          if (buf >= nS) {
            buf -= nS;
            phase ^= 1u;
          }
        }
      }
      tma_store_wait_read<0>();
    }
  } else if (warp == 13) {
    // ------------------------------------------------------------ slabs of t
    {
      int b = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x) {
        const TcTile tl = pixels(tile);
        for (int c = 0; c < p.K2; c += 32) {
          if (!mbar_wait_warp(t_full(b), phase, abort_flag)) {
            err_code = 8;
            break;
          }
          store_4d_warp(&p.tmT, sT + b * PR_T, c, tl.q0, tl.p0, tl.n0);
          tma_store_commit();
          tma_store_wait_read<0>();
          arrive_warp(t_empty(b));
          b ^= 1;
          if (b == 0) phase ^= 1u;
        }
      }
      tma_store_wait_read<0>();
    }
  } else if (warp < 10) {
    // ------------------------------------------------------------ epilogues
    const int quad = warp & 3, part = (warp - 2) >> 2, row = quad * 32 + lane;
    const int et = threadIdx.x - 64;
    for (int i = et; i < p.K1; i += 256) bias1[i] = (p.bias1 ? p.bias1[i] : 0.0f) + (p.bias1b ? p.bias1b[i] : 0.0f);
    for (int i = et; i < p.K2; i += 256) bias2[i] = p.bias2 ? p.bias2[i] : 0.0f;
    epi_bar();
    uint32_t soff[4], toff[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) soff[i] = slab_off(row, part * 4 + i, 128);
#pragma unroll
    for (int i = 0; i < 2; ++i) toff[i] = slab_off(row, part * 2 + i, 64);
    const uint32_t t_lane = (uint32_t)(quad * 32) << 16;
    int d1 = 0, ss = 0, tb = 0;
    uint32_t d1_phase = 0, d2_phase = 0, s_phase = 0, t_phase = 0;
    // epilogue 2 of the tile whose products 2 are done next
    auto finish_t = [&]() {
      if (!mbar_wait(d2_full, d2_phase, abort_flag)) {
        err_code = 4;
        return;
      }
      d2_phase ^= 1u;
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < p.K2; c += 32) {
        uint32_t r[16], pk[8];
        tc_ld16(tmem2 + t_lane + (uint32_t)(c + part * 16), r);
        tc_ld_wait();
        if (c + 32 >= p.K2) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(d2_empty);
        }
        const float4 *b4 = reinterpret_cast<const float4 *>(bias2 + c + part * 16);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 b = b4[j];
          pk[2 * j] = f2_to_bf16x2_relu<F16>(
              f2_add(f2_pack(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1])), f2_pack(b.x, b.y)));
          pk[2 * j + 1] = f2_to_bf16x2_relu<F16>(
              f2_add(f2_pack(__uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])), f2_pack(b.z, b.w)));
        }
        if (!mbar_wait(t_empty(tb), t_phase ^ 1u, abort_flag)) {
          err_code = 5;
          return;
        }
        uint8_t *dst = smem_raw + (sT - sA) + tb * PR_T;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<uint4 *>(dst + toff[i]) = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(t_full(tb));
        tb ^= 1;
        if (tb == 0) t_phase ^= 1u;
      }
    };
    auto slab = [&](const uint32_t *r, int c0) -> bool {   // 64 channels of y from c0 on, this thread's 32 of them in r
      if (!mbar_wait(s_ready(ss), s_phase, abort_flag)) return false;
      uint8_t *dst = smem_raw + (sS - sA) + ss * PR_BLOCK;
      const float4 *b4 = reinterpret_cast<const float4 *>(bias1 + c0 + part * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 b0 = b4[2 * i], b1 = b4[2 * i + 1];
        uint64_t v[4] = {f2_pack(b0.x, b0.y), f2_pack(b0.z, b0.w), f2_pack(b1.x, b1.y), f2_pack(b1.z, b1.w)};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          v[e] = f2_add(f2_pack(__uint_as_float(r[8 * i + 2 * e]), __uint_as_float(r[8 * i + 2 * e + 1])), v[e]);
        if constexpr (RES) {
          const uint4 rv = *reinterpret_cast<const uint4 *>(dst + soff[i]);
          const uint32_t w[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) v[e] = f2_add(v[e], pair16_to_f2<F16>(w[e]));
        }
        *reinterpret_cast<uint4 *>(dst + soff[i]) = make_uint4(f2_to_bf16x2_relu<F16>(v[0]), f2_to_bf16x2_relu<F16>(v[1]),
                                                               f2_to_bf16x2_relu<F16>(v[2]), f2_to_bf16x2_relu<F16>(v[3]));
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_full(ss));
      if (++ss == nS) {
        ss = 0;
        s_phase ^= 1u;
      }
      return true;
    };
    bool first = true;
    for (int tile = blockIdx.x; tile < p.total_tiles && !err_code; tile += gridDim.x, first = false) {
#pragma unroll 1
      for (int c = 0; c < chunks && !err_code; ++c) {
        if (!mbar_wait(d1_full(d1), d1_phase, abort_flag)) {
          err_code = 4;
          break;
        }
        tc_fence_after();
        uint32_t ra[32], rb[32];
        const uint32_t t_row = tmem + t_lane + (uint32_t)(d1 * 128 + part * 32);
        tc_ld32(t_row, ra);
        tc_ld_wait();
        tc_ld32(t_row + 64u, rb);
        bool ok = slab(ra, c * 128);
        tc_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d1_empty(d1));
        ok = ok && slab(rb, c * 128 + 64);
        if (!ok) {
          err_code = 5;
          break;
        }
        d1 ^= 1;
        if (d1 == 0) d1_phase ^= 1u;
        if (c == 0 && !first) finish_t();   // of the tile before this one
      }
    }
    if (!first && !err_code) finish_t();
  }

  if (err_code) {
    atomicExch(p.err, 1000 + err_code);
    *abort_flag = 1;
    for (int i = 0; i < 50; ++i) __nanosleep(20000);   // copies in flight land before memory goes
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

template <bool F16, bool RES>
void pair_launch_one(const PairParams &p, int grid, size_t smem, cudaStream_t s) {
  static unsigned char attr_done[TC_MAX_DEVICES] = {};
  if (tc_first_use_on_device(attr_done))
    cudaFuncSetAttribute(tc_pair_kernel<F16, RES>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT);
  tc_launch_pdl(tc_pair_kernel<F16, RES>, grid, PR_THREADS, smem, s, p);
}

}  // namespace

// Shares out shared memory; false when a tile does not fit.
bool pair_layout(PairParams &p, size_t *smem) {
  const int k1 = p.blocks1 + p.blocks2;
  const size_t fixed = 2 * PR_T + (size_t)(p.K1 + p.K2) * 4 + PR_MISC_BYTES;
  int left = (int)(((size_t)TC_SMEM_LIMIT - fixed) / PR_BLOCK);   // blocks of 16 KB
  left -= k1 + 4 + 4;   // a tile's x, the slabs of two chunks, two weight tiles of either product
  if (left < 0 || k1 > 4) return false;
  p.a_blocks = k1; p.slabs = 4; p.w1_tiles = p.w2_tiles = 2;
  // What is left: with a shortcut tensor, slabs for its values on their way and then the next tile's first x; without,
  // the next tile's x; weights.
  if (p.has_res && left > 1) p.slabs += 2, left -= 2;
  while (left > 0 && p.a_blocks < 2 * k1 && p.a_blocks < PR_MAX_A && !(p.has_res && p.a_blocks > k1)) ++p.a_blocks, --left;
  for (; left > 0 && p.w2_tiles < PR_MAX_W; --left) ++(p.w1_tiles > p.w2_tiles ? p.w2_tiles : p.w1_tiles);
  *smem = fixed + (size_t)(p.a_blocks + p.slabs + p.w1_tiles + p.w2_tiles) * PR_BLOCK;
  return true;
}

void pair_launch(const PairParams &p, bool f16, int grid, size_t smem, cudaStream_t s) {
  if (f16) {
    if (p.has_res) pair_launch_one<true, true>(p, grid, smem, s);
    else pair_launch_one<true, false>(p, grid, smem, s);
  } else {
    if (p.has_res) pair_launch_one<false, true>(p, grid, smem, s);
    else pair_launch_one<false, false>(p, grid, smem, s);
  }
}

}  // namespace occ
