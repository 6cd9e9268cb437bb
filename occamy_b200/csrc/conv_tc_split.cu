// Implicit-GEMM convolution / GEMM for problems with few output tiles: small batches, late layers,
// classifier heads.
//
// The persistent kernel (conv_tc_dev.cuh) gives a tile to one CTA, which walks its whole reduction;
// with 13 tiles of 72 k-steps (a 3x3 layer on 512 channels, batch 8) most SMs are idle and a layer
// takes the 18 us of that serial chain.  Here a cluster of up to eight CTAs shares a tile: each
// multiplies its share of the k-steps into its own TMEM, the partial sums meet over distributed
// shared memory, and every CTA finishes (bias, residual, clamp, store) its share of the tile's rows.
// One tile per cluster, nothing persistent: what counts is the latency from the end of the previous
// layer to the start of the next, so
//   * the first stages' weight tiles are requested before the wait for the previous kernel;
//   * the loading thread never waits for a stage when a CTA's share fits the ring;
//   * the residual and the bias are fetched while the products are being accumulated;
//   * results go from registers to global memory as 16-byte pieces.  (Through shared memory and one
//     TMA store the tile's end took 0.5 to 0.9 us longer: 256->64 at 56x56, batch 1, 3.3 -> 4.2 us.)
// Measured times are at the dispatch rule (conv_tc.cu, sk_choose).
//
// Up to four warps issue the MMAs (whole warps, k-steps in turn, an accumulator of their own each)
// and as many load (k-steps in turn), then all eight warps drain the accumulators (two
// per TMEM lane quadrant, half of the columns each).  Several warps per role, because a
// round of barrier poll, issue and commit takes longer than the four MMAs of a k-step (200 to 260 cycles): a lone
// thread's took 450 to 600, whatever it moved.  A ring that is reused has a multiple of that many stages: a stage then always
// belongs to the same two warps, and no barrier can be two phases behind the one that waits on it.
#include "conv_tc_split.cuh"

#include "kernels.h"
#include "runtime.h"

namespace occ {

namespace {

__device__ __forceinline__ void cluster_arrive_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait_acquire() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Stores that happen when `on` is set: predicated instructions, not branches, so that the code in front of
// them runs (and is fetched) either way -- see the rehearsal below.
// (to another CTA's shared memory, counted there on the barrier `bar` as the bytes arrive)
__device__ __forceinline__ void st_async_v4_if(bool on, uint32_t addr, uint32_t bar, uint32_t a, uint32_t b,
                                               uint32_t c, uint32_t d) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.u32 p, %6, 0;\n"
      "@p st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];\n}" ::"r"(addr),
      "r"(a), "r"(b), "r"(c), "r"(d), "r"(bar), "r"((uint32_t)on)
      : "memory");
}
__device__ __forceinline__ void st_shared_v4_if(bool on, uint32_t addr, uint32_t a, uint32_t b, uint32_t c,
                                                uint32_t d) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n@p st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n}" ::"r"(addr),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"((uint32_t)on)
               : "memory");
}
__device__ __forceinline__ void st_global_v4_if(bool on, void *addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %5, 0;\n@p st.global.v4.b32 [%0], {%1, %2, %3, %4};\n}" ::"l"(addr),
               "r"(a), "r"(b), "r"(c), "r"(d), "r"((uint32_t)on)
               : "memory");
}
__device__ __forceinline__ void st_global_if(bool on, float *addr, float v) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.global.f32 [%0], %1;\n}" ::"l"(addr), "f"(v),
               "r"((uint32_t)on)
               : "memory");
}

// Eight channels, sum + bias in v -> residual, clamp, 16-bit values.
template <bool F16>
__device__ __forceinline__ uint4 sk_pack16(const SkParams &p, float *v, const uint4 &res) {
  if (p.residual) {
    const uint32_t w[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a, b;
      f2_unpack(pair16_to_f2<F16>(w[j]), a, b);
      v[2 * j] += a;
      v[2 * j + 1] += b;
    }
  }
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    o[j] = f2_to_bf16x2<F16>(f2_pack(tc_act(v[2 * j], p.floor, p.lo, p.hi), tc_act(v[2 * j + 1], p.floor, p.lo, p.hi)));
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void sk_finish32(const SkParams &p, bool on, float *v, int64_t lin, int c) {
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = tc_act(v[j], p.floor, p.lo, p.hi);
  int64_t step = 1;
  float *o = p.out_f32 + lin * p.ldo + c;
  if (p.out_hw) {
    const uint32_t img = (uint32_t)lin / (uint32_t)p.out_hw;
    step = p.out_hw;
    o = p.out_f32 + ((int64_t)img * p.K + c) * step + ((uint32_t)lin - img * (uint32_t)p.out_hw);
  }
  if (p.out_vec4 && c + 8 <= p.K) {
    st_global_v4_if(on, o, __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
    st_global_v4_if(on, o + 4, __float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]),
                    __float_as_uint(v[7]));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) st_global_if(on && c + j < p.K, o + j * step, v[j]);
  }
}

// The same for three-part output: the residual's parts add up to its fp32 value exactly, the result is
// cut into parts again.
__device__ __forceinline__ void sk_finish_parts(const SkParams &p, bool on, float *v, const uint4 *r, int64_t lin,
                                                int c) {
  const int64_t at = lin * p.K + c;
  if (p.residual) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float a[3], b[3];
#pragma unroll
      for (int j = 0; j < 3; ++j)
        f2_unpack(pair16_to_f2<false>(e == 0 ? r[j].x : e == 1 ? r[j].y : e == 2 ? r[j].z : r[j].w), a[j], b[j]);
      v[2 * e] += (a[0] + a[1]) + a[2];
      v[2 * e + 1] += (b[0] + b[1]) + b[2];
    }
  }
  uint32_t o[3][4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float a = tc_act(v[2 * e], p.floor, p.lo, p.hi), b = tc_act(v[2 * e + 1], p.floor, p.lo, p.hi);
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      o[j][e] = f2_to_bf16x2<false>(f2_pack(a, b));
      const float ta = __uint_as_float(o[j][e] << 16), tb = __uint_as_float(o[j][e] & 0xffff0000u);
      a = fabsf(ta) < INFINITY ? a - ta : 0.0f;   // exact: what the part left over
      b = fabsf(tb) < INFINITY ? b - tb : 0.0f;
    }
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
    st_global_v4_if(on, reinterpret_cast<uint16_t *>(p.y) + j * p.plane + at, o[j][0], o[j][1], o[j][2], o[j][3]);
}

}  // namespace

//   BN     output channels of a tile (N of the MMA)
//   F16    operands and 16-bit output are fp16, else bf16
//   SPLIT  fp32 operands carried as three bf16 parts hi + mid + lo (24 mantissa bits).  A product is the
//          sum of six part products (the three left out are below 2^-24 of it), each exact in fp32:
//          hi*hi goes to the main accumulator, hi*mid, hi*lo, mid*hi, mid*mid, lo*hi to others (one more
//          at 128 channels, else two, so that an activation part meets its filter parts in one MMA).
//          The tensor core truncates when it adds into an fp32 accumulator, a bias toward zero that
//          grows with the number of additions at full magnitude; kept apart, the small terms cost the
//          main sum none.  A stage holds the three parts of either operand once for all six products.
//   CL     a tile has more than one CTA
//   F32    fp32 output (else 16-bit values; with SPLIT the three parts of fp32 ones)
// One flavour per instantiation: these kernels run for a few microseconds, and every stretch of code
// that is not in the instruction cache yet costs a tenth of that.
template <int BN, bool F16, bool SPLIT, bool CL, bool F32>
__global__ void __launch_bounds__(SK_THREADS, 2)
    tc_split_kernel(const __grid_constant__ SkParams p) {
  constexpr uint32_t IDESC0 = (1u << 4) | (F16 ? 0u : ((1u << 7) | (1u << 10))) | ((uint32_t)(128 >> 4) << 24);
  constexpr uint32_t NSHIFT = 17 - 3;   // of N in the instruction descriptor
  constexpr int NI = sk_issuers(BN, SPLIT);
  constexpr int NACC = SPLIT ? (BN == 128 ? 2 : 3) : NI;           // accumulators
  static_assert(NACC * BN <= 256, "two CTAs share the 512 TMEM columns of an SM");
  constexpr int HALF = BN / 2;          // columns of one epilogue thread
  constexpr int G8 = BN / 8;            // eight-channel groups of a tile row

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  if ((smem_u32(smem_raw) & 1023u) != 0u) {
    if (threadIdx.x == 0) atomicExch(p.err, 1007);
    return;
  }
  const int stages = p.stages, bk = p.bk, splits = CL ? p.splits : 1;
  constexpr int PARTS = sk_parts(SPLIT);
  // Sums that pass through shared memory, so that neighbouring threads finish neighbouring channels: those
  // of a cluster, and results in three planes, whose 16-byte pieces written row by row cost twice the
  // products' time (256->1024 at 14x14, batch 16, with residual: 36.8 us, this way 22.6).
  constexpr bool ITEMS = CL || (SPLIT && !F32);
  const uint32_t a_tile = (uint32_t)p.a_bytes, b_tile = (uint32_t)BN * bk * 2u;
  const uint32_t a_bytes = PARTS * a_tile, b_bytes = PARTS * b_tile;   // of a stage
  const uint32_t sA = smem_u32(smem_raw), sB = sA + stages * a_bytes;
  // partial sums: behind the ring, or (of one CTA) where the ring was
  const uint32_t sX = CL ? sB + stages * b_bytes : sA, x_bytes = ITEMS ? (uint32_t)(splits * p.rows_owner) * BN * 4u : 0u;
  uint8_t *misc = smem_raw + max(sX + x_bytes - sA, stages * (a_bytes + b_bytes));
  float *bias_s = reinterpret_cast<float *>(misc);                       // BN floats
  int *lin_s = reinterpret_cast<int *>(misc + BN * 4);                   // 128 pixel numbers, -1: none
  uint64_t *bars = reinterpret_cast<uint64_t *>(misc + BN * 4 + 512);
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (stages + s); };
  const uint32_t done_bar = bar0 + 16u * stages, sums_bar = done_bar + 8u;
  volatile uint32_t *tmem_holder = reinterpret_cast<volatile uint32_t *>(bars + 2 * stages + 2);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * stages + 3);
  // which accumulators hold anything, one word per issuer
  volatile int *used = reinterpret_cast<volatile int *>(bars + 2 * stages + 4);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  // Fewer accumulators when there are fewer k-steps: CTAs of the next layer that share this SM need
  // TMEM columns as well.  A power of two.
  const int ni = p.issuers;
  const uint32_t cols = SPLIT ? (BN == 128 ? 256u : 4u * BN) : (uint32_t)(ni == 3 ? 4 : ni) * BN;
  const int rank = CL ? (int)cluster_ctarank() : 0;
  const int tile = (int)blockIdx.x / splits;
  // channel tiles fastest, then columns, rows and images of the pixel grid
  TcTile tl;
  {
    const uint32_t sp = tc_fdiv((uint32_t)tile, p.div_k);
    const uint32_t s2 = tc_fdiv(sp, p.div_w), nn = tc_fdiv(s2, p.div_h);
    tl.k0 = (int)((uint32_t)tile - sp * (uint32_t)p.tiles_k) * BN;
    tl.q0 = (int)(sp - s2 * (uint32_t)p.tiles_w) * p.tw;
    tl.p0 = (int)(s2 - nn * (uint32_t)p.tiles_h) * p.th;
    tl.n0 = (int)nn * p.tn;
  }
  const int ks0 = (int)((int64_t)p.ksteps * rank / splits), ks1 = (int)((int64_t)p.ksteps * (rank + 1) / splits);
  const int mine = ks1 - ks0;           // k-steps of this CTA
  int err_code = 0;

  if (threadIdx.x == 0) {
    tma_prefetch_map(&p.tmB);
    tma_prefetch_map(&p.tmA[p.taps[0].map]);
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(done_bar, (uint32_t)ni);
    mbar_init(sums_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if constexpr (CL) {   // partial sums to come: my rows, from every CTA of the cluster
      const int n = min(p.rows_owner, p.rows - rank * p.rows_owner);
      mbar_expect_tx(sums_bar, n > 0 ? (uint32_t)(splits * n * BN * 4) : 0u);
    }
  }
  if (warp == 3) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void *)tmem_holder)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (warp >= 4) {   // pixel number of every row of the tile
    const int row = (int)threadIdx.x - 128;
    const int r2 = row / p.tw, q = tl.q0 + row - r2 * p.tw;
    const int r3 = r2 / p.th, pp = tl.p0 + r2 - r3 * p.th, n = tl.n0 + r3;
    const bool ok = row < p.rows && q < p.gq && pp < p.gp && n < p.gn;
    lin_s[row] = ok ? (n * p.gp + pp) * p.gq + q : -1;
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CL) cluster_arrive_release();   // waited for before the first remote store
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;
  const uint32_t tx_bytes = PARTS * (uint32_t)p.rows * bk * 2u + b_bytes;
  const int ahead = min(stages, mine);        // k-steps that need no stage to become free

  // (tap, channel block) of a k-step of this CTA
  auto load_b = [&](int i, int s) {
    const int k = ks0 + i;
    const bool second = k >= p.ksteps1;
    const int t = second ? 0 : (int)tc_fdiv((uint32_t)k, p.div_cb);
    const CUtensorMap *m = second ? &p.tmB2 : &p.tmB;
    const int c = (second ? k - p.ksteps1 : k - t * p.cblocks) * bk;
#pragma unroll
    for (int j = 0; j < PARTS; ++j)
      load_3d_warp(sB + s * b_bytes + j * b_tile, m, full_bar(s), c, tl.k0, t * PARTS + j);
  };
  auto load_a = [&](int i, int s) {
    const int k = ks0 + i;
    const bool second = k >= p.ksteps1;
    const int t = second ? 0 : (int)tc_fdiv((uint32_t)k, p.div_cb);
    const SkTap tap = p.taps[t];
    const int map = second ? p.map2 : tap.map, c = (second ? k - p.ksteps1 : k - t * p.cblocks) * bk;
    const int q = tl.q0 + (second ? 0 : tap.dw), h = tl.p0 + (second ? 0 : tap.dh);
#pragma unroll
    for (int j = 0; j < PARTS; ++j)
      load_4d_warp(sA + s * a_bytes + j * a_tile, &p.tmA[map + j], full_bar(s), c, q, h, tl.n0);
  };
  // The k-steps of the first ring turn are requested by four warps in turn.
  const int first = warp >= 4 ? warp - 4 : SK_MAX_STAGES;
  if (p.consts_ready)
    for (int i = first; i < ahead; i += 4) {
      expect_tx_warp(full_bar(i), tx_bytes);
      load_b(i, i);
    }
  pdl_launch_dependents();
  pdl_wait();   // from here on memory that other kernels write is read and written

  // residual pieces this thread will add: fetched now, used after the products
  uint4 res[BN / 16];
  const int row0 = rank * p.rows_owner;
  const int nrows = ITEMS ? min(p.rows_owner, p.rows - row0) : 0;   // rows this CTA finishes
  const int items = nrows * G8;
  const int quad = warp & 3, part = warp >> 2, row = quad * 32 + lane;

  for (int i = first; i < ahead; i += 4) {
    if (!p.consts_ready) expect_tx_warp(full_bar(i), tx_bytes);
    load_a(i, i);
    if (!p.consts_ready) load_b(i, i);
  }
  if (warp >= 4) {   // (the other four warps issue MMAs)
    const int i = (int)threadIdx.x - 128;
    if (i < BN)
      bias_s[i] = ((p.bias && tl.k0 + i < p.K) ? p.bias[tl.k0 + i] : 0.0f) +
                  ((p.bias2 && tl.k0 + i < p.K) ? p.bias2[tl.k0 + i] : 0.0f);
  }
  if (!F32 && !SPLIT && p.residual) {
    if constexpr (CL) {
#pragma unroll
      for (int u = 0; u < BN / 16; ++u) {
        const int it = (int)threadIdx.x + u * SK_THREADS;
        const int r = it / G8, c = tl.k0 + (it % G8) * 8;
        const int lin = it < items ? lin_s[row0 + r] : -1;
        if (lin >= 0 && c < p.K)
          res[u] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p.residual) +
                                                    (int64_t)lin * p.K + c);
      }
    } else {
      const int lin = lin_s[row];
#pragma unroll
      for (int u = 0; u < BN / 16; ++u) {
        const int c = tl.k0 + part * HALF + u * 8;
        if (lin >= 0 && c < p.K)
          res[u] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p.residual) +
                                                    (int64_t)lin * p.K + c);
      }
    }
  }

  // what this thread does with the sums, worked out while they are being made
  constexpr int CH = NACC > 1 || HALF < 32 ? 16 : 32;   // columns per step: of all accumulators at once
  const uint32_t t_row = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * HALF);
  const int lin_row = lin_s[row];
  uint32_t dst = 0, dst_bar = 0;   // CL: where my row's partial sums go, and who counts them there
  if constexpr (CL) {
    const int owner = row / p.rows_owner;
    if (row < p.rows) {
      dst = cluster_map(sX, (uint32_t)owner) +
            (uint32_t)(rank * p.rows_owner + row - owner * p.rows_owner) * (BN * 4u);
      dst_bar = cluster_map(sums_bar, (uint32_t)owner);
    }
  }
  auto finish = [&](bool on, float *v, const uint4 &rs, int lin, int c) {
    if constexpr (F32) {
      sk_finish32(p, on, v, lin, c);
    } else if constexpr (!SPLIT) {
      const uint4 o = sk_pack16<F16>(p, v, rs);
      st_global_v4_if(on, reinterpret_cast<uint16_t *>(p.y) + (int64_t)lin * p.K + c, o.x, o.y, o.z, o.w);
    }
  };

  // Warps 4-7 go through the epilogue twice.  The first time is a rehearsal, right after the first
  // loads have been requested: whatever it computes is not stored.  It brings the code into the
  // instruction cache while the operands travel; fetched when the sums are ready it took 1000 to 2000
  // cycles of a layer's 6000 to 10000 (times at the dispatch rule).
#pragma unroll 1
  for (int pass = warp >= 4 ? 0 : 1; pass < 2; ++pass) {
    const bool real = pass != 0;
    int used_all[NI];
    if (real) {
    if (warp >= 4 && warp < 4 + ni) {
      // later turns (stages is a multiple of ni then): k-step i goes to stage i % stages, loader i % ni
      int s = warp - 4;
      uint32_t phase = 0;
      for (int i = stages + s; i < mine; i += ni) {
        if (!mbar_wait_warp(empty_bar(s), phase, abort_flag)) {
          err_code = 1;
          break;
        }
        expect_tx_warp(full_bar(s), tx_bytes);
        load_b(i, s);
        load_a(i, s);
        s += ni;
        if (s >= stages) {
          s -= stages;
          phase ^= 1u;
        }
      }
    } else if (warp < ni) {
      const uint64_t a0 = make_smem_desc(sA, bk), b0 = make_smem_desc(sB, bk);
      const uint32_t a_hi = (uint32_t)(a0 >> 32), b_hi = (uint32_t)(b0 >> 32);
      const uint32_t a_step = a_bytes >> 4, b_step = b_bytes >> 4;
      const uint32_t d0 = tmem + (uint32_t)(warp * BN);
      uint32_t seen = 0;
      auto run = [&](auto nk_c) {
        constexpr int NK = decltype(nk_c)::value;
        uint32_t phase = 0;
        int s = warp;
        for (int i = warp; i < mine; i += ni) {
          const uint32_t a_lo = (uint32_t)a0 + (uint32_t)s * a_step, b_lo = (uint32_t)b0 + (uint32_t)s * b_step;
          const uint32_t more = seen;
          if (!mbar_wait_warp(full_bar(s), phase, abort_flag)) {
            err_code = 3;
            return;
          }
          tc_fence_after();
          // activation part PA times N / BN filter parts from PB on, which lie one after the other, into
          // as many accumulators from D on
          auto products = [&](int pa, int pb, int d, uint32_t n, bool opens) {
#pragma unroll
            for (int kk = 0; kk < NK; ++kk)
              mma_warp(d0 + (uint32_t)(d * BN), a_lo + (uint32_t)pa * (a_tile >> 4) + 2u * kk, a_hi,
                       b_lo + (uint32_t)pb * (b_tile >> 4) + 2u * kk, b_hi, IDESC0 | (n << NSHIFT),
                       opens && kk == 0 ? more : 1u);
          };
          if constexpr (!SPLIT) {
            products(0, 0, 0, BN, true);
          } else if constexpr (BN == 128) {
            products(0, 0, 0, 2 * BN, true);
            products(0, 2, 1, BN, false);
            products(1, 0, 1, BN, false);
            products(1, 1, 1, BN, false);
            products(2, 0, 1, BN, false);
          } else {
            products(0, 0, 0, 3 * BN, true);
            products(1, 0, 1, 2 * BN, false);
            products(2, 0, 2, BN, false);
          }
          seen = 1u;
          if (i + stages < mine) commit_warp(empty_bar(s));   // nobody waits for the last ones
          s += ni;
          if (s >= stages) {   // (a ring as long as the share is never reused)
            s -= stages;
            phase ^= 1u;
          }
        }
        commit_warp(done_bar);
      };
      if (bk == 64) run(std::integral_constant<int, 4>{});
      else if (bk == 32) run(std::integral_constant<int, 2>{});
      else run(std::integral_constant<int, 1>{});
      used[warp] = (int)seen;
    }
      __syncwarp();
      if (!err_code && !mbar_wait(done_bar, 0, abort_flag)) err_code = 4;
      tc_fence_after();
      __syncthreads();   // bias_s, used
    }
#pragma unroll
    for (int w = 0; w < NI; ++w) used_all[w] = w >= ni ? 0 : real ? used[w] : 1;
    // CH columns of this thread's row from column h * CH on: the sum of the accumulators, which are all
    // requested before the first is waited for
    auto load_sum = [&](int h, uint32_t *r) {
      uint32_t t[NACC][CH];
#pragma unroll
      for (int k = 0; k < NACC; ++k) {
        if (used_all[SPLIT ? 0 : k]) {   // the same for all threads
          tc_ld<CH>(t_row + (uint32_t)(k * BN + h * CH), t[k]);
        } else {
#pragma unroll
          for (int j = 0; j < CH; ++j) t[k][j] = 0u;
        }
      }
      tc_ld_wait();
#pragma unroll
      for (int j = 0; j < CH; ++j) {
        float v = __uint_as_float(t[0][j]);
#pragma unroll
        for (int k = 1; k < NACC; ++k) v += __uint_as_float(t[k][j]);
        r[j] = __float_as_uint(v);
      }
    };
    if constexpr (ITEMS) {
      if constexpr (CL) {
        if (real) cluster_wait_acquire();   // every CTA of the cluster has started
      }
      const bool on = real && row < p.rows && !err_code;
#pragma unroll
      for (int h = 0; h < HALF / CH; ++h) {
        uint32_t r[CH];
        load_sum(h, r);
#pragma unroll
        for (int j = 0; j < CH / 4; ++j) {
          // 16-byte pieces of a row are permuted by its number: eight lanes, eight bank groups
          const uint32_t piece = (uint32_t)((part * HALF + h * CH) / 4 + j) ^ (uint32_t)(row & 7);
          if constexpr (CL)
            st_async_v4_if(on, dst + piece * 16u, dst_bar, r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
          else
            st_shared_v4_if(on, sX + (uint32_t)row * (BN * 4u) + piece * 16u, r[4 * j], r[4 * j + 1], r[4 * j + 2],
                            r[4 * j + 3]);
        }
      }
      __syncwarp();
      if constexpr (CL) {
        if (real && !err_code && !mbar_wait(sums_bar, 0, abort_flag)) err_code = 6;
      } else {
        if (real) __syncthreads();
      }
      const uint8_t *xs = smem_raw + (sX - sA);
      auto item = [&](bool live, int r, int g, const uint4 *rs) {
        r = live ? r : 0;
        g = live ? g : 0;
        const int lin = lin_s[row0 + r < 128 ? row0 + r : 0], c = tl.k0 + g * 8;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = bias_s[g * 8 + j];
        const uint32_t sw = (uint32_t)((row0 + r) & 7);
#pragma unroll 4
        for (int k = 0; k < splits; ++k) {
          const uint8_t *b = xs + (size_t)(k * p.rows_owner + r) * (BN * 4);
          const float4 a = *reinterpret_cast<const float4 *>(b + (((uint32_t)(2 * g)) ^ sw) * 16u);
          const float4 e = *reinterpret_cast<const float4 *>(b + (((uint32_t)(2 * g + 1)) ^ sw) * 16u);
          v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
          v[4] += e.x; v[5] += e.y; v[6] += e.z; v[7] += e.w;
        }
        const bool store = real && live && lin >= 0 && c < p.K && !err_code;
        if constexpr (SPLIT && !F32) sk_finish_parts(p, store, v, rs, lin, c);
        else finish(store, v, *rs, lin, c);
      };
      if (F32 && p.out_hw) {   // consecutive threads on consecutive pixels of one channel
        const int n = nrows > 0 ? nrows : 1, end = real ? items : (int)threadIdx.x + 1;
        for (int it = threadIdx.x; it < end; it += SK_THREADS) item(it < items, it % n, it / n, res);
      } else if constexpr (SPLIT && !F32) {
        constexpr int B = 2;   // residuals of so many items are requested at a time
#pragma unroll 1
        for (int u = 0; u < (real ? BN / 16 : B); u += B) {
          uint4 rs[B][3];
#pragma unroll
          for (int b = 0; b < B; ++b) {
            const int it = (int)threadIdx.x + (u + b) * SK_THREADS, r = it / G8, c = tl.k0 + (it % G8) * 8;
            const int lin = real && it < items ? lin_s[row0 + r] : -1;
            if (p.residual && lin >= 0 && c < p.K)
#pragma unroll
              for (int j = 0; j < 3; ++j)
                rs[b][j] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(p.residual) +
                                                            j * p.plane + (int64_t)lin * p.K + c);
          }
#pragma unroll
          for (int b = 0; b < B; ++b) {
            const int it = (int)threadIdx.x + (u + b) * SK_THREADS;
            item(it < items, it / G8, it % G8, rs[b]);
          }
        }
      } else {
#pragma unroll
        for (int u = 0; u < BN / 16; ++u) {
          const int it = (int)threadIdx.x + u * SK_THREADS;
          if (u == 0 || it < items) item(it < items, it / G8, it % G8, res + u);
        }
      }
    } else {
#pragma unroll
      for (int h = 0; h < HALF / CH; ++h) {
        uint32_t r[CH];
        load_sum(h, r);
#pragma unroll
        for (int u = 0; u < CH / 8; ++u) {
          const int cl = part * HALF + h * CH + u * 8;
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[u * 8 + j]) + bias_s[cl + j];
          finish(real && lin_row >= 0 && tl.k0 + cl < p.K && !err_code, v, res[h * (CH / 8) + u], lin_row,
                 tl.k0 + cl);
        }
      }
    }
    tc_fence_before();
  }

  if (err_code) {
    atomicExch(p.err, 1000 + err_code);
    *abort_flag = 1;
    for (int i = 0; i < 50; ++i) __nanosleep(20000);   // copies in flight land before memory goes
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CL) {
    // A CTA that has its partial sums has heard from all the others and may go.  One that gave up stays
    // until the others have gone (each of their waits is bounded): they may still be sending to it.
    if (*abort_flag) {
      cluster_arrive_release();
      cluster_wait_acquire();
    }
  }
  if (warp == 3)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(cols)
                 : "memory");
}

size_t sk_smem_bytes(int bn, int stages, int a_bytes, int bk, int splits, int rows_owner, bool split) {
  const size_t ring = (size_t)stages * sk_parts(split) * (a_bytes + bn * bk * 2);
  const size_t x = (size_t)splits * rows_owner * bn * 4;
  return (splits > 1 ? ring + x : split && x > ring ? x : ring) + bn * 4 + 512 + 8 * (2 * stages + 7);
}

template <int BN, bool F16, bool SPLIT, bool CL, bool F32>
static void sk_launch_one(const SkParams &p, int tiles, size_t smem, cudaStream_t s) {
  auto kernel = tc_split_kernel<BN, F16, SPLIT, CL, F32>;
  static unsigned char attr_done[TC_MAX_DEVICES] = {};
  if (tc_first_use_on_device(attr_done)) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT);
    cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  }
  tc_launch_pdl(kernel, tiles * p.splits, SK_THREADS, smem, s, p, p.splits);
}

template <int BN>
static void sk_launch_bn(const SkParams &p, bool f16, bool split, int tiles, size_t smem, cudaStream_t s) {
  const bool cl = p.splits > 1, f32 = p.out_f32 != nullptr;
  if (split) {
    if (cl && f32) sk_launch_one<BN, false, true, true, true>(p, tiles, smem, s);
    else if (cl) sk_launch_one<BN, false, true, true, false>(p, tiles, smem, s);
    else if (f32) sk_launch_one<BN, false, true, false, true>(p, tiles, smem, s);
    else sk_launch_one<BN, false, true, false, false>(p, tiles, smem, s);
  } else if (f16) {
    if (cl && f32) sk_launch_one<BN, true, false, true, true>(p, tiles, smem, s);
    else if (cl) sk_launch_one<BN, true, false, true, false>(p, tiles, smem, s);
    else if (f32) sk_launch_one<BN, true, false, false, true>(p, tiles, smem, s);
    else sk_launch_one<BN, true, false, false, false>(p, tiles, smem, s);
  } else {
    if (cl && f32) sk_launch_one<BN, false, false, true, true>(p, tiles, smem, s);
    else if (cl) sk_launch_one<BN, false, false, true, false>(p, tiles, smem, s);
    else if (f32) sk_launch_one<BN, false, false, false, true>(p, tiles, smem, s);
    else sk_launch_one<BN, false, false, false, false>(p, tiles, smem, s);
  }
}

bool sk_launch(const SkParams &p, int bn, bool f16, bool split, int tiles, size_t smem, cudaStream_t s) {
  if (bn == 32) sk_launch_bn<32>(p, f16, split, tiles, smem, s);
  else if (bn == 64) sk_launch_bn<64>(p, f16, split, tiles, smem, s);
  else if (bn == 128) sk_launch_bn<128>(p, f16, split, tiles, smem, s);
  else return false;
  return true;
}

}  // namespace occ
