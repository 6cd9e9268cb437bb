// Few-channel convolution (an RGB stem) fused with the 3x3 / stride 2 / pad 1 max pool that
// follows it: conv + bias + clamp + pool in one pass, the full-resolution convolution
// output never leaves the SM.
//
// Input: the padded channels-last image rows the folded convolution uses,
// x[n][h][wp][Cp] bf16 with 16 bytes per output-column step, so the A vector of output
// column q (Cf = Sp*Cp values starting at pixel q*stride) is a window at byte 16*q of the
// row and neighbouring windows overlap.  One MMA row block is one convolution output row
// (Q <= 128 columns).
//   TILED  TMA writes a row's windows out side by side (a tensor map whose pixel stride is shorter than its innermost
//          extent), rows of 32, 64 or 128 bytes in the swizzle of that width.  Four times the bytes in shared memory.
//   else   a row is copied once and the tensor core reads the overlapping windows in place: the operand descriptor is
//          the un-swizzled K-major form with 16 bytes from one 8-element K chunk to the next and 128 bytes from one
//          group of 8 rows to the next, "row m starts at byte 16*m".
// 256 images of 224x224: 139 us tiled, 155 in place; the first where its shared memory suffices.
//
// One persistent CTA per SM works through units of (image, band of pooled rows):
//   warp 0      producer: the weights once, then input rows into a ring
//   2 warps     MMA issuers (alternate convolution rows): per row R taps x
//               Cf/16 tcgen05.mma (128 x 64 x 16) into one of four TMEM accumulators;
//               release input rows
//   16 warps    epilogue: accumulator -> + bias -> clamp -> bf16, the largest of a window's three
//               rows in registers (a thread owns 16 channels of one column) -> a buffer in shared
//               memory (swizzled so that a warp's 128-byte rows spread over banks)
//   4 warps     pool: the largest of three columns -> global memory
// Every wait is bounded; a wait that runs out records a code and the kernel drains.
#include <map>

#include "conv_tc_dev.cuh"
#include "kernels.h"
#include "runtime.h"

namespace occ {

namespace {

constexpr int ST_EPI_WARPS = 16;   // four per TMEM lane quadrant, 16 channels each
constexpr int ST_POOL_WARPS = 4;
constexpr int ST_ISSUERS = 2;
// warps: producer, the first issuer, epilogue, pool, the other issuers
constexpr int ST_ISSUER_B = 2 + ST_EPI_WARPS + ST_POOL_WARPS;
constexpr int ST_THREADS = 32 * (ST_ISSUER_B + ST_ISSUERS - 1);
constexpr int ST_MAX_CHUNKS = 8;   // of the input ring (StemParams::ring)
constexpr int ST_NMR = 3;     // buffers of a pooled row before its columns are taken together
constexpr int ST_NACC = 4;    // TMEM accumulators (64 columns each)
constexpr int ST_K = 64;      // output channels

struct alignas(64) StemParams {
  CUtensorMap tmX, tmW;   // TILED
  const bf16 *x;       // [N][H][row_bytes / 2]
  const bf16 *w;       // packed [R][Cf / 8][64][8]
  const float *bias;   // [64] or null
  bf16 *y;             // [N][PP][QP][64]
  int N, H, row_bytes;
  int in_row, slot_bytes;     // an input row in shared memory, a group of stride_h of them
  int bk;                     // TILED: channels of a window there (16, 32 or 64)
  int ring, chunk;            // groups the input ring holds, and how many of them one copy brings (powers of two)
  int G;                      // groups one convolution row reads
  int P, Q;            // convolution output
  int R, Cf, pad_h, stride_h;
  int PP, QP;          // pooled output
  int bands, band_rows, units;
  int mr_bytes;        // bytes of such a buffer
  float lo, hi;
  int descending;      // units are taken from the last to the first (Runtime::descending)
  int *err;
};

// An MMA that is issued only when `valid` is non-zero (a predicated instruction, not a branch:
// a taken branch costs the issuing warp more than the MMA it would skip).
__device__ __forceinline__ void mma_lohi_if(uint32_t valid, uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi,
                                            uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p, q, e;\n.reg .b64 da, db;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "elect.sync _|e, 0xffffffff;\n"
      "setp.ne.and.b32 q, %7, 0, e;\n"
      "mov.b64 da, {%1, %2};\n"
      "mov.b64 db, {%3, %4};\n"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}" ::"r"(d_tmem),
      "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(valid)
      : "memory");
}

// All MMAs of one convolution row, straight-line: R taps x KK K-steps, taps outside
// [r_lo, r_hi] predicated off.  Tap r reads row r % SH of the group in ring slot
// s0 + r / SH.
template <int R, int KK, int SH>
__device__ __forceinline__ void issue_row(uint32_t d_tmem, int r_lo, int r_hi, uint32_t s0,
                                          uint32_t ring, uint32_t a_lo0, uint32_t a_hi, uint32_t slot_desc,
                                          uint32_t row_desc, uint32_t b_lo0, uint32_t b_hi,
                                          uint32_t tap_desc, uint32_t kstep_desc, uint32_t idesc) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t valid = (r >= r_lo && r <= r_hi) ? 1u : 0u;
    const uint32_t s = (s0 + (uint32_t)(r / SH)) & (ring - 1u);
    const uint32_t a_lo = a_lo0 + s * slot_desc + (uint32_t)(r % SH) * row_desc;
    const uint32_t b_lo = b_lo0 + (uint32_t)r * tap_desc;
#pragma unroll
    for (int kk = 0; kk < KK; ++kk)
      mma_lohi_if(valid, d_tmem, a_lo + 2 * kk, a_hi, b_lo + kk * kstep_desc, b_hi, idesc,
                  (r != r_lo || kk != 0) ? 1u : 0u);
  }
}

// ... of a row whose taps all lie inside the image.
template <int R, int KK, int SH>
__device__ __forceinline__ void issue_whole_row(uint32_t d_tmem, uint32_t s0, uint32_t ring, uint32_t a_lo0, uint32_t a_hi,
                                                uint32_t slot_desc, uint32_t row_desc, uint32_t b_lo0, uint32_t b_hi,
                                                uint32_t tap_desc, uint32_t kstep_desc, uint32_t idesc) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t s = (s0 + (uint32_t)(r / SH)) & (ring - 1u);
    const uint32_t a_lo = a_lo0 + s * slot_desc + (uint32_t)(r % SH) * row_desc, b_lo = b_lo0 + (uint32_t)r * tap_desc;
#pragma unroll
    for (int kk = 0; kk < KK; ++kk)
      mma_warp(d_tmem, a_lo + 2 * kk, a_hi, b_lo + kk * kstep_desc, b_hi, idesc, (r | kk) ? 1u : 0u);
  }
}

// byte offset of 16-byte chunk `c` (0..7) of pixel `px` in such a buffer
__device__ __forceinline__ uint32_t mr_off(int px, int c) {
  return (uint32_t)(px * 128 + ((c ^ (px & 7)) << 4));
}

template <bool TILED>
__global__ void __launch_bounds__(ST_THREADS, 1) stem_pool_kernel(const __grid_constant__ StemParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t w_tap = (uint32_t)(TILED ? p.bk : p.Cf) * ST_K * 2, w_bytes = (uint32_t)p.R * w_tap;
  const uint32_t sW = base;
  const uint32_t sIn = sW + ((w_bytes + 1023u) & ~1023u);
  // (the MMA rows beyond Q reach into what lies behind a row: read, and left out; stem_pool_layout() has room for it)
  const uint32_t sMr = sIn + ((p.ring * p.slot_bytes + 1023u) & ~1023u);
  const uint32_t sMisc = sMr + ST_NMR * p.mr_bytes;
  uint8_t *misc_ptr = base_ptr + (sMisc - base);
  float *bias_s = reinterpret_cast<float *>(misc_ptr);                 // 64 floats
  uint64_t *bars = reinterpret_cast<uint64_t *>(misc_ptr + 256);
  const uint32_t bar0 = sMisc + 256;
  const uint32_t w_full = bar0;
  auto in_full = [&](int s) { return bar0 + 8u * (1 + s); };
  auto in_empty = [&](int s) { return bar0 + 8u * (1 + ST_MAX_CHUNKS + s); };
  auto tfull = [&](int s) { return bar0 + 8u * (1 + 2 * ST_MAX_CHUNKS + s); };
  auto tempty = [&](int s) { return bar0 + 8u * (1 + 2 * ST_MAX_CHUNKS + ST_NACC + s); };
  auto mr_full = [&](int s) { return bar0 + 8u * (1 + 2 * ST_MAX_CHUNKS + 2 * ST_NACC + s); };
  auto mr_empty = [&](int s) { return bar0 + 8u * (1 + 2 * ST_MAX_CHUNKS + 2 * ST_NACC + ST_NMR + s); };
  constexpr int NBARS = 1 + 2 * ST_MAX_CHUNKS + 2 * ST_NACC + 2 * ST_NMR;
  volatile uint32_t *tmem_holder = reinterpret_cast<volatile uint32_t *>(bars + NBARS);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + NBARS + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  constexpr uint32_t TMEM_COLS = ST_NACC * ST_K;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int s = 0; s < p.ring / p.chunk; ++s) {
      mbar_init(in_full(s), 1);
      mbar_init(in_empty(s), ST_ISSUERS);   // every MMA issuer hands a group back
    }
    for (int s = 0; s < ST_NACC; ++s) {
      mbar_init(tfull(s), 1);
      mbar_init(tempty(s), ST_EPI_WARPS);
    }
    for (int s = 0; s < ST_NMR; ++s) {
      mbar_init(mr_full(s), ST_EPI_WARPS);
      mbar_init(mr_empty(s), ST_POOL_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < ST_K) bias_s[threadIdx.x] = p.bias ? p.bias[threadIdx.x] : 0.0f;
  fence_async_smem();
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void *)tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  int err_code = 0;
  pdl_launch_dependents();   // the next kernel's prologue may overlap this one
  pdl_wait();

  // pooled rows [i0, i1) and convolution rows [h_lo, h_hi] of a unit
  auto unit_rows = [&](int unit, int &n, int &i0, int &i1, int &h_lo, int &h_hi) {
    if (p.descending) unit = p.units - 1 - unit;
    n = unit / p.bands;
    const int b = unit - n * p.bands;
    i0 = b * p.band_rows;
    i1 = min(i0 + p.band_rows, p.PP);
    h_lo = max(2 * i0 - 1, 0);
    h_hi = min(2 * (i1 - 1) + 1, p.P - 1);
  };

  const uint32_t chunks = (uint32_t)(p.ring / p.chunk);
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    // Group g of a unit is rows (h_lo + g) * stride_h - pad_h ... + stride_h - 1; convolution row k of the unit reads
    // groups k ... k + G - 1 and is the last reader of group k.  `chunk` groups lie next to one another in memory
    // and come in one copy.
    {
      expect_tx_warp(w_full, w_bytes);
      if constexpr (TILED) {
        for (int r = 0; r < p.R; ++r) load_3d_warp(sW + r * w_tap, &p.tmW, w_full, 0, 0, r);
      } else {
        bulk_load_warp(sW, p.w, w_bytes, w_full);
      }
      uint32_t q = 0;   // chunks loaded so far
      for (int unit = blockIdx.x; unit < p.units && !err_code; unit += gridDim.x) {
        int n, i0, i1, h_lo, h_hi;
        unit_rows(unit, n, i0, i1, h_lo, h_hi);
        const uint8_t *img = reinterpret_cast<const uint8_t *>(p.x) + (size_t)n * p.H * p.row_bytes;
        const int groups = h_hi - h_lo + p.G;
        for (int g = 0; g < groups; g += p.chunk, ++q) {
          const uint32_t s = q % chunks, ph = (q / chunks) & 1u;
          if (!mbar_wait_warp(in_empty(s), ph ^ 1u, abort_flag)) {
            err_code = 1;
            break;
          }
          const int j0 = (h_lo + g) * p.stride_h - p.pad_h;
          if constexpr (TILED) {   // (rows outside the image arrive as zeros)
            expect_tx_warp(in_full(s), (uint32_t)(p.chunk * p.slot_bytes));
            load_4d_warp(sIn + s * p.chunk * p.slot_bytes, &p.tmX, in_full(s), 0, 0, j0, n);
            continue;
          }
          const int lo = max(j0, 0), hi = min(j0 + min(p.chunk, groups - g) * p.stride_h, p.H);
          const uint32_t bytes = hi > lo ? (uint32_t)((hi - lo) * p.row_bytes) : 0u;
          expect_tx_warp(in_full(s), bytes);   // 0 bytes: a plain arrival
          if (bytes)
            bulk_load_warp(sIn + s * p.chunk * p.slot_bytes + (lo - j0) * p.row_bytes, img + (size_t)lo * p.row_bytes, bytes,
                     in_full(s));
        }
      }
    }
  } else if (warp == 1 || warp >= ST_ISSUER_B) {
    // ------------------------------------------------------------ MMA issuers
    // Two warps take alternate convolution rows: the MMAs are short (64
    // columns) and one cannot issue them as fast as the tensor core retires them.
    // Both read every input group, so a group goes back to the producer when both have
    // committed it (each does so once it will not read the group again).
    {
      const int me = warp == 1 ? 0 : warp - ST_ISSUER_B + 1;
      constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) |
                                 ((uint32_t)(ST_K >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      if (!mbar_wait_warp(w_full, 0, abort_flag)) err_code = 2;
      uint32_t gbase = 0;   // ring index of the unit's first group (whole chunks)
      uint32_t cbase = 0;   // convolution rows before this unit
      const int kk_n = (TILED ? p.bk : p.Cf) / 16;
      const uint64_t adesc0 = TILED ? make_smem_desc(sIn, p.bk) : desc_plain(sIn, 16, 128);
      const uint64_t bdesc0 = TILED ? make_smem_desc(sW, p.bk) : desc_plain(sW, ST_K * 16, 128);
      const uint32_t a_lo0 = (uint32_t)adesc0, a_hi = (uint32_t)(adesc0 >> 32);
      const uint32_t b_lo0 = (uint32_t)bdesc0, b_hi = (uint32_t)(bdesc0 >> 32);
      const uint32_t slot_desc = (uint32_t)p.slot_bytes >> 4;        // descriptor steps
      const uint32_t row_desc = (uint32_t)p.in_row >> 4, ring = (uint32_t)p.ring;
      const uint32_t tap_desc = w_tap >> 4;
      const uint32_t kstep_desc = TILED ? 2u : (2 * ST_K * 16) >> 4;
      for (int unit = blockIdx.x; unit < p.units && !err_code; unit += gridDim.x) {
        int n, i0, i1, h_lo, h_hi;
        unit_rows(unit, n, i0, i1, h_lo, h_hi);
        const int rows = h_hi - h_lo + 1;
        const int groups = (rows + p.G - 1 + p.chunk - 1) / p.chunk * p.chunk;   // of the chunks loaded for this unit
        int waited = 0, released = 0;             // groups (unit-relative) waited for / committed
        auto arrived = [&](int upto) {
          for (; waited < upto; waited += p.chunk) {
            const uint32_t q = (gbase + (uint32_t)waited) / (uint32_t)p.chunk;
            if (!mbar_wait_warp(in_full(q % chunks), (q / chunks) & 1u, abort_flag)) {
              err_code = 4;
              return false;
            }
          }
          return true;
        };
        // chunks whose groups are all below `upto` are of no more use to me (none is handed back before it has come, or this thread
        // could be a turn of the ring ahead of the others)
        auto release = [&](int upto) {
          for (; released + p.chunk <= upto; released += p.chunk) {
            if (!arrived(released + 1)) return;
            commit_warp(in_empty((gbase + (uint32_t)released) / (uint32_t)p.chunk % chunks));
          }
        };
        // rows of the unit whose running number (over all units) has my parity
        for (int k = (int)(((uint32_t)me + ST_ISSUERS - cbase % ST_ISSUERS) % ST_ISSUERS); k < rows && !err_code; k += ST_ISSUERS) {
          const uint32_t c = cbase + (uint32_t)k;
          const uint32_t a = c % ST_NACC, aph = (c / ST_NACC) & 1u;
          if (!mbar_wait_warp(tempty(a), aph ^ 1u, abort_flag)) {
            err_code = 3;
            break;
          }
          if (!arrived(k + p.G)) break;            // row k reads groups k ... k + G - 1
          tc_fence_after();
          // taps whose input row lies inside the image (a row of padding contributes nothing)
          const int h = h_lo + k;
          const int jb = h * p.stride_h - p.pad_h;
          const int r_lo = max(0, -jb), r_hi = min(p.R - 1, p.H - 1 - jb);
          const uint32_t d_tmem = tmem_base + a * ST_K;
          const uint32_t s0 = (gbase + (uint32_t)k) & (ring - 1u);
          // The issue code is straight-line: every taken branch costs the issuing warp more
          // than an MMA.
          if (p.R == 7 && kk_n == 2 && p.stride_h == 2 && r_lo == 0 && r_hi == 6) {
            issue_whole_row<7, 2, 2>(d_tmem, s0, ring, a_lo0, a_hi, slot_desc, row_desc, b_lo0, b_hi, tap_desc, kstep_desc,
                                     IDESC);
          } else if (p.R == 7 && kk_n == 2 && p.stride_h == 2) {
            issue_row<7, 2, 2>(d_tmem, r_lo, r_hi, s0, ring, a_lo0, a_hi, slot_desc, row_desc, b_lo0, b_hi,
                               tap_desc, kstep_desc, IDESC);
          } else {
            uint32_t accumulate = 0;
            for (int r = r_lo; r <= r_hi; ++r) {
              const uint32_t s = (s0 + (uint32_t)(r / p.stride_h)) & (ring - 1u);
              const uint32_t a_lo = a_lo0 + s * slot_desc + (uint32_t)(r % p.stride_h) * row_desc;
              const uint32_t b_lo = b_lo0 + (uint32_t)r * tap_desc;
              // 16 K values further on: 32 bytes along the row for A, two K chunks for B
              for (int kk = 0; kk < kk_n; ++kk) {
                mma_warp(d_tmem, a_lo + 2 * kk, a_hi, b_lo + kk * kstep_desc, b_hi, IDESC, accumulate);
                accumulate = 1;
              }
            }
          }
          commit_warp(tfull(a));
          release(min(k + ST_ISSUERS, groups));   // (my next row)
        }
        // whatever of the unit I have not committed yet (also when none of its rows was mine)
        if (!err_code) release(groups);
        gbase += (uint32_t)groups;
        cbase += (uint32_t)rows;
      }
      // The last commits are waited for, so that none arrives when this CTA has gone.
      if (!err_code && gbase) {
        const uint32_t q = gbase / (uint32_t)p.chunk - 1;
        if (!mbar_wait_warp(in_empty(q % chunks), (q / chunks) & 1u, abort_flag)) err_code = 8;
      }
    }
  } else if (warp < 2 + ST_EPI_WARPS) {
    // ------------------------------------------------------------ epilogue
    // The accumulator of the next row is requested before this one's is worked on.  What bounds the kernel: a row's 14
    // MMAs (680 cycles of the tensor core, 48 each whatever N up to 64), and the chain from a row's last product to its
    // accumulator being free again, which sixteen warps shorten: 256 images at 224x224, 167 us with eight warps here, eight
    // for 3x3 windows of a ring of rows, and issuers and loader that were single lanes; eight and four 160; sixteen and
    // four 137 to 139; three issuers 148, one 184.
    const int quad = warp & 3;               // TMEM lane quadrant this warp may read
    const int part = (warp - 2) >> 2;        // channels [16 * part, 16 * part + 16)
    const int px = quad * 32 + lane;         // convolution output column
    const float lo = p.lo, hi = p.hi;
    const bool relu_only = lo == 0.0f && hi == INFINITY;
    uint32_t off[2];                         // this thread's two 16-byte pieces of a buffer
#pragma unroll
    for (int k = 0; k < 2; ++k) off[k] = mr_off(px, part * 2 + k);
    const uint32_t t_row = tmem_base + ((uint32_t)(quad * 32) << 16) + part * 16;
    uint32_t c = 0, pooled = 0;              // rows and pooled rows so far
    int unit = blockIdx.x, n, i0, i1, h_lo = 0, h_hi = 0, h = 0;
    uint32_t m[8], prev[8];                 // largest so far of the window's rows; its last row, the next one's first
    auto request = [&](uint32_t *r) -> bool {   // the accumulator of row `c`
      if (!mbar_wait_hot(tfull(c % ST_NACC), (c / ST_NACC) & 1u, abort_flag)) {
        err_code = 5;
        return false;
      }
      tc_fence_after();
      tc_ld16(t_row + (c % ST_NACC) * ST_K, r);
      return true;
    };
    // one row, whose accumulator arrives in `r`; false when it was the last
    auto row = [&](uint32_t *r, uint32_t *next) -> bool {
      const int this_h = h, this_lo = h_lo;
      tc_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty(c % ST_NACC));
      ++c;
      if (++h > h_hi) {
        unit += gridDim.x;
        if (unit < p.units) {
          unit_rows(unit, n, i0, i1, h_lo, h_hi);
          h = h_lo;
        }
      }
      const bool more = unit < p.units;
      if (more && !request(next)) return false;
      uint32_t pk[8];
      const float4 *b4 = reinterpret_cast<const float4 *>(bias_s + part * 16);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 b = b4[j];
        const uint64_t v0 =
            f2_add(f2_pack(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1])), f2_pack(b.x, b.y));
        const uint64_t v1 =
            f2_add(f2_pack(__uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])), f2_pack(b.z, b.w));
        if (relu_only) {
          pk[2 * j] = f2_to_bf16x2_relu(v0);
          pk[2 * j + 1] = f2_to_bf16x2_relu(v1);
        } else {
          float x0, x1, x2, x3;
          f2_unpack(v0, x0, x1);
          f2_unpack(v1, x2, x3);
          pk[2 * j] = f2_to_bf16x2(f2_pack(tc_clip(x0, lo, hi), tc_clip(x1, lo, hi)));
          pk[2 * j + 1] = f2_to_bf16x2(f2_pack(tc_clip(x2, lo, hi), tc_clip(x3, lo, hi)));
        }
      }
      // Pooled row i takes rows 2i - 1 ... 2i + 1, those of them that exist.
      if (this_h & 1) {
        if (this_h == this_lo) {   // the unit's first row belongs to the window above as well
#pragma unroll
          for (int j = 0; j < 8; ++j) prev[j] = pk[j];
          return more;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          m[j] = tc_max2<false>(m[j], pk[j]);
          prev[j] = pk[j];
        }
      } else {
        const bool first = this_h == 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) m[j] = first ? pk[j] : tc_max2<false>(prev[j], pk[j]);
        if (this_h != p.P - 1) return more;
      }
      const uint32_t buf = pooled % ST_NMR, buf_phase = (pooled / ST_NMR) & 1u;
      uint8_t *mr = base_ptr + (sMr - base) + buf * p.mr_bytes;
      ++pooled;
      if (!mbar_wait_hot(mr_empty(buf), buf_phase ^ 1u, abort_flag)) {
        err_code = 6;
        return false;
      }
      if (px < p.Q) {
#pragma unroll
        for (int k = 0; k < 2; ++k)
          *reinterpret_cast<uint4 *>(mr + off[k]) = make_uint4(m[4 * k], m[4 * k + 1], m[4 * k + 2], m[4 * k + 3]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(mr_full(buf));
      return more;
    };
    if (unit < p.units) {
      unit_rows(unit, n, i0, i1, h_lo, h_hi);
      h = h_lo;
      uint32_t ra[16], rb[16];
      if (request(ra)) {
#pragma unroll 1
        while (row(ra, rb) && row(rb, ra)) {
        }
      }
    }
  } else {
    // ------------------------------------------------------------ pool
    const int pt = threadIdx.x - 32 * (2 + ST_EPI_WARPS);
    const int items = p.QP * 8;              // (pooled column, 16-byte channel chunk)
    uint32_t pooled = 0;
    for (int unit = blockIdx.x; unit < p.units && !err_code; unit += gridDim.x) {
      int n, i0, i1, h_lo, h_hi;
      unit_rows(unit, n, i0, i1, h_lo, h_hi);
      for (int i = i0; i < i1; ++i, ++pooled) {
        const uint32_t buf = pooled % ST_NMR;
        if (!mbar_wait_sleepy(mr_full(buf), (pooled / ST_NMR) & 1u, abort_flag)) {
          err_code = 7;
          break;
        }
        const uint8_t *mr = base_ptr + (sMr - base) + buf * p.mr_bytes;
        bf16 *yrow = p.y + ((size_t)n * p.PP + i) * p.QP * ST_K;
        for (int it = pt; it < items; it += 32 * ST_POOL_WARPS) {
          const int jq = it >> 3, ch = it & 7;
          // (a column outside the image is replaced by the nearest inside it: a duplicate changes no maximum)
          const uint4 a = *reinterpret_cast<const uint4 *>(mr + mr_off(max(2 * jq - 1, 0), ch));
          const uint4 b = *reinterpret_cast<const uint4 *>(mr + mr_off(2 * jq, ch));
          const uint4 d = *reinterpret_cast<const uint4 *>(mr + mr_off(min(2 * jq + 1, p.Q - 1), ch));
          *reinterpret_cast<uint4 *>(yrow + (size_t)jq * ST_K + ch * 8) =
              make_uint4(tc_max2<false>(tc_max2<false>(a.x, b.x), d.x), tc_max2<false>(tc_max2<false>(a.y, b.y), d.y),
                         tc_max2<false>(tc_max2<false>(a.z, b.z), d.z), tc_max2<false>(tc_max2<false>(a.w, b.w), d.w));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(mr_empty(buf));
      }
    }
  }

  if (err_code) {
    atomicExch(p.err, 1100 + err_code);
    *abort_flag = 1;
    for (int i = 0; i < 50; ++i) __nanosleep(20000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(TMEM_COLS)
                 : "memory");
  }
}

// fp32 KCRS (C <= Cp) -> bf16 [R][Cf/8][64][8]: tap row r, K chunk j, output channel n, and
// within the chunk k = 8j + e = s*Cp + c.
__global__ void pack_stem_kernel(const float *__restrict__ w, bf16 *__restrict__ out, int C, int R,
                                 int S, int Cp, int Cf, int total) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int e = i & 7;
    const int n = (i >> 3) % ST_K;
    const int j = (i / (8 * ST_K)) % (Cf / 8);
    const int r = i / (8 * ST_K * (Cf / 8));
    const int k = j * 8 + e;
    const int s2 = k / Cp, c = k % Cp;
    float v = 0.0f;
    if (s2 < S && c < C) v = w[(((int64_t)n * C + c) * R + r) * S + s2];
    out[i] = __float2bfloat16_rn(v);
  }
}

}  // namespace

bool stem_pool_supported(const StemPoolArgs &a) {
  if (a.K != ST_K || a.Cf % 16 || a.Cf > 64 || a.R < 1 || a.R > 11) return false;
  if (a.w_step_bytes != 16 || a.row_bytes % 16 || a.row_bytes > 8192) return false;
  if (a.Q < 1 || a.Q > 128 || a.P < 1 || a.stride_h < 1 || a.stride_h > 4) return false;
  if ((a.R - 1) / a.stride_h + 1 > 6) return false;   // groups a row holds at once
  if (a.pad_h >= a.R) return false;   // every row of the output has a filter row inside the image
  if (a.PP != (a.P + 2 - 3) / 2 + 1 || a.QP != (a.Q + 2 - 3) / 2 + 1) return false;
  if ((uintptr_t)a.x % 16 || (uintptr_t)a.w % 16 || (uintptr_t)a.y % 16) return false;
  // the last window the tensor core reads for a real column must lie inside the row
  if (16 * (a.Q - 1) + a.Cf * 2 > a.row_bytes) return false;
  return true;
}

size_t stem_pool_weight_bytes(int R, int Cf) { return (size_t)R * Cf * ST_K * 2; }

void launch_pack_stem_bf16(const float *w, bf16 *out, int C, int R, int S, int Cp, int Cf,
                           cudaStream_t s) {
  const int total = R * Cf * ST_K;
  launch_apart(pack_stem_kernel, (total + 255) / 256, 256, s, w, out, C, R, S, Cp, Cf, total);
  count(CNT_LAUNCHES);
}

// As many groups of input rows as fit, sixteen or eight; tiled where that suffices.
bool stem_pool_layout(int R, int Cf, int stride_h, int Q, int row_bytes, bool may_tile, StemPoolLayout *l) {
  auto fits = [&](bool tiled, int ring, int chunk) {
    l->tiled = tiled;
    l->ring = ring;
    l->chunk = chunk;
    l->bk = Cf <= 16 ? 16 : Cf <= 32 ? 32 : 64;
    l->in_row = tiled ? (Q + 7) / 8 * 8 * l->bk * 2 : row_bytes;
    l->slot_bytes = l->in_row * stride_h;
    l->mr_bytes = (Q * 128 + 1023) / 1024 * 1024;
    l->in_at = (R * (tiled ? l->bk : Cf) * ST_K * 2 + 1023) / 1024 * 1024;
    const int ring_bytes = ring * l->slot_bytes;
    const int used = l->in_at + (ring_bytes + 1023) / 1024 * 1024 + ST_NMR * l->mr_bytes + 256 + 8 * 64;
    // An MMA reads 128 windows from the start of a row, of the ring's last one too, however few the row has.
    const int reach = l->in_at + ring_bytes - l->in_row + (tiled ? 128 * l->bk * 2 : 127 * 16 + Cf * 2);
    l->smem = 1024 + (used > reach ? used : reach);   // (the first 1024 to align the rest)
    // at least half of the shared memory, so that one CTA (one TMEM allocation) runs per SM
    if (l->smem < 120 * 1024) l->smem = 120 * 1024;
    return l->smem <= TC_SMEM_LIMIT;
  };
  return (may_tile && (fits(true, 16, 4) || fits(true, 8, 2))) || fits(false, 16, 4) || fits(false, 8, 1);
}

namespace {

struct StemPlan {
  StemParams p;
  StemPoolLayout l;
  int grid;
  bool ok;
};

StemPlan stem_plan(const StemPoolArgs &a, int *err_word, int num_sms) {
  StemPlan pl;
  memset(&pl, 0, sizeof(pl));
  StemParams &p = pl.p;
  StemPoolLayout &l = pl.l;
  if (!stem_pool_supported(a)) return pl;
  p.x = a.x; p.w = a.w; p.bias = a.bias; p.y = a.y;
  p.N = a.N; p.H = a.H; p.row_bytes = a.row_bytes;
  p.G = (a.R - 1) / a.stride_h + 1;
  p.P = a.P; p.Q = a.Q; p.R = a.R; p.Cf = a.Cf; p.pad_h = a.pad_h; p.stride_h = a.stride_h;
  p.PP = a.PP; p.QP = a.QP;
  p.lo = a.lo; p.hi = a.hi;
  p.err = err_word;
  // bands: enough units to balance the SMs, each band re-computes one convolution row
  int bands = 1;
  while ((int64_t)a.N * bands < 6ll * num_sms && a.PP / (bands * 2) >= 4) bands *= 2;
  p.bands = bands;
  p.band_rows = (a.PP + bands - 1) / bands;
  p.bands = (a.PP + p.band_rows - 1) / p.band_rows;
  p.units = a.N * p.bands;
  if (p.units == 0 || !stem_pool_layout(a.R, a.Cf, a.stride_h, a.Q, a.row_bytes, a.w_fold != nullptr, &l)) return pl;
  p.ring = l.ring; p.chunk = l.chunk; p.bk = l.bk;
  p.in_row = l.in_row; p.slot_bytes = l.slot_bytes; p.mr_bytes = l.mr_bytes;
  if (l.tiled) {
    const uint64_t dims[4] = {(uint64_t)a.Cf, (uint64_t)a.Q, (uint64_t)a.H, (uint64_t)a.N};
    const uint64_t st[3] = {16, (uint64_t)a.row_bytes, (uint64_t)a.H * a.row_bytes};
    const uint32_t box[4] = {(uint32_t)p.bk, (uint32_t)(a.Q + 7) / 8 * 8, (uint32_t)(a.stride_h * p.chunk), 1};
    const uint64_t wdims[3] = {(uint64_t)a.Cf, ST_K, (uint64_t)a.R};
    const uint64_t wst[2] = {(uint64_t)a.Cf * 2, (uint64_t)a.Cf * 2 * ST_K};
    const uint32_t wbox[3] = {(uint32_t)p.bk, ST_K, 1};
    if (!make_map(&p.tmX, a.x, 4, dims, st, box, p.bk * 2, true) || !make_map(&p.tmW, a.w_fold, 3, wdims, wst, wbox, p.bk * 2, true))
      return pl;
  }
  pl.grid = p.units < num_sms ? p.units : num_sms;
  pl.ok = true;
  return pl;
}

}  // namespace

bool launch_stem_pool(const StemPoolArgs &a, int *err_word, int num_sms, cudaStream_t s) {
  struct Key {
    unsigned char b[sizeof(StemPoolArgs)];
    bool operator<(const Key &o) const { return memcmp(b, o.b, sizeof(b)) < 0; }
  };
  static std::map<Key, StemPlan> plans;   // (two tensor maps take longer to encode than the launch)
  Key key;
  memcpy(key.b, &a, sizeof(key.b));
  auto it = plans.find(key);
  if (it == plans.end()) {
    if (plans.size() > 256) plans.clear();
    it = plans.emplace(key, stem_plan(a, err_word, num_sms)).first;
  }
  StemPlan &pl = it->second;
  if (!pl.ok) return false;
  auto kernel = pl.l.tiled ? stem_pool_kernel<true> : stem_pool_kernel<false>;
  static unsigned char attr_done[TC_MAX_DEVICES] = {};
  if (tc_first_use_on_device(attr_done)) {
    cudaFuncSetAttribute(stem_pool_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT);
    cudaFuncSetAttribute(stem_pool_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_LIMIT);
  }
  Runtime &r = rt();
  pl.p.descending = r.descending;
  r.descending ^= 1;
  int prof_slot = -1;
  if (r.profiling) {   // timed like the other tensor-core launches
    prof_slot = r.prof_count++;
    while ((int)r.prof_events.size() < 2 * (prof_slot + 1)) {
      cudaEvent_t e;
      OCC_CUDA(cudaEventCreate(&e));
      r.prof_events.push_back(e);
    }
    OCC_CUDA(cudaEventRecord(r.prof_events[2 * prof_slot], s));
  }
  tc_launch_pdl(kernel, pl.grid, ST_THREADS, (size_t)pl.l.smem, s, pl.p);
  if (prof_slot >= 0) OCC_CUDA(cudaEventRecord(r.prof_events[2 * prof_slot + 1], s));
  count(CNT_LAUNCHES);
  count(CNT_TC_LAUNCHES);
  return cudaGetLastError() == cudaSuccess;
}

}  // namespace occ
