// Parameter block of the split-reduction convolution kernel (conv_tc_split.cu) and its launcher.
#pragma once
#include "conv_tc_dev.cuh"

namespace occ {

constexpr int SK_THREADS = 256;
constexpr int SK_MAX_SPLITS = 8;       // portable cluster size
constexpr int SK_MAX_STAGES = 16;
constexpr int SK_MAX_AMAPS = 12;       // A tensor maps: 4 stride phases of 3 operand parts, or of one and the second summand's

struct SkTap {
  int8_t map, dw, dh, pad;
};

struct alignas(64) SkParams {
  CUtensorMap tmA[SK_MAX_AMAPS];
  CUtensorMap tmB;
  CUtensorMap tmB2;                    // weights of the second summand
  SkTap taps[TC_MAX_TAPS];
  int cblocks, bk, stages, ksteps;     // ksteps = taps * cblocks, and the second summand's
  int ksteps1, map2;                   // k-steps before the second summand's (TcConvArgs::x2), its A map
  int issuers;                         // threads that issue MMAs: sk_issuers(), but no more than k-steps
  int splits;                          // CTAs (one cluster) that share a tile's reduction
  TcFastDiv div_k, div_w, div_h, div_cb;
  int tiles_k, tiles_w, tiles_h;
  int tw, th, tn;
  int rows;                            // pixels of a tile's box (<= 128)
  int rows_owner;                      // rows each CTA of the cluster sums up and stores
  int a_bytes;                         // bytes of an activation tile in a stage (multiple of 1024)
  int K, gq, gp, gn;
  const float *bias, *bias2;           // bias2 is added to bias (either may be null)
  const void *residual;                // in the form of y, or null
  void *y;                             // 16-bit NHWC output (when out_f32 is null); with split operands
                                       // three planes (hi, mid, lo) of `plane` elements each
  int64_t plane;
  float *out_f32;
  int ldo, out_hw;                     // as in TcParams
  int out_vec4;                        // row-major fp32 output whose rows are 16-byte aligned
  float floor, lo, hi;                 // tc_act()
  int consts_ready;
  int *err;
};

// Threads that issue MMAs (and that load) in a kernel: as many accumulators as fit the 256 TMEM
// columns a CTA may use, four at most; one for split operands, whose k-step has 12 or 24 MMAs.  A ring
// with fewer stages than the CTA has k-steps must have a multiple of this many.
__host__ __device__ constexpr int sk_issuers(int bn, bool split) {
  return split ? 1 : 256 / bn < 4 ? 256 / bn : 4;
}
// Operand tiles of either side in a stage: fp32 values travel as three bf16 parts (hi, mid, lo).
__host__ __device__ constexpr int sk_parts(bool split) { return split ? 3 : 1; }
// Shared memory a launch needs.
size_t sk_smem_bytes(int bn, int stages, int a_bytes, int bk, int splits, int rows_owner, bool split);
// `split` selects the kernels whose operands are bf16 parts of fp32 values.
bool sk_launch(const SkParams &p, int bn, bool f16, bool split, int tiles, size_t smem, cudaStream_t s);

}  // namespace occ
