// Parameter block of the two-layer kernel (conv_pair.cu) and its launcher.
#pragma once
#include "conv_tc_dev.cuh"

namespace occ {

constexpr int PR_MISC_BYTES = 512;

struct alignas(64) PairParams {
  CUtensorMap tmA[2];      // x, the second summand's (TcConvArgs::x2)
  CUtensorMap tmB1[2];     // their weights
  CUtensorMap tmB2;        // the second layer's
  CUtensorMap tmY, tmR;    // y; its shortcut tensor
  CUtensorMap tmT;
  int blocks1, blocks2;    // 64-channel blocks of x and of the second summand
  int K1, K2;              // channels of y (a multiple of 128) and of t (64 or 128)
  int tw, th, tn, rows;    // pixels of a tile's box
  int tiles_w, tiles_h, total_tiles;
  TcFastDiv div_w, div_h;
  int a_blocks, w1_tiles, w2_tiles, slabs;   // shared memory, in blocks of 16 KB
  const float *bias1, *bias1b, *bias2;
  int has_res, consts_ready, descending;
  int *err;
};

bool pair_layout(PairParams &p, size_t *smem);
void pair_launch(const PairParams &p, bool f16, int grid, size_t smem, cudaStream_t s);

}  // namespace occ
