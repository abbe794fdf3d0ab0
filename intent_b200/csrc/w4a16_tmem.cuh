// Internal entry of the W4A16 kernel that keeps the expanded weights in tensor memory (w4a16_tmem.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ib200 {

struct TmemCall {
  const void* x;               // [rows, K]
  int64_t rows, K;
  const void* w;               // [experts, K / 8, WN]
  const void* s;               // [experts, K / group_size, WN]
  int64_t experts, WN;
  void* out;
  int64_t out_cols;
  int group_size, zero_point;
  int row_tile;                // rows of a tile, a multiple of 16 up to 128 (with pairs of 32 up to 256; grouped: 128)
  int split;                   // dense: CTAs of a cluster that share the k blocks of a tile
  const int* total_rows;       // grouped modes, as in w4a16_gemm.cu
  const int* tile_expert;
  int block_rows;
  const int* row_route;        // route of every row, or null when all rows of a block count
  const float* route_weight;
  int64_t routes;
  int top_k;
  float* clear;                // up|gate: a buffer that the call fills with zeros beside its work, or null
  int64_t clear_vectors;       // its size in 16 bytes
};

// mode: the MODE_* numbers of w4a16_gemm.cu
template <typename T>
int w4a16_tmem(const TmemCall& call, int mode, bool pairs, cudaStream_t stream);
int w4a16_tmem_take_status(int* value);

}  // namespace ib200
