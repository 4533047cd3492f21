// One launch of the few-rows matmul kernel (gemm_decode_sm100.cu).
#pragma once
#include <algorithm>

#include "gemm_sm100.cuh"

namespace gcb {

struct DecodeParams {
  int kpb;        // K blocks of a stage
  int tiles;      // 128 output columns each
  int split;      // CTAs (a cluster) that share a tile's K range, every one with at least one K block
  uint32_t parts_bytes;   // shared memory for a CTA's partial sums: rows x 512 when split > 1
  int k_blocks;   // K blocks (128 bytes of K) of one tile
  int BN;         // rows of X, rounded up to a multiple of 16
  int stages, bk_elems;
  int early_weights;   // nothing in flight on the device writes the weights
  OperandGeom w, x;
  uint32_t idesc, tmem_cols;
  int out_kind, bias_kind, relu, out_rows, out_cols;
  void *out;
  long long ld_out, ld_dump;
  const void *bias;
  const float *scale;
  const int32_t *comp;
  int32_t *acc_dump;
  int *error;
};

int decode_stages(const DecodeParams &p);
int decode_clusters_at_once(bool int8, int device, int split);   // 0: that size does not run
template <int KIND>
cudaError_t launch_gemm_decode(const CUtensorMap &tmW, const CUtensorMap &tmX, const DecodeParams &p, int grid, int device, cudaStream_t stream);

} // namespace gcb
