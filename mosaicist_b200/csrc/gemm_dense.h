// What the two dense GEMM translation units share.
#pragma once

#include "gemm_common.cuh"

namespace msc {

// Tile form of the one-tile-per-cluster kernel (gemm_dense_split.cu): tiles of 128 rows by tile_n
// columns, the K stages dealt out to the `splits` CTAs of a cluster.  splits == 0: the persistent
// kernel of gemm_dense_f16.cu.
struct DenseForm {
  int tile_n;
  int splits;
};

DenseForm pick_dense_form(int m, int n, int k, int lda, int ldb);

int launch_dense_split(const DenseForm& form, const void* a, const void* b, void* c, int m, int n, int k, int lda,
                       int ldb, int ldc, int is_bf16, int* status, cudaStream_t stream);

}  // namespace msc
