// Shared between the two bf16 GEMM kernels: epilogue flags and the launchers of the two-CTA and the cluster split-K kernels.
#pragma once
#include <cuda_runtime.h>

namespace tb {

enum : int {
  EPI_BIAS = 1,          // += bias[n] (bf16)
  EPI_GELU = 2,          // tanh-GELU after bias
  EPI_RESIDUAL = 4,      // += residual[m,n] (bf16) after activation
  EPI_OUT_F32 = 8,       // D is fp32 (default bf16)
  EPI_ATOMIC = 16,       // fp32 atomic accumulate into D (split-K / grad accumulation)
  EPI_STORE_PREACT = 32, // also store the pre-activation (after bias) as bf16
  EPI_MUL_DGELU = 64,    // *= gelu'(aux[m,n]) (aux = forward pre-activation, bf16)
  EPI_ACCUM = 128,       // D = D + result (non-atomic read-modify-write)
  EPI_RASTER_M = 256,    // walk tiles with m fastest (B panel shared by concurrent CTAs)
};

struct GemmArgs {
  const void *A, *B;
  void* D;
  int M, N, K, a_major, b_major, lda, ldb, ldd;
  const void *bias, *residual;
  int ldr;
  void* preact;
  const void* aux;
  int flags, split_k;
  int* status;
  // sums of A over K (a_major = 1: the columns of the stored [K, M] matrix), CTA-pair kernel only: null, or M values that the
  // launch adds to (fp32) or, with colsum_store, writes in bf16 (split_k 1)
  void* colsum = nullptr;
  int colsum_store = 0;
};

// True when the kernel can run this product (alignment, epilogue).
bool gemm_pair_ok(const GemmArgs& a);
bool gemm_split_ok(const GemmArgs& a);
// CTA pairs on 256 x 256 tiles (gemm_pair_sm100.cu); split_k > 1 needs EPI_ATOMIC.
int gemm_pair_launch(const GemmArgs& a, cudaStream_t stream);
// 128 x bn tiles (bn 64 or 128), K split over a cluster of S = 1, 2, 4 or 8 CTAs (gemm_split_sm100.cu); bf16 output.
int gemm_split_launch(const GemmArgs& a, int bn, int S, cudaStream_t stream);

}  // namespace tb
