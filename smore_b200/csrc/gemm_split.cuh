// fp32-accurate products on the bf16 tensor cores (gemm_split_sm100.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace smore {

// bytes of the three bf16 planes of [rows, k]
size_t split_plane_bytes(size_t rows, size_t k);
// fp32 [rows, cols] (cols and rows multiples of 4, ld_x floats from row to row, a multiple of 4 too) -> planes of it
// and / or of its transpose; either may be nullptr
int split_planes(const float* x, size_t ld_x, size_t rows, size_t cols, void* plain, void* transposed, cudaStream_t st);
// D[M, N] = A . B^T (add: D += ...) from planes of A [M, K] and B [N, K]; N and ld_d multiples of 4; scratch:
// split_gemm_scratch_bytes(M, N, K) bytes, 16-byte aligned
size_t split_gemm_scratch_bytes(size_t M, size_t N, size_t K);
int split_gemm(const void* a_planes, const void* b_planes, float* d, size_t ld_d, bool add, size_t M, size_t N, size_t K,
               void* scratch, cudaStream_t st);

}  // namespace smore
