// The order in which the 32-bit products sum, and the entry of their aligned kernels (gemm_f32.cu).
#pragma once

#include <cuda_runtime.h>

constexpr int F32_CHUNK = 128;  // k's of a run: its even and its odd k's are added one after the other, then the two sums
constexpr int F32_PARTS = 8;    // parts of K, each of as many runs (two at least); a cluster's CTAs can take a part each
__host__ __device__ inline int f32_runs_per_part(int runs) {
    const int per = (runs + F32_PARTS - 1) / F32_PARTS;
    return per < 2 ? 2 : per;
}

bool ferris_gemm_f32_takes(const void* x, const void* w, const void* out, int K, int ldx, int ldw);
// `taken` false: nothing was launched (sizes that no form takes).
// early_weights: no launch that may still run writes w.
int ferris_gemm_f32(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldx, int ldw,
                    int ldo, int accumulate, int early_weights, cudaStream_t s, bool* taken);

// Products of many tokens on the tensor cores, operands and sums of 32 bits (gemm_f32_split.cu): which it takes (rows as
// ferris_gemm_f32_takes has them; `rows`: weight rows), and the product (up_offset > 0: SwiGLU of N gate rows and the N rows up_offset
// further).
bool ferris_gemm_f32_split_takes(int M, int rows, int K, int ldx, int ldw);
int ferris_gemm_f32_split(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int ldx, int ldw,
                          int ldo, int accumulate, int up_offset, int early_weights, cudaStream_t s);
