// The 32-bit path's attention of prompts on tensor cores (attention_f32_split.cu): heads of 64, plain scores, an optional window.
#pragma once

#include <cuda_runtime.h>

bool ferris_attention_f32_split_takes(int nh, int nkv, int d, int dv);
int ferris_attention_f32_split(const float* q, int ldq, float* out, int ldo, const float* k_cache, const float* v_cache,
                               const int* block_tables, int max_blocks, const int* token_seq, const int* positions, int tokens, int nh,
                               int nkv, int page_size, int window, float scale, int seqs, cudaStream_t s);
