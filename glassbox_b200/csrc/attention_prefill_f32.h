// The float32 prompt attention on the tensor cores (attention_prefill_f32_mma.cu), as the entry point in attention_prefill_f32.cu
// launches it.
#pragma once
#include <cuda_runtime.h>

template <int HD>
int gb_launch_prefill_f32_mma(const float* q, long long q_stride, float* out, long long out_stride, const float* kcache, const float* vcache,
                              const int* block_tables, int max_pages, const int* seq_first_row, const int* seq_start_pos, int rows, int num_seqs,
                              int max_rows_per_seq, int nh, int nkv, int page_size, long long num_pages, float scale, int window,
                              int* status, cudaStream_t stream);
