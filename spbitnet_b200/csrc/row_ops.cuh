// Register-resident vector ops of a batch of rows (row_ops.cu); reached through the launchers of fused_ops.cuh.
#pragma once
#include "spb_common.cuh"

namespace spb {

// rows of n elements (a multiple of 8, at most 32768), every operand on a 16-byte boundary (absent ones null)
bool row_ops_take(int n, const void* a, const void* b, const void* c, const void* d, const void* e, const void* q);
int rows_residual_norm_quant(const __half* delta, const float* sub_w, __half* x, const float* w, __half* xn_out, int8_t* xq,
                             float* d_absmax, int n, float eps, void* stream, int vectors);
int rows_relu2_norm_quant(const __half* gate, const __half* up, const float* sub_w, __half* h_out, int8_t* hq, float* d_absmax,
                          int n, float eps, void* stream, int vectors);
int rows_absmax_quantize(const __half* in, int8_t* out, float* d_absmax, int n, void* stream, int vectors);
// whole 16-byte pieces: head_dim and the sequences' stride multiples of 8, operands on 16-byte boundaries
bool rows_rope_scatter_takes(const void* q, const void* k, const void* v, const void* kcache, const void* vcache, int head_dim,
                             size_t seq_stride);
int rows_rope_scatter(__half* q, const __half* k, const __half* v, __half* kcache, __half* vcache, int num_heads,
                      int num_kv_heads, int head_dim, int max_seq_len, float theta, const int* d_pos, void* stream, int vectors,
                      size_t seq_stride);

}  // namespace spb
