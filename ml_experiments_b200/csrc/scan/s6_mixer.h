// The small passes around the S6 scan (torch-free interface). C channels, 16 states, a depthwise convolution of width 4.
#pragma once
#include <cuda_runtime.h>

namespace b200 {
// conv weight [C][4], conv bias [C], A_log [C][16], D [C], step bias [C], each fp32 or bf16
struct S6Tensors {
  const void* ptr[5];
  bool bf16[5];
};
// packed: fp32 [23 C], the five after each other with A = -exp(A_log) for A_log
void s6_params(const S6Tensors& t, float* packed, int C, cudaStream_t s);
// grads: fp32 [23 C], laid out like packed, with the gradient of A; writes the five gradients in their types
void s6_param_grads(const S6Tensors& t, const float* grads, const float* packed, int C, cudaStream_t s);
// dbc: bf16 [rows][ld] (16-byte aligned, ld a multiple of 8) with B and C in its last 32 columns; bc: fp32 [2][rows][16]
void s6_split_bc(const void* dbc, float* bc, long long rows, int ld, cudaStream_t s);
// parts: fp32 [2][batch][blocks][L][16] as the scan's backward writes dB and dC; ddbc: bf16 [batch * L][ld], its last 32 columns
void s6_join_bc(const float* parts, void* ddbc, int batch, int blocks, int L, int ld, cudaStream_t s);
}  // namespace b200
