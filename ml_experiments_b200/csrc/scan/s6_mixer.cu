// See s6_mixer.h. What surrounds the scan of an S6 mixer: parameters in the types that the convolution and the scan read, B and C out
// of the projection's rows, and the way back. One launch each where a cast, a copy or a reduction per tensor is five to nine; at
// 3 x 1531 tokens and 1024 channels each of those took 2 us and its launch 5.
#include "s6_mixer.h"

#include <cuda_bf16.h>

#include <cstdint>
#include <stdexcept>
#include <string>

#include "../common/ptx.cuh"

namespace b200 {
namespace {
using bf16 = __nv_bfloat16;
constexpr int NS = 16;

__device__ __forceinline__ float get(const void* p, bool b, long long i) {
  return b ? __bfloat162float(reinterpret_cast<const bf16*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}
__device__ __forceinline__ void put(void* p, bool b, long long i, float v) {
  if (b) reinterpret_cast<bf16*>(p)[i] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(p)[i] = v;
}

// Element i of the packed buffer: [C][4] taps, [C] conv bias, [C][16] A, [C] D, [C] step bias.
struct Part {
  int which;
  long long at;
};
__device__ __forceinline__ Part part_of(long long i, int C) {
  if (i < 4ll * C) return {0, i};
  if (i < 5ll * C) return {1, i - 4ll * C};
  if (i < 21ll * C) return {2, i - 5ll * C};
  if (i < 22ll * C) return {3, i - 21ll * C};
  return {4, i - 22ll * C};
}

__global__ void s6_params_kernel(S6Tensors t, float* __restrict__ packed, int C) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 23ll * C) return;
  const Part p = part_of(i, C);
  const float v = get(t.ptr[p.which], t.bf16[p.which], p.at);
  packed[i] = p.which == 2 ? (float)-exp((double)v) : v;      // A = -exp(A_log), rounded once
}

__global__ void s6_param_grads_kernel(S6Tensors t, const float* __restrict__ grads, const float* __restrict__ packed, int C) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 23ll * C) return;
  const Part p = part_of(i, C);
  put(const_cast<void*>(t.ptr[p.which]), t.bf16[p.which], p.at, p.which == 2 ? grads[i] * packed[i] : grads[i]);   // dA / dA_log = A
}

// A thread takes eight columns of a row of dbc: [rows][ld], B and C in the last 32 columns.
__global__ void s6_split_bc_kernel(const bf16* __restrict__ dbc, float* __restrict__ bc, long long rows, int ld) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, row = i >> 2;
  if (row >= rows) return;
  const int part = i & 3;
  const uint4 u = *reinterpret_cast<const uint4*>(dbc + row * ld + ld - 32 + part * 8);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  float4* dst = reinterpret_cast<float4*>(bc + (part >> 1) * rows * NS + row * NS + (part & 1) * 8);
  dst[0] = make_float4(a.x, a.y, b.x, b.y);
  dst[1] = make_float4(c.x, c.y, d.x, d.y);
}

// dbc's last 32 columns from the scan's partial sums, [2][batch][blocks][L][16]. A thread adds four columns over all blocks; several loads
// are under way at a time. Bound: the read of the partial sums, 268 MB at 8 x 4096 x 64 blocks.
__global__ void s6_join_bc_kernel(const float* __restrict__ parts, bf16* __restrict__ ddbc, int batch, int blocks, int L, int ld) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x, row = i >> 3;
  if (row >= (long long)batch * L) return;
  const int part = i & 7, b = (int)(row / L), l = (int)(row % L);
  const long long plane = (long long)L * NS, one = (long long)batch * blocks * plane;
  const float4* src = reinterpret_cast<const float4*>(parts + (part >> 2) * one + (long long)b * blocks * plane + (long long)l * NS + (part & 3) * 4);
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int k = 0; k < blocks; ++k) {
    const float4 v = src[k * (plane / 4)];
    s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
  }
  *reinterpret_cast<uint2*>(ddbc + row * ld + ld - 32 + part * 4) = make_uint2(pack_bf16x2(s.x, s.y), pack_bf16x2(s.z, s.w));
}

unsigned blocks_of(long long n) { return (unsigned)((n + 255) / 256); }
void check(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}
}  // namespace

void s6_params(const S6Tensors& t, float* packed, int C, cudaStream_t s) {
  s6_params_kernel<<<blocks_of(23ll * C), 256, 0, s>>>(t, packed, C);
  check("s6_params");
}
void s6_param_grads(const S6Tensors& t, const float* grads, const float* packed, int C, cudaStream_t s) {
  s6_param_grads_kernel<<<blocks_of(23ll * C), 256, 0, s>>>(t, grads, packed, C);
  check("s6_param_grads");
}
void s6_split_bc(const void* dbc, float* bc, long long rows, int ld, cudaStream_t s) {
  s6_split_bc_kernel<<<blocks_of(rows * 4), 256, 0, s>>>((const bf16*)dbc, bc, rows, ld);
  check("s6_split_bc");
}
void s6_join_bc(const float* parts, void* ddbc, int batch, int blocks, int L, int ld, cudaStream_t s) {
  s6_join_bc_kernel<<<blocks_of((long long)batch * L * 8), 256, 0, s>>>(parts, (bf16*)ddbc, batch, blocks, L, ld);
  check("s6_join_bc");
}

}  // namespace b200
