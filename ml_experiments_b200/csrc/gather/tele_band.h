// Telephone attention (the operator of fused_taps.h, same arguments) as products with band matrices on the tensor cores.
#pragma once
#include <cuda_runtime.h>

namespace b200 {
// Whether the kernels below take a call; x and y (output or its gradient) are the tensors that TMA and 16-byte accesses touch.
bool tele_band_takes(const void* x, const void* y, int B, int L, int H, int D, int K, int half, float max_rec, bool backward);
void tele_band_fwd(const void* x, const float* freq, const float* phase, const float* kern, const float* expo, void* out, int B, int L, int H,
                   int D, int K, int half, float max_rec, int* status, cudaStream_t s);
// dx: bf16 or fp32, written whole. queries: 3072 bytes (16-byte aligned) and ranges: 8 bytes for each of B * H * ceil(L / 64) query tiles.
void tele_band_bwd(const void* x, const float* freq, const float* phase, const float* kern, const float* expo, const void* dout, void* dx,
                   bool dx_f32, float* dfreq, float* dphase, float* dkern, float* dexpo_h, void* ranges, void* queries, int B, int L, int H, int D,
                   int K, int half, float max_rec, int* status, cudaStream_t s);
}  // namespace b200
