// S6 (Mamba-1) selective scan, forward and backward.
//
//   dt_t[d]  = softplus(delta_t[d] + delta_bias[d])            (both optional: plain delta when softplus is off)
//   h_t[d,n] = exp(dt_t[d] * A[d,n]) * h_{t-1}[d,n] + dt_t[d] * B_t[n] * u_t[d]
//   y_t[d]   = sum_n C_t[n] * h_t[d,n] + D[d] * u_t[d] ;   out = y * silu(z)
//
// Time is processed in tiles of 16 steps. The forward stores the state at the start of every tile; the backward walks
// the tiles in reverse, recomputes the states of a tile from that checkpoint and runs the adjoint recurrence. The gate
// (silu(z)), the softplus of delta and its bias are applied inside the kernels, so no elementwise pass is left outside.
// dB / dC leave as partial sums per 32-channel block [B][ceil(Din/32)][L][N] that the caller adds up, the same on every run.
//
// Two forms, with the same checkpoints. Channels in multiples of 8 and 16-byte aligned tensors take the pipelined kernels
// (further down): all states of a channel in one warp, inputs copied tiles ahead. Other rows take the general kernels, which
// come first: a block owns 32 channels, lane = channel, warp = QS of the 16 states in registers (four warps at QS = 4, eight
// at 2). There B_t / C_t are warp-uniform shared-memory broadcasts, the partial sums over states meet in shared memory, and the
// backward's dB_t / dC_t, sums over channels, are reduced across the 32 lanes by a halving butterfly (9 shuffles for 8 values).
//
// Semantics follow selective_scan_ref of the reference (zoology/mixers/mamba_ssm/ops/selective_scan_interface.py:91-157)
// with real A and input-dependent B and C shared across channels.
#include "s6_scan.h"

#include "../common/per_device.h"
#include "../common/ptx.cuh"

#include <cuda_bf16.h>

#include <cstdint>
#include <initializer_list>

#include <stdexcept>
#include <string>

namespace b200 {
namespace {

using bf16 = __nv_bfloat16;
constexpr int NS = 16;    // states per channel
constexpr int CB = 32;    // channels per block (= lanes)
constexpr int SUB = 16;   // time steps per tile and per state checkpoint
// States a thread: what a program has asked for; -1: by the size of the call. Measured on 8 x 4096 x 2048 in the general kernels:
// forward 0.72 ms at 2 (0.80 at 4); backward 2.6 ms at 4 (5.5 at 2: spills).
int g_fwd_qs = -1, g_bwd_qs = 4;

// State checkpoints are stored in groups of four states whatever QS the kernels run with:
// [B][tiles][4][Din][4]; a thread's QS states (from n0 on) are contiguous in it.
__device__ __forceinline__ long long state_off(int b, int nsub, int tile, int n0, int Din, int d) {
  return ((((long long)b * nsub + tile) * 4 + (n0 >> 2)) * Din + d) * 4 + (n0 & 3);
}

template <int QS>
struct Shape {
  static constexpr int NW = NS / QS;          // warps per block
  static constexpr int NT = 32 * NW;          // threads per block
  static constexpr int RPT = SUB / NW;        // rows of a [16][32] tile staged per thread
  static constexpr int BCPT = SUB * NS / NT;  // B (and C) elements staged per thread
};

// QS consecutive floats as one vector access
template <int QS>
__device__ __forceinline__ void ldv(float (&o)[QS], const float* p) {
  if constexpr (QS == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
  } else {
    const float2 v = *reinterpret_cast<const float2*>(p);
    o[0] = v.x, o[1] = v.y;
  }
}
template <int QS>
__device__ __forceinline__ void stv(float* p, const float (&o)[QS]) {
  if constexpr (QS == 4) *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  else *reinterpret_cast<float2*>(p) = make_float2(o[0], o[1]);
}
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Request a line into L1 (and L2) without holding a register for it.
__device__ __forceinline__ void prefetch_near(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }
__device__ __forceinline__ float ld(const float* p, long long i) { return p[i]; }
__device__ __forceinline__ float ld(const bf16* p, long long i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void st(float* p, long long i, float v) { p[i] = v; }
__device__ __forceinline__ void st(bf16* p, long long i, float v) { p[i] = __float2bfloat16_rn(v); }

// Softplus and sigmoid without a branch, so that those of several steps and channels are under way at once (a division and log1pf
// have branches). Both from t = exp(-|x|); quotients are the hardware's approximate reciprocal and one Newton step on the exact
// remainder, which also takes in the rounding of the denominator.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sigmoid_of(float x, float t) {
  const float r = rcp_approx(1.f + t), n = x < 0.f ? t : 1.f, y = n * r;          // n / (1 + t)
  return fmaf(fmaf(-y, t, n - y), r, y);
}
// softplus(x) = max(x, 0) + log(1 + t), and log(1 + t) = 2 atanh(s) = 2 (s + s^3 / 3 + s^5 / 5 + ...) with s = t / (2 + t) <= 1/3: what
// is left out of the series is 1.4e-9 of it. Root mean square error against 64 bits, |x| <= 5: 6.0e-8, of the sigmoid 5.7e-8 (log1pf of
// __expf and the division: 6.2e-8 both). Results below 2^-126 are 0. Backward, 8 x 4096 x 2048: 1.82 -> 1.76 ms.
__device__ __forceinline__ float softplus_of(float x, float t) {
  const float r = rcp_approx(2.f + t), s0 = t * r, s = fmaf(fmaf(-s0, t, fmaf(-2.f, s0, t)), r, s0), q = s * s;
  float p = fmaf(q, 1.f / 15, 1.f / 13);
  p = fmaf(q, p, 1.f / 11);
  p = fmaf(q, p, 1.f / 9);
  p = fmaf(q, p, 1.f / 7);
  p = fmaf(q, p, 1.f / 5);
  p = fmaf(q, p, 1.f / 3);
  return fmaxf(x, 0.f) + fmaf(-s, fmaf(-2.f * q, p, t), t);          // 2 s = t - s t
}
__device__ __forceinline__ float exp_minus_abs(float x) { return ex2(-LOG2E * fabsf(x)); }
__device__ __forceinline__ float sigmoidf(float x) { return sigmoid_of(x, exp_minus_abs(x)); }
__device__ __forceinline__ float softplusf(float x) { return softplus_of(x, exp_minus_abs(x)); }
__device__ __forceinline__ float softplusf(float x, float& derivative) {
  const float t = exp_minus_abs(x);
  derivative = sigmoid_of(x, t);
  return softplus_of(x, t);
}

template <int QS>
struct FwdSmem {
  float dt[SUB][CB];
  float u[SUB][CB];
  float B[SUB][NS];
  float C[SUB][NS];
  float yp[NS / QS][SUB][CB];
};

// grid (ceil(Din / 32), batch), 32 * 16 / QS threads. DT = element type of delta (fp32 or bf16).
template <typename DT, int QS>
__global__ void __launch_bounds__(Shape<QS>::NT, 1024 / Shape<QS>::NT)
s6_fwd_kernel(const bf16* __restrict__ u, const DT* __restrict__ delta, const float* __restrict__ delta_bias,
              int softplus, const float* __restrict__ A, const float* __restrict__ Bm, const float* __restrict__ Cm,
              const float* __restrict__ Dv, const bf16* __restrict__ z, bf16* __restrict__ y_pre,
              bf16* __restrict__ out, float* __restrict__ state, int L, int Din) {
  constexpr int NW = Shape<QS>::NW, NT = Shape<QS>::NT, RPT = Shape<QS>::RPT, BCPT = Shape<QS>::BCPT;
  __shared__ __align__(16) FwdSmem<QS> s;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int b = blockIdx.y, d0 = blockIdx.x * CB, d = d0 + lane;
  const bool dok = d < Din;
  const int nsub = (L + SUB - 1) / SUB;
  float h[QS], a2[QS];
#pragma unroll
  for (int k = 0; k < QS; ++k) {
    h[k] = 0.f;
    a2[k] = dok ? A[(long long)d * NS + w * QS + k] * LOG2E : 0.f;
  }
  const float bias = (dok && delta_bias) ? delta_bias[d] : 0.f;
  const float dsk = (dok && Dv) ? Dv[d] : 0.f;
  // staging registers for the next tile: the thread covers rows w + NW * j of the [16][32] tiles and BCPT B / C elements
  float pdt[RPT], pu[RPT], pz[RPT], pB[BCPT], pC[BCPT];
  auto fetch = [&](int tile) {
    const int t0 = tile * SUB;
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int t = t0 + w + NW * j;
      const bool ok = dok && t < L;
      const long long off = ((long long)b * L + t) * Din + d;
      pdt[j] = ok ? ld(delta, off) : 0.f;
      pu[j] = ok ? __bfloat162float(u[off]) : 0.f;
      pz[j] = (ok && z) ? __bfloat162float(z[off]) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < BCPT; ++j) {
      const int i = tid + NT * j, t = t0 + i / NS;
      const long long off = ((long long)b * L + t) * NS + (i % NS);
      pB[j] = t < L ? Bm[off] : 0.f;
      pC[j] = t < L ? Cm[off] : 0.f;
    }
  };
  fetch(0);
  for (int tile = 0; tile < nsub; ++tile) {
    const int t0 = tile * SUB;
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int t = w + NW * j;
      float dtv = pdt[j];
      if (softplus) dtv = (dok && t0 + t < L) ? softplusf(dtv + bias) : 0.f;
      s.dt[t][lane] = dtv;
      s.u[t][lane] = pu[j];
    }
#pragma unroll
    for (int j = 0; j < BCPT; ++j) {
      const int i = tid + NT * j;
      s.B[i / NS][i % NS] = pB[j];
      s.C[i / NS][i % NS] = pC[j];
    }
    float zc[RPT];  // this tile's gate inputs (the staging registers are about to be refilled)
#pragma unroll
    for (int j = 0; j < RPT; ++j) zc[j] = pz[j];
    __syncthreads();
    if (tile + 1 < nsub) fetch(tile + 1);
    if (state && dok)
      stv<QS>(&state[state_off(b, nsub, tile, w * QS, Din, d)], h);
#pragma unroll
    for (int t = 0; t < SUB; ++t) {
      const float dt = s.dt[t][lane], dtu = dt * s.u[t][lane];
      float bb[QS], cc[QS];
      ldv<QS>(bb, &s.B[t][w * QS]);
      ldv<QS>(cc, &s.C[t][w * QS]);
      float y = 0.f;
#pragma unroll
      for (int k = 0; k < QS; ++k) {
        h[k] = fmaf(ex2(dt * a2[k]), h[k], dtu * bb[k]);
        y = fmaf(h[k], cc[k], y);
      }
      s.yp[w][t][lane] = y;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int t = w + NW * j;
      if (dok && t0 + t < L) {
        const long long off = ((long long)b * L + t0 + t) * Din + d;
        float yv = dsk * s.u[t][lane];
#pragma unroll
        for (int q = 0; q < NW; ++q) yv += s.yp[q][t][lane];
        if (y_pre) y_pre[off] = __float2bfloat16_rn(yv);
        float o = yv;
        if (z) o = yv * zc[j] * sigmoidf(zc[j]);
        out[off] = __float2bfloat16_rn(o);
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------------
// Pipelined kernels: rows of 16-byte aligned 8-channel pieces (Din % 8 == 0, aligned pointers)
// ------------------------------------------------------------------------------------------------
// A warp owns CW = 32 / G channels with all their 16 states: lane = (group g of QS states, channel). What is summed over
// the states then stays inside the warp, and G time steps are reduced together by a halving exchange that leaves lane
// group g with step g: every lane ends up with the elementwise work (softplus, gate, skip, stores) of its own steps, so
// none of it is done twice. A block is 16 channels; tiles of 16 steps are copied by cp.async two tiles ahead.
//
// Bound: one exponential per state and step (SFU: 8 cycles per warp instruction), 0.24 ms of 8 x 4096 x 2048 x 16; the
// softplus and the gate add a quarter to it. Shared memory takes 3 vector loads and 3/4 of a shuffle per warp step.
// Measured, with the states stored: 0.611 ms there (0.661 ms with log1pf, divisions and a loop over the pieces to copy), 1 x 4096 x
// 2048: 0.223 ms (0.252 ms). The general kernel (a warp per two states of 32 channels, partial sums in shared memory) takes 0.17 ms
// for 3 x 1531 x 1024, this one 0.112.
constexpr int PC = 16;   // channels per block of the forward

template <typename DT>
struct FwdRaw {
  DT delta[SUB][PC];
  bf16 u[SUB][PC];
  bf16 z[SUB][PC];
  float B[SUB][NS];
  float C[SUB][NS];
};

// 16 bytes global -> shared; `bytes` (0..16) of them are read, the rest of the destination is zero-filled
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Sums y[i] of step i over the G lane groups (lanes CW apart); group g is left with the total of step g.
template <int G, int CW>
__device__ __forceinline__ float steps_to_groups(float (&y)[G], int g) {
#pragma unroll
  for (int m = G / 2; m >= 1; m /= 2) {
    const bool up = g & m;
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const float send = up ? y[i] : y[i + m], keep = up ? y[i + m] : y[i];
      y[i] = keep + __shfl_xor_sync(0xffffffffu, send, m * CW);
    }
  }
  return y[0];
}

// QS consecutive floats of shared memory as packed pairs
template <int QS>
__device__ __forceinline__ void ld2(uint64_t (&o)[QS / 2], const float* p) {
  if constexpr (QS == 4) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    o[0] = v.x, o[1] = v.y;
  } else {
    o[0] = *reinterpret_cast<const uint64_t*>(p);
  }
}
__device__ __forceinline__ uint64_t f2_ex2(uint64_t v) {
  float x, y;
  f2_unpack(v, x, y);
  return f2_pack(ex2(x), ex2(y));
}

// grid (ceil(Din / 16), batch), 256 / QS threads.
template <typename DT, int QS>
__global__ void __launch_bounds__(256 / QS, QS == 4 ? 8 : 4)
s6_fwd_pipe_kernel(const bf16* __restrict__ u, const DT* __restrict__ delta, const float* __restrict__ delta_bias,
                   int softplus, const float* __restrict__ A, const float* __restrict__ Bm, const float* __restrict__ Cm,
                   const float* __restrict__ Dv, const bf16* __restrict__ z, bf16* __restrict__ y_pre,
                   bf16* __restrict__ out, float* __restrict__ state, int L, int Din) {
  constexpr int G = NS / QS, CW = 32 / G, NT = 256 / QS, KS = SUB / G, STAGES = 3;
  __shared__ __align__(16) FwdRaw<DT> raw[STAGES];
  __shared__ __align__(16) float2 step[SUB][PC];    // {dt, dt * u}
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane / CW, c = warp * CW + (lane & (CW - 1));
  const int b = blockIdx.y, d0 = blockIdx.x * PC, d = d0 + c;
  const bool dok = d < Din;
  const int nsub = (L + SUB - 1) / SUB;
  uint64_t h[QS / 2], a2[QS / 2];
#pragma unroll
  for (int p = 0; p < QS / 2; ++p) {
    const long long o = (long long)d * NS + g * QS + 2 * p;
    h[p] = 0;
    a2[p] = dok ? f2_pack(A[o] * LOG2E, A[o + 1] * LOG2E) : 0;
  }
  const float bias = (dok && delta_bias) ? delta_bias[d] : 0.f;
  const float dsk = (dok && Dv) ? Dv[d] : 0.f;

  // a thread copies one 16-byte piece of each pair of 32-byte rows and of B and C; where there are 128, half of that
  const int row = (tid & 63) >> 2, piece = tid & 3, ch = (piece & 1) * 8;
  const bool first = NT == 64 || tid < 64, second = NT == 64 || tid >= 64;
  auto issue = [&](int tile) {
    if (tile < nsub) {
      FwdRaw<DT>& r = raw[tile % STAGES];
      const bool rok = tile * SUB + row < L;
      const long long bt = (long long)b * L + min(tile * SUB + row, L - 1), off = bt * Din + min(d0 + ch, Din - 8);
      const int n16 = (rok && d0 + ch < Din) ? 16 : 0;
      if (first) {
        if (sizeof(DT) == 4) cp_async16(&r.delta[row][piece * 4], delta + bt * Din + min(d0 + piece * 4, Din - 4), (rok && d0 + piece * 4 < Din) ? 16 : 0);
        else if (piece < 2) cp_async16(&r.delta[row][ch], delta + off, n16);
        cp_async16(&r.B[row][piece * 4], Bm + bt * NS + piece * 4, rok ? 16 : 0);
      }
      if (second) {
        if (piece < 2) cp_async16(&r.u[row][ch], u + off, n16);
        else if (z) cp_async16(&r.z[row][ch], z + off, n16);
        cp_async16(&r.C[row][piece * 4], Cm + bt * NS + piece * 4, rok ? 16 : 0);
      }
    }
    cp_async_commit();       // also when empty: the groups are counted
  };
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) issue(i);
  for (int tile = 0; tile < nsub; ++tile) {
    const int t0 = tile * SUB;
    cp_async_wait<STAGES - 2>();
    __syncthreads();         // the tile is visible to all, and nobody works on the one before it any more
    issue(tile + STAGES - 1);
    const FwdRaw<DT>& r = raw[tile % STAGES];
    float uu[KS], zz[KS], dt[KS];
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      const int t = k * G + g;
      dt[k] = (float)r.delta[t][c];
      uu[k] = __bfloat162float(r.u[t][c]);
      zz[k] = z ? __bfloat162float(r.z[t][c]) : 0.f;
      if (softplus) dt[k] = softplusf(dt[k] + bias);
      if (t0 + t >= L) dt[k] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < KS; ++k) step[k * G + g][c] = make_float2(dt[k], dt[k] * uu[k]);
    __syncwarp();
    if (state && dok) {
      float o[QS];
#pragma unroll
      for (int p = 0; p < QS / 2; ++p) f2_unpack(h[p], o[2 * p], o[2 * p + 1]);
      stv<QS>(&state[state_off(b, nsub, tile, g * QS, Din, d)], o);
    }
#pragma unroll
    for (int k = 0; k < KS; ++k) {
      float y[G];
#pragma unroll
      for (int i = 0; i < G; ++i) {
        const float2 e = step[k * G + i][c];
        const uint64_t dt = f2_pack(e.x, e.x), dtu = f2_pack(e.y, e.y);
        uint64_t bb[QS / 2], cc[QS / 2], yy = 0;
        ld2<QS>(bb, &r.B[k * G + i][g * QS]);
        ld2<QS>(cc, &r.C[k * G + i][g * QS]);
#pragma unroll
        for (int p = 0; p < QS / 2; ++p) {
          h[p] = f2_fma(f2_ex2(f2_mul(dt, a2[p])), h[p], f2_mul(dtu, bb[p]));
          yy = p == 0 ? f2_mul(h[p], cc[p]) : f2_fma(h[p], cc[p], yy);
        }
        float y0, y1;
        f2_unpack(yy, y0, y1);
        y[i] = y0 + y1;
      }
      const float yv = fmaf(dsk, uu[k], steps_to_groups<G, CW>(y, g));
      const int t = t0 + k * G + g;
      if (dok && t < L) {
        const long long off = ((long long)b * L + t) * Din + d;
        if (y_pre) y_pre[off] = __float2bfloat16_rn(yv);
        out[off] = __float2bfloat16_rn(z ? yv * zz[k] * sigmoidf(zz[k]) : yv);
      }
    }
  }
}

template <int QS>
struct BwdSmem {
  float dt[SUB][CB];
  float u[SUB][CB];
  float dy[SUB][CB];
  float B[SUB][NS];
  float C[SUB][NS];
  float dB[SUB][NS];
  float dC[SUB][NS];
  float pddt[NS / QS][SUB][CB];
  float pdu[NS / QS][SUB][CB];
};

// Sum each of 8 per-lane values over the 32 lanes; afterwards every lane holds the total of value
// ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1).
__device__ __forceinline__ float reduce8(const float (&v)[8], int lane) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
  float r[4], q[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float send = b4 ? v[i] : v[i + 4], keep = b4 ? v[i + 4] : v[i];
    r[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float send = b3 ? r[i] : r[i + 2], keep = b3 ? r[i + 2] : r[i];
    q[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const float send = b2 ? q[0] : q[1], keep = b2 ? q[1] : q[0];
  float p = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  p += __shfl_xor_sync(0xffffffffu, p, 2);
  p += __shfl_xor_sync(0xffffffffu, p, 1);
  return p;
}

// Same for 4 per-lane values: afterwards every lane holds the total of value ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1).
__device__ __forceinline__ float reduce4(const float (&v)[4], int lane) {
  const bool b4 = lane & 16, b3 = lane & 8;
  float r[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float send = b4 ? v[i] : v[i + 2], keep = b4 ? v[i + 2] : v[i];
    r[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
  const float send = b3 ? r[0] : r[1], keep = b3 ? r[1] : r[0];
  float p = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  p += __shfl_xor_sync(0xffffffffu, p, 4);
  p += __shfl_xor_sync(0xffffffffu, p, 2);
  p += __shfl_xor_sync(0xffffffffu, p, 1);
  return p;
}

// grid (ceil(Din / 32), batch), 32 * 16 / QS threads. dout is the gradient of `out`; with z given the gate's backward is applied
// here (dy = dout * silu(z), dz = dout * y_pre * silu'(z)).
template <typename DT, int QS>
__global__ void __launch_bounds__(Shape<QS>::NT, 4)
s6_bwd_kernel(const bf16* __restrict__ u, const DT* __restrict__ delta, const float* __restrict__ delta_bias,
              int softplus, const float* __restrict__ A, const float* __restrict__ Bm, const float* __restrict__ Cm,
              const float* __restrict__ Dv, const bf16* __restrict__ z, const bf16* __restrict__ y_pre,
              const bf16* __restrict__ dout, const float* __restrict__ state, bf16* __restrict__ du,
              DT* __restrict__ ddelta, float* __restrict__ dA, float* __restrict__ dB_part,
              float* __restrict__ dC_part, float* __restrict__ dD, bf16* __restrict__ dz,
              float* __restrict__ ddelta_bias, int L, int Din) {
  constexpr int NW = Shape<QS>::NW, NT = Shape<QS>::NT, RPT = Shape<QS>::RPT, BCPT = Shape<QS>::BCPT;
  __shared__ __align__(16) BwdSmem<QS> s;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int b = blockIdx.y, d0 = blockIdx.x * CB, d = d0 + lane, nblk = gridDim.x;
  const bool dok = d < Din;
  const int nsub = (L + SUB - 1) / SUB;
  float ar[QS], a2[QS], cr[QS], dAa[QS];
#pragma unroll
  for (int k = 0; k < QS; ++k) {
    ar[k] = dok ? A[(long long)d * NS + w * QS + k] : 0.f;
    a2[k] = ar[k] * LOG2E;
    cr[k] = 0.f;
    dAa[k] = 0.f;
  }
  const float bias = (dok && delta_bias) ? delta_bias[d] : 0.f;
  const float dsk = (dok && Dv) ? Dv[d] : 0.f;
  float dDa = 0.f, dbias = 0.f;
  for (int tile = nsub - 1; tile >= 0; --tile) {
    const int t0 = tile * SUB;
    float sp[RPT];  // d softplus / d raw for the rows this thread stages (and writes back)
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int t = w + NW * j;
      const bool ok = dok && t0 + t < L;
      const long long off = ((long long)b * L + t0 + t) * Din + d;
      float dtv = ok ? ld(delta, off) : 0.f;
      sp[j] = 1.f;
      if (softplus) {
        const float raw = dtv + bias;
        dtv = softplusf(raw, sp[j]);
        if (!ok) dtv = 0.f;
      }
      float g = ok ? __bfloat162float(dout[off]) : 0.f;
      if (z && ok) {
        const float zv = __bfloat162float(z[off]), sg = sigmoidf(zv);
        if (dz) dz[off] = __float2bfloat16_rn(g * __bfloat162float(y_pre[off]) * sg * (1.f + zv * (1.f - sg)));
        g *= zv * sg;
      }
      s.dt[t][lane] = dtv;
      s.u[t][lane] = ok ? __bfloat162float(u[off]) : 0.f;
      s.dy[t][lane] = g;
    }
#pragma unroll
    for (int j = 0; j < BCPT; ++j) {
      const int i = tid + NT * j, t = t0 + i / NS;
      const long long off = ((long long)b * L + t) * NS + (i % NS);
      s.B[i / NS][i % NS] = t < L ? Bm[off] : 0.f;
      s.C[i / NS][i % NS] = t < L ? Cm[off] : 0.f;
    }
    float h0[QS];
#pragma unroll
    for (int k = 0; k < QS; ++k) h0[k] = 0.f;
    if (dok) ldv<QS>(h0, &state[state_off(b, nsub, tile, w * QS, Din, d)]);
    __syncthreads();
    if (tile > 0) {  // warm L1 with the rows of the tile processed next (one tile earlier in time)
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        const long long off = ((long long)b * L + t0 - SUB + w + NW * j) * Din + d;
        if (dok) {
          prefetch_near(delta + off);
          prefetch_near(u + off);
          prefetch_near(dout + off);
          if (z) {
            prefetch_near(z + off);
            prefetch_near(y_pre + off);
          }
        }
      }
      if (dok) prefetch_near(&state[state_off(b, nsub, tile - 1, w * QS, Din, d)]);
      if (tid < 2 * SUB) {
        const long long off = ((long long)b * L + t0 - SUB + (tid >> 1)) * NS;
        prefetch_near((tid & 1) ? Cm + off : Bm + off);
      }
    }
    float hs[SUB][QS];
    {
      float hh[QS];
#pragma unroll
      for (int k = 0; k < QS; ++k) hh[k] = h0[k];
#pragma unroll
      for (int t = 0; t < SUB; ++t) {
        const float dt = s.dt[t][lane], dtu = dt * s.u[t][lane];
        float bb[QS];
        ldv<QS>(bb, &s.B[t][w * QS]);
#pragma unroll
        for (int k = 0; k < QS; ++k) {
          hh[k] = fmaf(ex2(dt * a2[k]), hh[k], dtu * bb[k]);
          hs[t][k] = hh[k];
        }
      }
    }
#pragma unroll
    for (int t = SUB - 1; t >= 0; --t) {
      const float dt = s.dt[t][lane], uu = s.u[t][lane], gy = s.dy[t][lane], dtu = dt * uu;
      float bb[QS], cc[QS];
      ldv<QS>(bb, &s.B[t][w * QS]);
      ldv<QS>(cc, &s.C[t][w * QS]);
      float v[2 * QS], ddt_p = 0.f, du_p = 0.f;
#pragma unroll
      for (int k = 0; k < QS; ++k) {
        const float gh = fmaf(cc[k], gy, cr[k]);  // dL/dh_t
        const float hprev = t > 0 ? hs[t - 1][k] : h0[k];
        const float gha = gh * ex2(dt * a2[k]);
        dAa[k] = fmaf(gha * hprev, dt, dAa[k]);
        ddt_p = fmaf(gha * hprev, ar[k], ddt_p);
        du_p = fmaf(gh, bb[k], du_p);
        v[k] = gh * dtu;
        v[QS + k] = gy * hs[t][k];
        cr[k] = gha;
      }
      s.pddt[w][t][lane] = fmaf(du_p, uu, ddt_p);  // d(dt * B * u) / d dt = B * u
      s.pdu[w][t][lane] = du_p * dt;
      if constexpr (QS == 4) {
        const float p = reduce8(v, lane);
        if ((lane & 3) == 0) {
          const int idx = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
          if (idx < 4) s.dB[t][w * QS + idx] = p;
          else s.dC[t][w * QS + idx - 4] = p;
        }
      } else {
        const float p = reduce4(v, lane);
        if ((lane & 7) == 0) {
          const int idx = ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
          if (idx < 2) s.dB[t][w * QS + idx] = p;
          else s.dC[t][w * QS + idx - 2] = p;
        }
      }
      if (w == 0) dDa = fmaf(gy, uu, dDa);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int t = w + NW * j;
      if (dok && t0 + t < L) {
        const long long off = ((long long)b * L + t0 + t) * Din + d;
        float g = 0.f, gu = dsk * s.dy[t][lane];
#pragma unroll
        for (int q = 0; q < NW; ++q) {
          g += s.pddt[q][t][lane];
          gu += s.pdu[q][t][lane];
        }
        g *= sp[j];
        st(ddelta, off, g);
        dbias += g;
        du[off] = __float2bfloat16_rn(gu);
      }
    }
#pragma unroll
    for (int j = 0; j < BCPT; ++j) {
      const int i = tid + NT * j, t = t0 + i / NS;
      if (t < L) {
        const long long off = ((((long long)b * nblk + blockIdx.x) * L) + t) * NS + (i % NS);
        dB_part[off] = s.dB[i / NS][i % NS];
        dC_part[off] = s.dC[i / NS][i % NS];
      }
    }
    __syncthreads();
  }
  if (dok) {
#pragma unroll
    for (int k = 0; k < QS; ++k) atomicAdd(&dA[(long long)d * NS + w * QS + k], dAa[k]);
    if (w == 0 && dD) atomicAdd(&dD[d], dDa);
    if (ddelta_bias) atomicAdd(&ddelta_bias[d], dbias);
  }
}

// One tile's inputs of the backward exactly as they lie in memory: filled by 16-byte cp.async copies one tile ahead of its
// use, so the walk over the sequence, which is serial per block, never waits for global memory.
template <typename DT>
struct RawTile {
  DT delta[SUB][PC];
  bf16 u[SUB][PC];
  bf16 dout[SUB][PC];
  bf16 z[SUB][PC];
  bf16 yp[SUB][PC];
  float B[SUB][NS];
  float C[SUB][NS];
  float st[4][PC][4];   // the state checkpoint of the tile: [group of four states][channel][state in group]
};

// Two channels' values as a packed pair, and back to memory
__device__ __forceinline__ uint64_t ld_pair(const float* p) { return *reinterpret_cast<const uint64_t*>(p); }
__device__ __forceinline__ uint64_t ld_pair(const bf16* p) {
  const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
  return f2_pack(v.x, v.y);
}
__device__ __forceinline__ void st_pair(float* p, uint64_t v) { *reinterpret_cast<uint64_t*>(p) = v; }
__device__ __forceinline__ void st_pair(bf16* p, uint64_t v) {
  float x, y;
  f2_unpack(v, x, y);
  *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(x, y);
}
// What the lane `m` away sends of its (a, b), added to this lane's: b of both where `up`, else a.
__device__ __forceinline__ uint64_t pair_exchange(uint64_t a, uint64_t b, bool up, int m) {
  return f2_add(up ? b : a, __shfl_xor_sync(0xffffffffu, up ? a : b, m));
}

// Backward of the pipelined form. Block = 16 channels, two warps of 4 pairs of channels x 8 groups of 2 states, one tile of 16
// steps at a time from the last to the first, the next tile copied by cp.async meanwhile. All arithmetic is on packed pairs of
// neighbouring channels, so what depends on the channel and step alone (dt, dt u, dL/dy) is a pair as it lies in shared memory;
// B and C, the same for all channels, are laid out there twice. A tile is walked forwards once
// to get the states at its steps 4, 8 and 12, then four steps at a time: their decays and states are formed and kept in
// registers (28 exponentials per 16 steps instead of 32 or a register per step), then the adjoint runs back over them.
// Sums over channels (dB, dC: 4 values a step) are halving exchanges of 3 shuffles a step; sums over states (d dt, d u of four
// steps: 8 pairs, one for each group) 3.5. dB / dC of the two warps meet in shared memory at the end of the tile and
// those of the two blocks of a 32-channel partial sum in memory: two atomic additions to a cleared value, the same in either
// order. At 8 x 4096 x 2048 that clears 268 MB and adds to it twice where blocks of 32 channels stored it once.
// Blocks of two warps spread evenly (8 x 2048 channels: 6.9 of 7 on every SM) at 128 registers a thread; the states in front of steps
// 0, 4 and 8 wait in shared memory, where they would be spilled. Loads of shared memory stand in front of the stores of their
// section: nothing can move them there.
// Bound: issue slots (0.6 of them used on average, four warps on two of an SM's schedulers and three on the others; 117 warp
// instructions per 128 state steps) and, with fewer warps, the chain of one (334 cycles a step). Measured, 8 x 4096 x 2048:
// 1.68 ms (1.86 ms with states in pairs: a channel and four states a thread, 141 instructions; 1.89 ms with the loads between the
// stores and lanes in the plain order), 1 x 4096 x 2048: 0.72 ms (1.02 ms), 3 x 1531 x 1024: 0.288 ms (0.397 ms).
constexpr int BWD_NT = 64;

template <typename DT>
struct BwdPipe {
  RawTile<DT> raw[2];
  ulonglong2 dt[SUB][PC / 2];   // {dt, dt u} of a pair of channels
  ulonglong2 gy[SUB][PC / 2];   // {dL/dy, u}
  uint64_t sp[SUB][PC / 2];     // d softplus
  uint64_t B[SUB][NS], C[SUB][NS];   // each value twice
  ulonglong2 h[3][BWD_NT];      // a thread's states in front of steps 0, 4 and 8
  float part[2][SUB][32];       // [warp][step][dB of 16 states, dC of 16 states]
};

template <typename DT>
__global__ void __launch_bounds__(BWD_NT, 7)
s6_bwd_pipe_kernel(const bf16* __restrict__ u, const DT* __restrict__ delta, const float* __restrict__ delta_bias,
                   int softplus, const float* __restrict__ A, const float* __restrict__ Bm, const float* __restrict__ Cm,
                   const float* __restrict__ Dv, const bf16* __restrict__ z, const bf16* __restrict__ y_pre,
                   const bf16* __restrict__ dout, const float* __restrict__ state, bf16* __restrict__ du,
                   DT* __restrict__ ddelta, float* __restrict__ dA, float* __restrict__ dB_part,
                   float* __restrict__ dC_part, float* __restrict__ dD, bf16* __restrict__ dz,
                   float* __restrict__ ddelta_bias, int L, int Din) {
  constexpr int NT = BWD_NT;
  extern __shared__ __align__(16) unsigned char s6_dyn_smem[];
  BwdPipe<DT>& s = *reinterpret_cast<BwdPipe<DT>*>(s6_dyn_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // group of two states, pair of channels. A 16-byte load of shared memory takes two cycles instead of four where lanes whose number
  // differs in bit 0, or in bit 1, read the same: bit 0 is of the pair (B, C) and bit 1 of the group (what depends on the channel).
  const int g = (lane >> 1 & 1) | (lane >> 2 & 6), cp = warp * 4 + ((lane & 1) | (lane >> 1 & 2)), c = 2 * cp;
  const int b = blockIdx.y, d0 = blockIdx.x * PC, d = d0 + c, nblk = (Din + CB - 1) / CB;
  const bool dok = d < Din;                                             // (Din is even)
  const int nsub = (L + SUB - 1) / SUB;
  uint64_t ar[2], a2[2], cr[2] = {0, 0}, dAa[2] = {0, 0};
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    const long long o = (long long)d * NS + 2 * g + n;
    ar[n] = dok ? f2_pack(A[o], A[o + NS]) : 0;
    a2[n] = f2_mul(ar[n], f2_pack(LOG2E, LOG2E));
  }
  const float2 bias = (dok && delta_bias) ? make_float2(delta_bias[d], delta_bias[d + 1]) : make_float2(0.f, 0.f);
  const uint64_t dsk = (dok && Dv) ? f2_pack(Dv[d], Dv[d + 1]) : 0;
  uint64_t acc = 0;                                                     // groups 0-3: d delta_bias, 4-7: dD

  // a thread copies one 16-byte piece of each pair of 32-byte rows and of B, C and the state checkpoint
  const int row = tid >> 2, piece = tid & 3;
  auto issue = [&](int tile, int buf) {
    RawTile<DT>& r = s.raw[buf];
    const bool rok = tile * SUB + row < L;
    const long long bt = (long long)b * L + min(tile * SUB + row, L - 1);
    const int ch = (piece & 1) * 8, n16 = (rok && d0 + ch < Din) ? 16 : 0;
    const long long off = bt * Din + min(d0 + ch, Din - 8);
    if (sizeof(DT) == 4) cp_async16(&r.delta[row][piece * 4], delta + bt * Din + min(d0 + piece * 4, Din - 4), (rok && d0 + piece * 4 < Din) ? 16 : 0);
    else if (piece < 2) cp_async16(&r.delta[row][ch], delta + off, n16);
    cp_async16(piece < 2 ? &r.u[row][ch] : &r.dout[row][ch], (piece < 2 ? u : dout) + off, n16);
    if (z) cp_async16(piece < 2 ? &r.z[row][ch] : &r.yp[row][ch], (piece < 2 ? z : y_pre) + off, n16);
    cp_async16(&r.B[row][piece * 4], Bm + bt * NS + piece * 4, rok ? 16 : 0);
    cp_async16(&r.C[row][piece * 4], Cm + bt * NS + piece * 4, rok ? 16 : 0);
    const int grp = tid >> 4, chn = tid & 15;
    cp_async16(&r.st[grp][chn][0], &state[state_off(b, nsub, tile, grp * 4, Din, min(d0 + chn, Din - 1))], d0 + chn < Din ? 16 : 0);
    cp_async_commit();
  };

  if (nsub > 0) issue(nsub - 1, 0);
  for (int tile = nsub - 1; tile >= 0; --tile) {
    const int t0 = tile * SUB, buf = (nsub - 1 - tile) & 1;
    cp_async_wait<0>();
    __syncthreads();           // the tile is visible, and the other buffer and `part` are free
    if (tile > 0) issue(tile - 1, buf ^ 1);
    const RawTile<DT>& r = s.raw[buf];
    // (all loads in front of the first store: neither compiler nor hardware can know that they do not meet)
    uint64_t in[2][5];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t = k * 8 + g;
      in[k][0] = ld_pair(&r.delta[t][c]), in[k][1] = ld_pair(&r.u[t][c]), in[k][2] = ld_pair(&r.dout[t][c]);
      if (z) in[k][3] = ld_pair(&r.z[t][c]), in[k][4] = ld_pair(&r.yp[t][c]);
    }
    const float4 vb = *reinterpret_cast<const float4*>(&r.B[row][piece * 4]), vc = *reinterpret_cast<const float4*>(&r.C[row][piece * 4]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int t = k * 8 + g;
      const bool ok = dok && t0 + t < L;
      float dt[2], sp[2] = {1.f, 1.f}, uu[2], gy[2];
      f2_unpack(in[k][0], dt[0], dt[1]);
      f2_unpack(in[k][1], uu[0], uu[1]);
      f2_unpack(in[k][2], gy[0], gy[1]);
      if (softplus) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          dt[q] = softplusf(dt[q] + (q ? bias.y : bias.x), sp[q]);
        }
      }
      if (z) {
        float zv[2], yp[2], o[2];
        f2_unpack(in[k][3], zv[0], zv[1]);
        f2_unpack(in[k][4], yp[0], yp[1]);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float sg = sigmoidf(zv[q]);
          o[q] = gy[q] * yp[q] * sg * (1.f + zv[q] * (1.f - sg));
          gy[q] *= zv[q] * sg;
        }
        if (dz && ok) st_pair(&dz[((long long)b * L + t0 + t) * Din + d], f2_pack(o[0], o[1]));
      }
      const ulonglong2 e1 = make_ulonglong2(f2_pack(dt[0], dt[1]), f2_pack(dt[0] * uu[0], dt[1] * uu[1]));
      const ulonglong2 e2 = make_ulonglong2(f2_pack(gy[0], gy[1]), f2_pack(uu[0], uu[1]));
      s.dt[t][cp] = ok ? e1 : make_ulonglong2(0, 0);
      s.gy[t][cp] = ok ? e2 : make_ulonglong2(0, 0);
      s.sp[t][cp] = f2_pack(sp[0], sp[1]);
    }
    {
      float4* ob = reinterpret_cast<float4*>(&s.B[row][piece * 4]);
      float4* oc = reinterpret_cast<float4*>(&s.C[row][piece * 4]);
      ob[0] = make_float4(vb.x, vb.x, vb.y, vb.y), ob[1] = make_float4(vb.z, vb.z, vb.w, vb.w);
      oc[0] = make_float4(vc.x, vc.x, vc.y, vc.y), oc[1] = make_float4(vc.z, vc.z, vc.w, vc.w);
    }
    __syncthreads();
    uint64_t h[2];
    {
      const float2 v0 = *reinterpret_cast<const float2*>(&r.st[g >> 1][c][2 * (g & 1)]);
      const float2 v1 = *reinterpret_cast<const float2*>(&r.st[g >> 1][c + 1][2 * (g & 1)]);
      h[0] = f2_pack(v0.x, v1.x), h[1] = f2_pack(v0.y, v1.y);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      s.h[k][tid] = make_ulonglong2(h[0], h[1]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 e = s.dt[4 * k + i][cp], bb = *reinterpret_cast<const ulonglong2*>(&s.B[4 * k + i][2 * g]);
        h[0] = f2_fma(f2_ex2(f2_mul(e.x, a2[0])), h[0], f2_mul(e.y, bb.x));
        h[1] = f2_fma(f2_ex2(f2_mul(e.x, a2[1])), h[1], f2_mul(e.y, bb.y));
      }
    }
#pragma unroll 1
    for (int k = 3; k >= 0; --k) {
      uint64_t hs[5][2], av[4][2], bb[4][2];
      hs[0][0] = h[0], hs[0][1] = h[1];
      if (k > 0) {
        const ulonglong2 v = s.h[k - 1][tid];
        h[0] = v.x, h[1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 e = s.dt[4 * k + i][cp], v = *reinterpret_cast<const ulonglong2*>(&s.B[4 * k + i][2 * g]);
        bb[i][0] = v.x, bb[i][1] = v.y;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          av[i][n] = f2_ex2(f2_mul(e.x, a2[n]));
          hs[i + 1][n] = f2_fma(av[i][n], hs[i][n], f2_mul(e.y, bb[i][n]));
        }
      }
      uint64_t ddt[4], duv[4];
      float bc[4];
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        const ulonglong2 e = s.dt[4 * k + i][cp], f = s.gy[4 * k + i][cp];
        const ulonglong2 cc = *reinterpret_cast<const ulonglong2*>(&s.C[4 * k + i][2 * g]);
        uint64_t dd = 0, dv = 0;
        float sum[4];                                          // dB of the two states, dC of them
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const uint64_t gh = f2_fma(n ? cc.y : cc.x, f.x, cr[n]);        // dL / dh_t
          cr[n] = f2_mul(gh, av[i][n]);
          const uint64_t w = f2_mul(cr[n], hs[i][n]);
          dAa[n] = f2_fma(w, e.x, dAa[n]);
          dd = n == 0 ? f2_mul(w, ar[n]) : f2_fma(w, ar[n], dd);
          dv = n == 0 ? f2_mul(gh, bb[i][n]) : f2_fma(gh, bb[i][n], dv);
          float x, y;
          f2_unpack(f2_mul(gh, e.y), x, y);
          sum[n] = x + y;
          f2_unpack(f2_mul(f.x, hs[i + 1][n]), x, y);
          sum[2 + n] = x + y;
        }
        duv[i] = f2_mul(dv, e.x);
        ddt[i] = f2_fma(dv, f.y, dd);                          // d(dt * B * u) / d dt = B * u
        // four sums over the 4 lanes of the warp's channels: lane q of them is left with value q
        const bool b2 = lane & 4, b1 = lane & 1;
        float p, q;
        f2_unpack(pair_exchange(f2_pack(sum[0], sum[1]), f2_pack(sum[2], sum[3]), b2, 4), p, q);
        const float send = b1 ? p : q, keep = b1 ? q : p;
        bc[i] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
      }
      const int t = 4 * k + (g & 3);
      const ulonglong2 f = s.gy[t][cp];
      const uint64_t sp = s.sp[t][cp];
      // sums over the eight groups of states: group i of the lower four is left with d dt of step i, of the upper four with d u
#pragma unroll
      for (int i = 0; i < 4; ++i) ddt[i] = pair_exchange(ddt[i], duv[i], g & 4, 16);
#pragma unroll
      for (int i = 0; i < 2; ++i) ddt[i] = pair_exchange(ddt[i], ddt[i + 2], g & 2, 8);
      const uint64_t v = pair_exchange(ddt[0], ddt[1], g & 1, 2);
#pragma unroll
      for (int i = 0; i < 4; ++i) s.part[warp][4 * k + i][(lane & 4 ? 16 : 0) + 2 * g + (lane & 1)] = bc[i];
      if (dok && t0 + t < L) {
        const long long off = ((long long)b * L + t0 + t) * Din + d;
        if (g & 4) {
          st_pair(&du[off], f2_fma(dsk, f.x, v));
          acc = f2_fma(f.x, f.y, acc);
        } else {
          st_pair(&ddelta[off], f2_mul(v, sp));
          acc = f2_fma(v, sp, acc);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SUB * 8 / NT; ++j) {
      const int i = tid + NT * j, t = i / 8, n = i % 8 * 4;
      if (t0 + t < L) {
        float* dst = (n < 16 ? dB_part : dC_part) + ((((long long)b * nblk + blockIdx.x / (CB / PC)) * L) + t0 + t) * NS + (n & 15);
        const float4 p = *reinterpret_cast<const float4*>(&s.part[0][t][n]), q = *reinterpret_cast<const float4*>(&s.part[1][t][n]);
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(p.x + q.x), "f"(p.y + q.y), "f"(p.z + q.z),
                     "f"(p.w + q.w) : "memory");
      }
    }
  }
  float x, y;
#pragma unroll
  for (int m = 2; m < 16; m <<= 2) acc = f2_add(acc, __shfl_xor_sync(0xffffffffu, acc, m));
  if (dok) {
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      f2_unpack(dAa[n], x, y);
      atomicAdd(&dA[(long long)d * NS + 2 * g + n], x);
      atomicAdd(&dA[(long long)(d + 1) * NS + 2 * g + n], y);
    }
    float* sum = g == 0 ? ddelta_bias : g == 4 ? dD : nullptr;
    if (sum) {
      f2_unpack(acc, x, y);
      atomicAdd(&sum[d], x);
      atomicAdd(&sum[d + 1], y);
    }
  }
}

void check(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace

int s6_channel_blocks(int Din) { return (Din + CB - 1) / CB; }
int s6_num_chunks(int L) { return (L + SUB - 1) / SUB; }

void s6_set_states_per_thread(int fwd_qs, int bwd_qs) {
  if ((fwd_qs != 2 && fwd_qs != 4 && fwd_qs != -1) || (bwd_qs != 2 && bwd_qs != 4))
    throw std::runtime_error("s6_scan: states per thread must be 2 or 4");
  g_fwd_qs = fwd_qs;
  g_bwd_qs = bwd_qs;
}

// What the 16-byte copies of the pipelined kernels need: channels in pieces of 8 and aligned tensors.
bool rows_aligned(int Din, std::initializer_list<const void*> ptrs) {
  if (Din % 8 != 0) return false;
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

template <typename DT>
void launch_bwd_pipe(dim3 grid, const void* u, const void* delta, const float* delta_bias, bool softplus, const float* A,
                     const float* Bm, const float* Cm, const float* Dv, const void* z, const void* y_pre, const void* dout,
                     const float* state, void* du, void* ddelta, float* dA, float* dB_part, float* dC_part, float* dD,
                     void* dz, float* ddelta_bias, int L, int Din, cudaStream_t st) {
  constexpr int bytes = (int)sizeof(BwdPipe<DT>);
  auto kern = s6_bwd_pipe_kernel<DT>;
  static PerDeviceOnce cfg;
  int dev = 0;
  if (cfg.pending(&dev)) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) throw std::runtime_error(std::string("s6_scan_bwd: ") + cudaGetErrorString(e));
    cfg.done(dev);
  }
  // two blocks of 16 channels add to every partial sum
  const size_t sums = (size_t)grid.y * grid.x * L * NS * sizeof(float);
  if (cudaMemsetAsync(dB_part, 0, sums, st) != cudaSuccess || cudaMemsetAsync(dC_part, 0, sums, st) != cudaSuccess)
    throw std::runtime_error("s6_scan_bwd: clearing the partial sums failed");
  const dim3 blocks((Din + PC - 1) / PC, grid.y);
  kern<<<blocks, BWD_NT, bytes, st>>>((const bf16*)u, (const DT*)delta, delta_bias, softplus ? 1 : 0, A, Bm, Cm, Dv, (const bf16*)z,
                                    (const bf16*)y_pre, (const bf16*)dout, state, (bf16*)du, (DT*)ddelta, dA, dB_part, dC_part,
                                    dD, (bf16*)dz, ddelta_bias, L, Din);
}

#define S6_FWD_PIPE(DT, QS)                                                                                           \
  s6_fwd_pipe_kernel<DT, QS><<<grid, 256 / QS, 0, st>>>((const bf16*)u, (const DT*)delta, delta_bias, softplus ? 1 : 0, \
                                                        A, Bm, Cm, Dv, (const bf16*)z, (bf16*)y_pre, (bf16*)out, state, L, Din)
#define S6_FWD(DT, QS)                                                                                               \
  s6_fwd_kernel<DT, QS><<<grid, Shape<QS>::NT, 0, st>>>((const bf16*)u, (const DT*)delta, delta_bias, softplus ? 1 : 0, \
                                                        A, Bm, Cm, Dv, (const bf16*)z, (bf16*)y_pre, (bf16*)out, state, L, Din)
#define S6_BWD(DT, QS)                                                                                               \
  s6_bwd_kernel<DT, QS><<<grid, Shape<QS>::NT, 0, st>>>((const bf16*)u, (const DT*)delta, delta_bias, softplus ? 1 : 0, \
                                                        A, Bm, Cm, Dv, (const bf16*)z, (const bf16*)y_pre,            \
                                                        (const bf16*)dout, state, (bf16*)du, (DT*)ddelta, dA, dB_part, \
                                                        dC_part, dD, (bf16*)dz, ddelta_bias, L, Din)

void s6_scan_fwd(const void* u, const void* delta, bool delta_bf16, const float* delta_bias, bool softplus,
                 const float* A, const float* Bm, const float* Cm, const float* Dv, const void* z, void* y_pre, void* out,
                 float* state, int batch, int L, int Din, int N, cudaStream_t st) {
  if (N != NS) throw std::runtime_error("s6_scan: state dimension must be 16");
  if (rows_aligned(Din, {u, delta, Bm, Cm, z})) {
    // Left alone: four states a thread while that gives every scheduler a warp (two warps a block, four schedulers a
    // multiprocessor); below that (few channels in flight) the time is the latency of one warp's walk over the sequence, which
    // two states a thread shorten.
    const int blocks = (Din + PC - 1) / PC;
    const bool q2 = g_fwd_qs == 2 || (g_fwd_qs < 0 && (long long)blocks * batch * 2 < 4ll * sm_count());
    const dim3 grid(blocks, batch);
    if (delta_bf16) {
      if (q2) S6_FWD_PIPE(bf16, 2); else S6_FWD_PIPE(bf16, 4);
    } else {
      if (q2) S6_FWD_PIPE(float, 2); else S6_FWD_PIPE(float, 4);
    }
    check("s6_scan_fwd");
    return;
  }
  dim3 grid(s6_channel_blocks(Din), batch);
  const bool q2 = g_fwd_qs != 4;
  if (delta_bf16) {
    if (q2) S6_FWD(bf16, 2); else S6_FWD(bf16, 4);
  } else {
    if (q2) S6_FWD(float, 2); else S6_FWD(float, 4);
  }
  check("s6_scan_fwd");
}

void s6_scan_bwd(const void* u, const void* delta, bool delta_bf16, const float* delta_bias, bool softplus,
                 const float* A, const float* Bm, const float* Cm, const float* Dv, const void* z, const void* y_pre,
                 const void* dout, const float* state, void* du, void* ddelta, float* dA, float* dB_part, float* dC_part,
                 float* dD, void* dz, float* ddelta_bias, int batch, int L, int Din, int N, cudaStream_t st) {
  if (N != NS) throw std::runtime_error("s6_scan: state dimension must be 16");
  if (z && !y_pre) throw std::runtime_error("s6_scan_bwd: the gate's backward needs y_pre");
  dim3 grid(s6_channel_blocks(Din), batch);
  if (g_bwd_qs == 4 && rows_aligned(Din, {u, delta, Bm, Cm, z, y_pre, dout, state, du, ddelta, dB_part, dC_part, dz})) {
    if (delta_bf16)
      launch_bwd_pipe<bf16>(grid, u, delta, delta_bias, softplus, A, Bm, Cm, Dv, z, y_pre, dout, state, du, ddelta, dA,
                            dB_part, dC_part, dD, dz, ddelta_bias, L, Din, st);
    else
      launch_bwd_pipe<float>(grid, u, delta, delta_bias, softplus, A, Bm, Cm, Dv, z, y_pre, dout, state, du, ddelta, dA,
                             dB_part, dC_part, dD, dz, ddelta_bias, L, Din, st);
    check("s6_scan_bwd");
    return;
  }
  const bool q2 = g_bwd_qs == 2;
  if (delta_bf16) {
    if (q2) S6_BWD(bf16, 2); else S6_BWD(bf16, 4);
  } else {
    if (q2) S6_BWD(float, 2); else S6_BWD(float, 4);
  }
  check("s6_scan_bwd");
}

}  // namespace b200
