// See tele_band.h. Telephone attention as products with band matrices on the tensor cores.
//
// A query's taps are W x with a sparse row of W: two neighbouring keys per tap, taps one stride apart, so with strides of 1..16
// about one key in eight of the band that 128 neighbouring queries reach has a weight. Gathering rows tap by tap moves 2 D
// values per tap through L2, and its transpose adds them there with fp32 atomics. Here the weights are written into dense tiles
// of W instead: eight times the multiplications, but on tcgen05.mma, where they cost less than the tap formulas.
//   forward   Y  = W X            queries stay, the block walks the keys of its band
//   rows      S  = dY Xᵀ, read at the taps: gradients of stride, phase, table and exponent; queries stay
//   dX        dX = Wᵀ dY          keys stay, the block walks the query tiles that reach them: nothing is added in memory
// 8 x 16384 tokens x 4 heads of 64, 235 taps: forward 1.12 ms (3.57 gathered), rows 1.35 + dX 2.0 (10.3 gathered). The bound is the
// issue of the tap formulas and of the conversion of tiles (54 to 62 % of the issue slots; the tensor pipe is 15 % busy).
//
// Weights are evaluated in fp32 and enter the product as a sum of three bf16 terms, which hold all 24 bits of them; x and dY are
// bf16 already, sums are fp32. (With two terms, 16 bits: 0.97 and 1.75 ms.)
// A thread builds 32 keys of one query in a column of shared memory of its own ([cell][thread]: whatever cells the lanes of a
// warp touch, they are in 32 different banks), then splits them into terms. The queries of a tile are sorted by stride, so the lanes
// of a warp have about the same number of taps in a step.
#include "tele_band.h"

#include <cuda_bf16.h>

#include <cfloat>
#include <climits>
#include <cmath>
#include <stdexcept>
#include <string>

#include "../common/per_device.h"
#include "../common/ptx.cuh"
#include "../common/tmap.h"

namespace b200 {
namespace {
using bf16 = __nv_bfloat16;

constexpr int ROWS = 128;             // queries of a block (forward, rows) / keys of a block (dX)
constexpr int STEP = 64;              // keys (dX: queries) of a step
constexpr int SEG = 32;               // keys that a thread builds in a step
constexpr int BUILDERS = 256;
constexpr int TERMS = 3;              // bf16 terms of a weight
constexpr int THREADS = BUILDERS + 64;   // two warps more: one issues the MMAs, one the TMA loads
// A tap of keys c - 1, c is written at cells c + 1, c + 2: cells 0, 1 and SEG + 2 are for what belongs to other segments
constexpr int CELL_BYTES = (SEG + 3) * BUILDERS * 4;

struct Query;
struct BP {
  const bf16* x;
  const float* freq;
  const float* phase;
  const float* kern;
  const float* expo;
  const bf16* dout;
  bf16* out;                // forward
  void* dx;                 // dX: bf16 or fp32
  float* dfreq;
  float* dphase;
  float* dkern;
  float* dexpo_h;
  const int2* ranges;       // dX: keys that a tile of 64 queries reaches
  const Query* queries;   // dX: the queries of a tile by stride
  int L, H, K, half, D, kvec;
  float inv_rec, invL;
  int* status;
};

template <int N>
__device__ __forceinline__ void builders_sync() { asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ bool builders_any(bool v) {
  int any;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\nselp.b32 %0, 1, 0, q;\n}\n" : "=r"(any) : "r"((int)v), "n"(N) : "memory");
  return any != 0;
}
__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) <= FLT_MAX; }
// The columns of `of` that are no number
__device__ __forceinline__ uint32_t nan_columns(const float (&of)[16]) {
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) m |= of[k] == of[k] ? 0u : 1u << k;
  return m;
}
// 16 columns of a row, times a weight
__device__ __forceinline__ void add_row(float (&acc)[16], float w, const uint4* row) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint4 u = row[i];
    const uint32_t v[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      acc[8 * i + 2 * k] = fmaf(w, __uint_as_float(v[k] << 16), acc[8 * i + 2 * k]);
      acc[8 * i + 2 * k + 1] = fmaf(w, __uint_as_float(v[k] & 0xffff0000u), acc[8 * i + 2 * k + 1]);
    }
  }
}

// The taps of one query. A position is rounded three times, as the operator states it, (l + tap * stride) + phase: which rows are read is
// part of its definition. Positions never fall along the taps; the sign of the stride only swaps the taps' names.
struct Taps {
  float f, ph;               // stride without its sign, phase
  float inv, from, to;       // taps of an interval of positions, see tap_range
  float lf;                  // the query's own position
  int l, lo, hi;             // the taps lo..hi are inside the sequence (none if lo > hi)
  int kmin, kmax;            // keys that they touch
};
__device__ __forceinline__ float tap_position(float lf, float f, float ph, float s) { return __fadd_rn(__fadd_rn(lf, __fmul_rn(s, f)), ph); }
__device__ __forceinline__ float tap_position(const Taps& t, float s) { return tap_position(t.lf, t.f, t.ph, s); }
// First tap of [lo, hi + 1] at a position of at least x: an estimate, made exact by looking at its neighbours.
__device__ __forceinline__ int first_tap(float lf, float f, float ph, float x, int lo, int hi) {
  const float est = ceilf((x - lf - ph) / f);
  int s = est >= (float)lo ? (est <= (float)hi ? (int)est : hi + 1) : lo;
  while (s > lo && tap_position(lf, f, ph, (float)(s - 1)) >= x) --s;
  while (s <= hi && tap_position(lf, f, ph, (float)s) < x) ++s;
  return s;
}
// Floor of a position in the low bits of a float, by an addition that is rounded down: the integer is bits(m) - MAGIC_BITS.
constexpr float MAGIC = 12582912.f;     // 1.5 * 2^23
constexpr int MAGIC_BITS = 0x4B400000;
__device__ __forceinline__ float floor_magic(float x) { return __fadd_rd(x, MAGIC); }
__device__ __forceinline__ int floor_int(float x) { return __float_as_int(floor_magic(x)) - MAGIC_BITS; }
// Positions are limited to L - 1.001, whose floor is L - 2 up to 32768 tokens.
__device__ __forceinline__ float last_position(int L) { return (float)L - 1.001f; }

// f without its sign; lo, hi as first_tap finds them
__device__ __forceinline__ Taps make_taps(float f, float phase, int l, int lo, int hi, int L) {
  Taps t;
  t.f = f, t.ph = phase, t.l = l, t.lf = (float)l, t.lo = lo, t.hi = hi;
  // An estimate of the taps in an interval is off by less than 1/8 for strides of 1/4 and phases of 8192 (inv: 2^-22 of up to 2^15 taps;
  // the positions themselves by 2^-8 of a row). Others look at all their taps wherever they have any.
  const bool tight = f >= 0.25f && fabsf(phase) <= 8192.f;
  t.inv = tight ? 1.f / f : 0.f;
  t.from = tight ? -phase * t.inv - 0.125f : -1e6f;
  t.to = tight ? -phase * t.inv + 0.125f : 1e6f;
  t.kmin = INT_MAX, t.kmax = -1;
  if (lo <= hi) {
    t.kmin = floor_int(fminf(tap_position(t, (float)lo), last_position(L)));
    t.kmax = floor_int(fminf(tap_position(t, (float)hi), last_position(L))) + 1;
  }
  return t;
}
__device__ __forceinline__ int2 inside(float f, float phase, int l, int L, int half) {
  if (!(f <= FLT_MAX && fabsf(phase) <= FLT_MAX)) return make_int2(0, -1);   // no tap is inside the sequence
  const int lo = first_tap((float)l, f, phase, 0.f, -half, half);
  return make_int2(lo, first_tap((float)l, f, phase, (float)L, lo, half) - 1);
}
// Taps that may touch the keys [k0, k1): all that do, and perhaps a neighbour on either side.
__device__ __forceinline__ int2 tap_range(const Taps& t, int k0, int k1, int L) {
  const int s0 = max(t.lo, (int)ceilf(fmaf((float)(k0 - 1 - t.l), t.inv, t.from)));
  const int s1 = k1 >= L - 1 ? t.hi : min(t.hi, (int)floorf(fmaf((float)(k1 - t.l), t.inv, t.to)));
  return make_int2(s0, k0 <= t.kmax && k1 > t.kmin ? s1 : s0 - 1);
}

__device__ __forceinline__ void tmem_ld(uint32_t at, uint32_t (&v)[16]) { tmem_ld_32x32b_x16(at, v); }
__device__ __forceinline__ void tmem_ld(uint32_t at, uint32_t (&v)[32]) { tmem_ld_32x32b_x32(at, v); }

struct Entry {
  int lo;
  float wh, v, slope;
};
// Entry of a table of K values at t (limited to [0, 1]); value k of this thread is tab[k * stride].
__device__ __forceinline__ Entry table_entry(const float* tab, int stride, int K, float t) {
  Entry e;
  const float idx = fminf(fmaxf(t, 0.f), 1.f) * (float)(K - 1);
  e.lo = min((int)idx, K - 2);
  e.wh = idx - (float)e.lo;
  const float a = tab[e.lo * stride], b = tab[(e.lo + 1) * stride];
  e.v = a * (1.f - e.wh) + b * e.wh;
  e.slope = (t >= 0.f && t <= 1.f) ? (b - a) * (float)(K - 1) : 0.f;
  return e;
}
__device__ __forceinline__ float decay(float expo, float ar, float invL) { return exp2f(-expo * log2f(1.f + ar * invL)); }

// The table rows of n queries into shared memory, value k of query r at tab[k * n + r]; thread r, r + n, ... share a row.
__device__ __forceinline__ void stage_table(float* tab, const float* row, bool ok, int r, int n, int part, int parts, int K, bool vec) {
  if (vec) {
    for (int k = part; k < K / 4; k += parts) {
      const float4 v = ok ? reinterpret_cast<const float4*>(row)[k] : make_float4(0.f, 0.f, 0.f, 0.f);
      tab[(4 * k) * n + r] = v.x;
      tab[(4 * k + 1) * n + r] = v.y;
      tab[(4 * k + 2) * n + r] = v.z;
      tab[(4 * k + 3) * n + r] = v.w;
    }
  } else {
    for (int k = part; k < K; k += parts) tab[k * n + r] = ok ? row[k] : 0.f;
  }
}

// Weights of the taps of one query that touch the keys [k0, k0 + SEG), into the thread's column of cells (key k0 + c in cell c + 2),
// which must be zero. Sums of taps on one row are kept in registers and a cell is written again with every addition, so nothing is
// read back. False if there are no taps.
template <typename W>
__device__ __forceinline__ bool add_taps(float* col, const Taps& t, int k0, int L, W weights) {
  const int2 r = tap_range(t, k0, k0 + SEG, L);
  const int shift = 2 - k0 - MAGIC_BITS;
  const float end = last_position(L);
  float a = 0.f, b = 0.f;          // of the row below the last tap and of the next
  int last = INT_MIN;
  for (int s = r.x; s <= r.y; s += 2) {
    float w[2];
    weights(s, w);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float pos = fminf(tap_position(t, (float)(s + j)), end), m = floor_magic(pos), fr = pos - (m - MAGIC);
      const int at = __float_as_int(m);
      a = (at == last ? a : at == last + 1 ? b : 0.f) + fmaf(-w[j], fr, w[j]);
      b = fmaf(w[j], fr, at == last ? b : 0.f);
      last = at;
      unsigned u = (unsigned)(at + shift);
      if (u > SEG + 1 || s + j > r.y) u = 0;
      col[u * BUILDERS] = a;
      col[u * BUILDERS + BUILDERS] = b;
    }
  }
  return r.x <= r.y;
}
// Two weights as pairs of bf16 terms; what is left of them after this term.
__device__ __forceinline__ uint32_t take_term(float& a, float& b) {
  const uint32_t h = pack_bf16x2(a, b);
  a -= __uint_as_float(h << 16);
  b -= __uint_as_float(h & 0xffff0000u);
  return h;
}

// What all three kernels do to set up and to end: barriers, tensor memory, one decision to leave.
struct Frame {
  uint32_t tmem;
  bool leave;
};
__device__ __forceinline__ Frame frame_begin(uint64_t* bars, int nbar, const int* counts, uint32_t* slot, volatile int* abort_flag, uint32_t cols,
                                             const int* status, int alloc_warp = 8) {
  const bool poisoned = status_poisoned(status);
  if (threadIdx.x == 0) {
    for (int i = 0; i < nbar; ++i) mbar_init(&bars[i], counts[i]);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (threadIdx.x / 32 == alloc_warp) {
    tmem_alloc(slot, cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  Frame f;
  f.leave = __syncthreads_or(poisoned);
  tc_fence_after_sync();
  f.tmem = *slot;
  return f;
}
__device__ __forceinline__ void frame_end(uint32_t tmem, uint32_t cols, volatile int* abort_flag, int alloc_warp = 8) {
  __syncwarp();
  if (*abort_flag && threadIdx.x == 0) {   // let loads still in flight land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (threadIdx.x / 32 == alloc_warp) tmem_dealloc(tmem, cols);
}

// The block's queries by stride: perm[slot] = query, and the keys that their taps reach. All threads call it.
struct Band {
  int lo, n;     // first key, number of steps
};
__device__ __forceinline__ Taps sorted_taps(const BP& p, int b, int h, int q0, uint32_t* key, uint8_t* perm, int* range, int step, Band* band) {
  const int tid = threadIdx.x;
  if (tid < ROWS) {
    const int l = q0 + tid;
    key[tid] = l < p.L ? __float_as_uint(fabsf(p.freq[((long long)b * p.L + l) * p.H + h])) : 0xffffffffu;
  }
  if (tid == ROWS) range[0] = INT_MAX, range[1] = -1;
  __syncthreads();
  if (tid < ROWS) {
    const uint32_t mine = key[tid];
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < ROWS; ++j) rank += (key[j] < mine || (key[j] == mine && j < tid)) ? 1 : 0;
    perm[rank] = (uint8_t)tid;
  }
  __syncthreads();
  const int l = q0 + perm[tid & (ROWS - 1)];
  float f = 0.f, ph = 0.f;
  int2 in = make_int2(0, -1);
  if (l < p.L) {
    const long long row = ((long long)b * p.L + l) * p.H + h;
    f = fabsf(p.freq[row]), ph = p.phase[row];
    in = inside(f, ph, l, p.L, p.half);
  }
  const Taps t = make_taps(f, ph, l, in.x, in.y, p.L);
  if (tid < ROWS) {
    const int wlo = __reduce_min_sync(0xffffffffu, t.kmin), whi = __reduce_max_sync(0xffffffffu, t.kmax);
    if ((tid & 31) == 0) atomicMin(&range[0], wlo), atomicMax(&range[1], whi);
  }
  __syncthreads();
  band->lo = range[0];
  band->n = range[1] >= range[0] ? (range[1] - range[0]) / step + 1 : 0;
  return t;
}

// Weights of a query by |tap|, at wt[tap * ROWS + row], by PARTS threads a row. The queries' tables are staged in `tab` first.
template <int PARTS>
__device__ __forceinline__ void fill_weights(const BP& p, float* wt, float* tab, const Taps& t, bool ok, long long row, float expo) {
  const int r = threadIdx.x & (ROWS - 1), part = threadIdx.x / ROWS;
  stage_table(tab, p.kern + row * p.K, ok, r, ROWS, part, PARTS, p.K, p.kvec);
  builders_sync<PARTS * ROWS>();
  for (int s = part; s <= p.half; s += 4 * PARTS) {          // four at a time: a store keeps later loads from starting early
    float w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float ar = (float)(s + j * PARTS) * t.f;
      w[j] = ok ? table_entry(tab + r, ROWS, p.K, ar * p.inv_rec).v * decay(expo, ar, p.invL) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (s + j * PARTS <= p.half) wt[(s + j * PARTS) * ROWS + r] = w[j];
  }
  builders_sync<PARTS * ROWS>();
}

// ------------------------------------------------------------------------------------------------ forward
template <int N>
struct FwdShape {
  static constexpr int NS = N / 64, XST = N == 128 ? 1 : 2;
  static constexpr int NAB = N == 128 ? 1 : 2;     // tiles of W in tensor memory, of which two blocks share the 512 columns
  static constexpr int X_BYTES = NS * STEP * 128;
  static constexpr uint32_t COLS = 256;            // N of results, the tiles in three terms of 32
  static size_t smem(int half) { return (size_t)XST * X_BYTES + CELL_BYTES + (size_t)(half + 2) * ROWS * 4 + 1024; }
};

// Results that are not finite: a row of x that the query does not sample may have spoiled them, as 0 * inf does. Tap by tap, then, 16 columns
// at a time, until all that are wanted are no numbers, which they then stay. 8 x 16384 x 4 heads of 64: 1.18 ms where all of x is NaN, 7.1
// with some NaN in every 64th row (3.6 in the gather, whatever the values).
__device__ __noinline__ void gathered(const Taps& t, const float* wt, const bf16* xcol, long long rs, int L, uint32_t wanted, float (&acc)[16]) {
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] = 0.f;
  for (int s = t.lo; s <= t.hi && (wanted & ~nan_columns(acc)); ++s) {
    const float w = wt[(s < 0 ? -s : s) * ROWS];
    if (w == 0.f) continue;
    const float pos = fminf(tap_position(t, (float)s), last_position(L));
    const int fl = floor_int(pos);
    const float fr = pos - (float)fl;
    add_row(acc, w * (1.f - fr), reinterpret_cast<const uint4*>(xcol + fl * rs));
    add_row(acc, w * fr, reinterpret_cast<const uint4*>(xcol + (fl + 1) * rs));
  }
}

template <int N>
__global__ void __launch_bounds__(THREADS, 2)
tele_band_fwd_kernel(const __grid_constant__ CUtensorMap tmX, const BP p) {
  using F = FwdShape<N>;
  constexpr int XST = F::XST, NAB = F::NAB, NBAR = 2 * NAB + 1 + 2 * XST;
  constexpr uint32_t A_COL = N, TERM = 32, BUF = TERMS * TERM;
  static_assert(A_COL + NAB * BUF <= F::COLS, "tensor memory");
  extern __shared__ __align__(1024) uint8_t raw[];
  // (rounded up by an offset: through an integer the compiler would lose sight of the address space and use generic accesses)
  uint8_t* sX = raw + (-smem_u32(raw) & 1023u);
  float* cells = reinterpret_cast<float*>(sX + XST * F::X_BYTES);
  float* wt = cells + CELL_BYTES / 4;
  __shared__ uint64_t bars[NBAR];
  __shared__ uint32_t key[ROWS];
  __shared__ uint8_t perm[ROWS];
  __shared__ int range[2];
  __shared__ uint32_t slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  uint64_t *a_full = bars, *a_free = bars + NAB, *done = bars + 2 * NAB, *x_full = done + 1, *x_empty = x_full + XST;
  int counts[NBAR];
#pragma unroll
  for (int i = 0; i < NBAR; ++i) counts[i] = i < NAB ? 8 : 1;
  const Frame fr = frame_begin(bars, NBAR, counts, &slot, abort_flag, F::COLS, p.status);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (fr.leave) {
    if (warp == 8) tmem_dealloc(fr.tmem, F::COLS);
    return;
  }
  const int nq = (p.L + ROWS - 1) / ROWS;
  const int q0 = (blockIdx.x % nq) * ROWS, h = (blockIdx.x / nq) % p.H, b = blockIdx.x / (nq * p.H);
  Band band;
  const Taps t = sorted_taps(p, b, h, q0, key, perm, range, STEP, &band);

  if (warp == 9) {
    if (elect_one_sync()) {
      for (int i = 0; i < band.n; ++i) {
        const int st = i % XST;
        cta_wait(&x_empty[st], ((i / XST) & 1) ^ 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(&x_full[st], F::X_BYTES);
        for (int s = 0; s < F::NS; ++s)
          tma_load_3d(sX + st * F::X_BYTES + s * STEP * 128, &tmX, &x_full[st], h * p.D + s * 64, band.lo + i * STEP, b);
      }
    }
  } else if (warp == 8) {
    const uint32_t idesc = make_idesc(FMT_BF16, FMT_BF16, 0, 1, 128, N);
    const uint64_t xd = make_smem_desc_sw128(smem_u32(sX), STEP * 128, 1024);
    for (int i = 0; i < band.n; ++i) {
      const int st = i % XST, bf = i % NAB;
      cta_wait(&x_full[st], (i / XST) & 1, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
      cta_wait(&a_full[bf], (i / NAB) & 1, abort_flag, p.status, ERR_WAIT_MISC);
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      tc_fence_after_sync();
      if (elect_one_sync()) {
#pragma unroll
        for (int term = 0; term < TERMS; ++term)
#pragma unroll
          for (int ks = 0; ks < STEP / 16; ++ks)
            tc_mma_f16_ts(fr.tmem, fr.tmem + A_COL + bf * BUF + term * TERM + ks * 8, xd + (st * F::X_BYTES + ks * 2048) / 16, idesc,
                          (i | term | ks) != 0);
        // only what somebody waits for is reported: nothing may arrive after the block has ended
        if (i + NAB < band.n) tc_commit(&a_free[bf]);
        if (i + XST < band.n) tc_commit(&x_empty[st]);
        if (i + 1 == band.n) tc_commit(done);
      }
      __syncwarp();
    }
  } else {
    const int row = tid & (ROWS - 1), part = tid / ROWS;
    const bool ok = t.l < p.L;
    const long long bl = (long long)b * p.L + (ok ? t.l : 0), grow = bl * p.H + h;
    fill_weights<2>(p, wt, cells, t, ok, grow, p.expo[bl]);
    float* col = cells + tid;
#pragma unroll
    for (int c = 2; c < SEG + 2; ++c) col[c * BUILDERS] = 0.f;
    const float* wrow = wt + row;
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    uint32_t zero = 0;                                    // buffers in which this warp's part is zero
    for (int i = 0; i < band.n; ++i) {
      const int bf = i % NAB;
      const bool any = __any_sync(0xffffffffu, add_taps(col, t, band.lo + i * STEP + part * SEG, p.L, [&](int s, float (&w)[2]) {
        w[0] = wrow[abs(s) * ROWS], w[1] = wrow[abs(s + 1) * ROWS];
      }));
      if (i >= NAB) cta_wait(&a_free[bf], ((i / NAB) & 1) ^ 1, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY);
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      tc_fence_after_sync();
      if (any || !(zero >> bf & 1)) {
        uint32_t o[TERMS][16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          float v0 = 0.f, v1 = 0.f;
          if (any) {
            float* c = col + (2 * k + 2) * BUILDERS;
            v0 = c[0], v1 = c[BUILDERS];
            c[0] = 0.f, c[BUILDERS] = 0.f;
          }
#pragma unroll
          for (int term = 0; term < TERMS; ++term) o[term][k] = take_term(v0, v1);
        }
        const uint32_t at = fr.tmem + lane_off + A_COL + bf * BUF + part * 16;
#pragma unroll
        for (int term = 0; term < TERMS; ++term) tmem_st_32x32b_x16(at + term * TERM, o[term]);
        tmem_st_wait();
        zero = any ? zero & ~(1u << bf) : zero | (1u << bf);
      }
      tc_fence_before_sync();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&a_full[bf]);
    }
    if (band.n > 0) cta_wait(done, 0, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
    tc_fence_after_sync();
    const int cols = p.D >= 32 ? p.D / 2 : p.D, first = part * cols;   // 16 wide: the first half of the threads has them all
    const bf16* xcol = p.x + (long long)b * p.L * p.H * p.D + h * p.D;
    bf16* orow = p.out + grow * p.D;
    for (int c0 = first; c0 < first + cols && c0 < p.D; c0 += 16) {
      uint32_t v[16];
      tmem_ld_32x32b_x16(fr.tmem + lane_off + c0, v);
      tmem_ld_wait();
      if (ok) {
        float y[16];
        uint32_t bad = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
          y[k] = band.n > 0 ? __uint_as_float(v[k]) : 0.f;
          bad |= is_finite(y[k]) ? 0u : 1u << k;
        }
        if (bad) {
          float g[16];
          gathered(t, wrow, xcol + c0, (long long)p.H * p.D, p.L, bad, g);
#pragma unroll
          for (int k = 0; k < 16; ++k)
            if (bad >> k & 1) y[k] = g[k];
        }
        uint32_t o[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) o[k] = pack_bf16x2(y[2 * k], y[2 * k + 1]);
        reinterpret_cast<uint4*>(orow + c0)[0] = make_uint4(o[0], o[1], o[2], o[3]);
        reinterpret_cast<uint4*>(orow + c0)[1] = make_uint4(o[4], o[5], o[6], o[7]);
      }
    }
  }
  frame_end(fr.tmem, F::COLS, abort_flag);
}

// ------------------------------------------------------------------------------------------------ gradients of the rows' scalars
// S = dY Xᵀ for 64 or 128 keys at a time, copied from tensor memory to shared memory ([key][row]: lanes are rows, so any key they look
// up is in their own bank). The four threads of a row take the taps by |tap| mod 4, so each |tap| belongs to one of them and
// its share of dW is added up in `sums` without atomics. What depends on |tap| alone (table, exponent, stride through
// the weight) is done once per |tap| at the end. The two tables of the taps leave room for one block on a multiprocessor, hence four
// threads a row: with two, most issue slots were lost to the latency of the look-ups.
constexpr int RPARTS = 4, RBUILDERS = RPARTS * ROWS, RTHREADS = RBUILDERS + 64;
template <int N>
struct RowsShape {
  static constexpr int NS = N / 64, RS = N == 128 ? 64 : 128, XST = N == 128 ? 2 : 1;   // keys of a step, stages of x
  static constexpr int X_BYTES = NS * RS * 128, Q_BYTES = NS * ROWS * 128;
  static constexpr int SCORES = (RS + 3) * ROWS * 4;           // scores of a step between guard rows of zeros, placed as cells are
  static constexpr int NSC = 512 / RS;             // scores in tensor memory: the warps, whose bands differ, may be that many steps apart
  static constexpr uint32_t COLS = 512;
  static constexpr int REGION = Q_BYTES + XST * X_BYTES + SCORES;    // at the end: the table and two sums of its gradient
  static size_t smem(int half) { return REGION + 2 * (size_t)(half + 1) * ROWS * 4 + 1024; }
  static_assert(REGION >= 3 * 64 * ROWS * 4, "tables of 64 values and two sums of their gradients");
};

template <int N>
__global__ void __launch_bounds__(RTHREADS, 1)
tele_band_rows_kernel(const __grid_constant__ CUtensorMap tmX, const BP p) {
  using F = RowsShape<N>;
  constexpr int RS = F::RS, XST = F::XST, NSC = F::NSC, RCOLS = RS / RPARTS, NBAR = 2 * NSC + 2 * XST, MMA_WARP = RBUILDERS / 32;
  extern __shared__ __align__(1024) uint8_t raw[];
  uint8_t* sQ = raw + (-smem_u32(raw) & 1023u);
  uint8_t* sX = sQ + F::Q_BYTES;
  float* scores = reinterpret_cast<float*>(sX + XST * F::X_BYTES);
  float* wt = reinterpret_cast<float*>(sQ + F::REGION);
  float* sums = wt + (p.half + 1) * ROWS;
  __shared__ uint64_t bars[NBAR];
  __shared__ uint32_t key[ROWS];
  __shared__ uint8_t perm[ROWS];
  __shared__ int range[2];
  __shared__ float other[RPARTS - 1][3][ROWS];
  __shared__ uint32_t slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  uint64_t *s_full = bars, *s_free = bars + NSC, *x_full = bars + 2 * NSC, *x_empty = x_full + XST;
  int counts[NBAR];
#pragma unroll
  for (int i = 0; i < NBAR; ++i) counts[i] = i >= NSC && i < 2 * NSC ? RBUILDERS / 32 : 1;
  const Frame fr = frame_begin(bars, NBAR, counts, &slot, abort_flag, F::COLS, p.status, MMA_WARP);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (fr.leave) {
    if (warp == MMA_WARP) tmem_dealloc(fr.tmem, F::COLS);
    return;
  }
  const int nq = (p.L + ROWS - 1) / ROWS;
  const int q0 = (blockIdx.x % nq) * ROWS, h = (blockIdx.x / nq) % p.H, b = blockIdx.x / (nq * p.H);
  Band band;
  const Taps t = sorted_taps(p, b, h, q0, key, perm, range, RS, &band);
  if (tid < RBUILDERS) {                                   // dY of the sorted queries: 128-byte swizzled rows
    const int row = tid & (ROWS - 1), l = q0 + perm[row];
    const uint4* src = reinterpret_cast<const uint4*>(p.dout + (((long long)b * p.L + l) * p.H + h) * p.D);
    for (int c = tid / ROWS; c < p.D / 8; c += RPARTS)
      *reinterpret_cast<uint4*>(sQ + (c / 8) * (ROWS * 128) + row * 128 + (((c & 7) ^ (row & 7)) * 16)) = l < p.L ? src[c] : make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
  }
  __syncthreads();

  if (warp == MMA_WARP + 1) {
    if (elect_one_sync()) {
      for (int i = 0; i < band.n; ++i) {
        const int st = i % XST;
        cta_wait(&x_empty[st], ((i / XST) & 1) ^ 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(&x_full[st], F::X_BYTES);
        for (int s = 0; s < F::NS; ++s)
          for (int k = 0; k < RS; k += STEP)
            tma_load_3d(sX + st * F::X_BYTES + (s * RS + k) * 128, &tmX, &x_full[st], h * p.D + s * 64, band.lo + i * RS + k, b);
      }
    }
  } else if (warp == MMA_WARP) {
    const uint32_t idesc = make_idesc(FMT_BF16, FMT_BF16, 0, 0, 128, RS);
    const uint64_t qd = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), xd = make_smem_desc_sw128(smem_u32(sX), 16, 1024);
    for (int i = 0; i < band.n; ++i) {
      const int st = i % XST, sc = i % NSC;
      cta_wait(&x_full[st], (i / XST) & 1, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
      cta_wait(&s_free[sc], ((i / NSC) & 1) ^ 1, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY);
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      tc_fence_after_sync();
      if (elect_one_sync()) {
        for (int ks = 0; ks < p.D / 16; ++ks)
          tc_mma_f16(fr.tmem + sc * RS, qd + ((ks / 4) * (ROWS * 128) + (ks % 4) * 32) / 16,
                     xd + (st * F::X_BYTES + (ks / 4) * (RS * 128) + (ks % 4) * 32) / 16, idesc, ks != 0);
        if (i + XST < band.n) tc_commit(&x_empty[st]);
        tc_commit(&s_full[sc]);
      }
      __syncwarp();
    }
  } else {
    const int row = tid & (ROWS - 1), part = tid / ROWS;
    const bool ok = t.l < p.L;
    const long long bl = (long long)b * p.L + (ok ? t.l : 0), grow = bl * p.H + h;
    const float expo = p.expo[bl];
    fill_weights<RPARTS>(p, wt, scores, t, ok, grow, expo);
    for (int s = part; s <= p.half; s += RPARTS) sums[s * ROWS + row] = 0.f;
    float* const sc = scores + row;
    sc[0] = 0.f, sc[ROWS] = 0.f, sc[(RS + 2) * ROWS] = 0.f;   // by all threads of a row: none waits for another's
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    const int row_bar = 2 + (warp & 3);
    const float end = last_position(p.L);
    float df = 0.f, dph = 0.f;
    for (int i = 0; i < band.n; ++i) {
      const int tm = i % NSC, k0 = band.lo + i * RS;
      cta_wait(&s_full[tm], (i / NSC) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      const bool mine = __any_sync(0xffffffffu, t.kmin < k0 + RS && t.kmax >= k0);   // the same for all threads of the rows
      uint32_t v[RCOLS];
      if (mine) {
        tmem_ld(fr.tmem + lane_off + tm * RS + part * RCOLS, v);
        tmem_ld_wait();
      }
      tc_fence_before_sync();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&s_free[tm]);
      if (!mine) continue;
      asm volatile("bar.sync %0, %1;" ::"r"(row_bar), "n"(RPARTS * 32) : "memory");
#pragma unroll
      for (int c = 0; c < RCOLS; ++c) sc[(part * RCOLS + c + 2) * ROWS] = __uint_as_float(v[c]);
      asm volatile("bar.sync %0, %1;" ::"r"(row_bar), "n"(RPARTS * 32) : "memory");
      const int2 r = tap_range(t, k0, k0 + RS, p.L);
      const int shift = 2 - k0 - MAGIC_BITS;
      // this thread's taps: ..., -4 - part, -part, part, 4 + part, ...
      int s = r.x <= -part ? -part - ((-part - r.x) & -RPARTS) : r.x <= part ? part : part + ((r.x - part + RPARTS - 1) & -RPARTS);
      auto next = [&](int u) { return RPARTS > 2 && u == -part && (part & 1) ? part : u + RPARTS; };
      while (s <= r.y) {
        const int sn = next(s), ss[2] = {s, sn};
        float dw[2], w[2], g[2];
        int as[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const bool in = j == 0 || sn <= r.y;
          as[j] = in ? abs(ss[j]) : as[0];
          const float at = tap_position(t, (float)ss[j]), pos = fminf(at, end), m = floor_magic(pos), q = pos - (m - MAGIC);
          unsigned u = (unsigned)(__float_as_int(m) + shift);
          if (u > RS + 1 || !in) u = 0;
          const float sa = sc[u * ROWS], sb1 = sc[u * ROWS + ROWS];
          w[j] = wt[as[j] * ROWS + row];
          g[j] = sums[as[j] * ROWS + row];
          dw[j] = fmaf(q, sb1 - sa, sa);
          const float dp = u == 0 || at > end ? 0.f : w[j] * (sb1 - sa);
          dph += dp;
          df = fmaf(dp, (float)ss[j], df);
        }
        if (as[0] == as[1]) dw[0] += dw[1];                // the taps -part and part, or one alone
        sums[as[0] * ROWS + row] = g[0] + dw[0];
        if (as[0] != as[1]) sums[as[1] * ROWS + row] = g[1] + dw[1];
        s = next(sn);
      }
    }
    builders_sync<RBUILDERS>();
    // per |tap|: the table's gradient in a copy of the thread's own, exponent and stride in registers
    float* tab = reinterpret_cast<float*>(sQ);
    const float f = ok ? p.freq[grow] : 0.f, sgn = f > 0.f ? 1.f : (f < 0.f ? -1.f : 0.f);
    stage_table(tab, p.kern + grow * p.K, ok, row, ROWS, part, RPARTS, p.K, p.kvec);
    if (part < 2) {
      for (int k = 0; k < p.K; ++k) tab[(p.K * (1 + part) + k) * ROWS + row] = 0.f;
    }
    builders_sync<RBUILDERS>();
    float de = 0.f, dfw = 0.f;
    if (part < 2) {                                        // two threads a row: there is room for two sums
      float* dk = tab + p.K * ROWS * (1 + part) + row;
      float a = 0.f, c = 0.f;                              // of the last tap's entry and the next (entries never fall)
      int last = -2;
      // a tap outside the sequence counts for nothing, whatever its formulas would give (a stride may be infinite, or no number)
      const int most = t.lo <= t.hi ? p.half : -1;
      for (int s = part; s <= most; s += 4) {
        float dw[2], ar[2];
        Entry e[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int u = min(s + 2 * j, p.half);
          const bool in = s + 2 * j <= p.half && ((u >= t.lo && u <= t.hi) || (-u >= t.lo && -u <= t.hi));
          ar[j] = in ? (float)u * t.f : 0.f;
          e[j] = table_entry(tab + row, ROWS, p.K, (float)u * t.f * p.inv_rec);
          dw[j] = in ? sums[u * ROWS + row] : 0.f;
          if (!in) e[j].v = e[j].slope = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float base = 1.f + ar[j] * p.invL, lg = log2f(base);
          const float dkv = dw[j] * exp2f(-expo * lg), dv = dkv * e[j].v;
          a = (e[j].lo == last ? a : e[j].lo == last + 1 ? c : 0.f) + dkv * (1.f - e[j].wh);
          c = (e[j].lo == last ? c : 0.f) + dkv * e[j].wh;
          last = e[j].lo;
          dk[e[j].lo * ROWS] = a;
          dk[(e[j].lo + 1) * ROWS] = c;
          de -= dv * (lg * 0.69314718f);
          dfw = fmaf(dkv * e[j].slope * p.inv_rec - dv * expo * p.invL / base, (float)(s + 2 * j), dfw);
        }
      }
    }
    df = (f < 0.f ? -df : df) + sgn * dfw;                 // taps were named by the stride without its sign
    if (part > 0) other[part - 1][0][row] = df, other[part - 1][1][row] = dph, other[part - 1][2][row] = de;
    builders_sync<RBUILDERS>();
    if (ok && !*abort_flag) {
      if (part == 0) {
#pragma unroll
        for (int j = 0; j < RPARTS - 1; ++j) df += other[j][0][row], dph += other[j][1][row], de += other[j][2][row];
        p.dfreq[grow] = df;
        p.dphase[grow] = dph;
        p.dexpo_h[grow] = de;
      }
      const float* d0 = tab + p.K * ROWS + row;
      const float* d1 = d0 + p.K * ROWS;
      if (p.kvec) {
        for (int k = part; k < p.K / 4; k += RPARTS)
          reinterpret_cast<float4*>(p.dkern + grow * p.K)[k] =
              make_float4(d0[(4 * k) * ROWS] + d1[(4 * k) * ROWS], d0[(4 * k + 1) * ROWS] + d1[(4 * k + 1) * ROWS],
                          d0[(4 * k + 2) * ROWS] + d1[(4 * k + 2) * ROWS], d0[(4 * k + 3) * ROWS] + d1[(4 * k + 3) * ROWS]);
      } else {
        for (int k = part; k < p.K; k += RPARTS) p.dkern[grow * p.K + k] = d0[k * ROWS] + d1[k * ROWS];
      }
    }
  }
  frame_end(fr.tmem, F::COLS, abort_flag, MMA_WARP);
}

// ------------------------------------------------------------------------------------------------ dX
// Keys that each tile of 64 queries reaches, and what the blocks of dX need of its queries, by stride in eight classes: slots 8 r to 8 r + 7
// are the queries of rank r among those of the same remainder by 8, whose rows in a swizzled tile are in different banks.
struct Query {
  float4 a, b;      // stride, phase, inv, from; to, position, exponent, packed: which query, taps inside the sequence
  int kmin, kmax;
  int2 unused;
};
static_assert(sizeof(Query) == 48, "the size that the caller allocates");
__device__ __forceinline__ int pack_query(int q, int lo, int hi) { return q | (lo + 512) << 8 | (hi + 512) << 20; }
__global__ void __launch_bounds__(STEP)
tele_band_plan_kernel(const float* __restrict__ freq, const float* __restrict__ phase, const float* __restrict__ expo, int2* __restrict__ ranges,
                      Query* __restrict__ queries, int L, int H, int half) {
  __shared__ uint32_t key[STEP];
  __shared__ int wlo[2], whi[2];
  const int nt = (L + STEP - 1) / STEP, tile = blockIdx.x % nt, h = (blockIdx.x / nt) % H, b = blockIdx.x / (nt * H);
  const int i = threadIdx.x, l = tile * STEP + i;
  Query rec;
  rec.a = rec.b = make_float4(0.f, 0.f, 0.f, __int_as_float(pack_query(i, 0, -1)));
  rec.unused = make_int2(0, 0);
  int kmin = INT_MAX, kmax = -1;
  key[i] = 0xffffffffu;
  if (l < L) {
    const long long bl = (long long)b * L + l, row = bl * H + h;
    const float f = fabsf(freq[row]), ph = phase[row];
    key[i] = __float_as_uint(f);
    const int2 in = inside(f, ph, l, L, half);
    const Taps t = make_taps(f, ph, l, in.x, in.y, L);
    kmin = t.kmin, kmax = t.kmax;
    rec.a = make_float4(f, ph, t.inv, t.from);
    rec.b = make_float4(t.to, t.lf, expo[bl], __int_as_float(pack_query(i, in.x, in.y)));
  }
  rec.kmin = kmin, rec.kmax = kmax;
  kmin = __reduce_min_sync(0xffffffffu, kmin);
  kmax = __reduce_max_sync(0xffffffffu, kmax);
  if ((i & 31) == 0) wlo[i / 32] = kmin, whi[i / 32] = kmax;
  __syncthreads();
  int rank = 0;
#pragma unroll
  for (int j = i & 7; j < STEP; j += 8) rank += (key[j] < key[i] || (key[j] == key[i] && j < i)) ? 1 : 0;
  queries[(long long)blockIdx.x * STEP + rank * 8 + (i & 7)] = rec;
  if (i == 0) ranges[blockIdx.x] = make_int2(min(wlo[0], wlo[1]), max(whi[0], whi[1]));
}

template <int N>
struct DxShape {
  static constexpr int NS = N / 64;
  static constexpr int A_BYTES = 2 * STEP * 128, Q_BYTES = NS * STEP * 128;    // one term of Wᵀ: 64 queries x 128 keys
  static constexpr uint32_t COLS = N;
  // Two blocks share a multiprocessor, which takes K up to 64 (N = 128: 43). One copy of the tables (a barrier a step more) or one stage of
  // dY is enough where the second would keep the other block off.
  static constexpr int ROOM = (233472 - 2 * 1024) / 2 - 2048 - 1024 - TERMS * A_BYTES - CELL_BYTES;   // for the two, beside the static part
  static __host__ __device__ bool fits(int stages, int tables, int K) { return stages * Q_BYTES + tables * (K + 1) * STEP * 4 <= ROOM; }
  static __host__ __device__ int stages(int K) { return fits(2, 2, K) ? 2 : 1; }
  static __host__ __device__ int tables(int K) { return !fits(1, 2, K) && fits(1, 1, K) ? 1 : 2; }
  static size_t smem(int K) { return (size_t)TERMS * A_BYTES + stages(K) * Q_BYTES + CELL_BYTES + tables(K) * (size_t)(K + 1) * STEP * 4 + 1024; }
};

// Weights of a query's taps by the formula, from its table's values at trow[k * STEP] (entry K is met with weight zero only)
struct TapWeights {
  const float* trow;
  float expo, step_entry, step_base, last_entry;
  __device__ __forceinline__ void operator()(int s, float (&w)[2]) const {
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float as = (float)abs(s + j), idx = fminf(as * step_entry, last_entry), m = floor_magic(idx);
      const float* e = trow + (__float_as_int(m) - MAGIC_BITS) * STEP;
      w[j] = fmaf(idx - (m - MAGIC), e[STEP] - e[0], e[0]) * exp2f(-expo * log2f(fmaf(as, step_base, 1.f)));
    }
  }
};
__device__ __forceinline__ TapWeights tap_weights(const BP& p, const float* trow, float expo, float f) {
  return TapWeights{trow, expo, f * p.inv_rec * (float)(p.K - 1), f * p.invL, (float)(p.K - 1)};
}
__device__ __forceinline__ Taps plan_taps(const float4& a, const float4& b, int kmin, int kmax, int l) {
  const int bits = __float_as_int(b.w);
  return Taps{a.x, a.y, a.z, a.w, b.x, b.y, l, ((bits >> 8) & 0xfff) - 512, (bits >> 20) - 512, kmin, kmax};
}

// As `gathered`, for a gradient: only the queries that sample this thread's key count. All builders together, tile by tile: the weights are
// formed as for the product, and read where they are not zero. cells: all zero, before and after; rows: 4 KB for 16 columns of the tile's
// dY, from c0 for the first half of the threads and from c0 + next for the others (none from D on). 8 x 16384 x 4 heads of 64, whole backward:
// 5.4 ms where all of dY is NaN, 31 with some NaN in every 64th row (10.3 in the gather; a thread with its own element's taps: 87).
__device__ __noinline__ void gathered_dx(const BP& p, int b, int h, int k0, const uint16_t* list, int n, long long plan, float* cells, float* tab, uint4* rows,
                                         int c0, int next, uint32_t wanted, float (&acc)[16]) {
  const int tid = threadIdx.x, slot_q = tid & (STEP - 1), seg = tid / STEP;
  float* col = cells + tid;
  const float* mine = cells + ((tid & 31) + 2) * BUILDERS + (tid & (ROWS - 1)) / SEG * STEP;     // this key's cells of the tile's queries
  const int half_row = (tid & 3) >> 1, c = c0 + half_row * next + (tid & 1) * 8;                 // what this thread copies
  const uint4* row = rows + tid / ROWS * 2;
#pragma unroll
  for (int k = 0; k < 16; ++k) acc[k] = 0.f;
  for (int i = 0; i < n && builders_any<BUILDERS>((wanted & ~nan_columns(acc)) != 0); ++i) {
    const Query* queries = p.queries + (plan + list[i]) * STEP;
    const float4 qa = queries[slot_q].a, qb = queries[slot_q].b;
    const int l = list[i] * STEP + (__float_as_int(qb.w) & 255);
    const bool ok = l < p.L;
    stage_table(tab, p.kern + (((long long)b * p.L + (ok ? l : 0)) * p.H + h) * p.K, ok, slot_q, STEP, seg, 4, p.K, p.kvec);
    if (seg == 3) tab[p.K * STEP + slot_q] = 0.f;
    const int lc = list[i] * STEP + (__float_as_int(queries[tid >> 2].b.w) & 255);
    rows[tid] = lc < p.L && c < p.D ? *reinterpret_cast<const uint4*>(p.dout + (((long long)b * p.L + lc) * p.H + h) * p.D + c) : make_uint4(0, 0, 0, 0);
    builders_sync<BUILDERS>();
    const bool any = add_taps(col, plan_taps(qa, qb, queries[slot_q].kmin, queries[slot_q].kmax, l), k0 + seg * SEG, p.L,
                              tap_weights(p, tab + slot_q, qb.z, qa.x));
    builders_sync<BUILDERS>();
    if (wanted) {
#pragma unroll 4
      for (int q = 0; q < STEP; ++q) {
        const float w = mine[q];
        if (w != 0.f) add_row(acc, w, row + q * 4);
      }
    }
    builders_sync<BUILDERS>();
    if (any) {
#pragma unroll
      for (int k = 2; k < SEG + 2; ++k) col[k * BUILDERS] = 0.f;
    }
  }
}

constexpr int MAX_TILES = 512;       // query tiles of a sequence: 32768 tokens

template <int N, typename TO>
__global__ void __launch_bounds__(THREADS, 2)
tele_band_dx_kernel(const __grid_constant__ CUtensorMap tmG, const BP p) {
  using F = DxShape<N>;
  constexpr int NBAR = 7;
  extern __shared__ __align__(1024) uint8_t raw[];
  uint8_t* sA = raw + (-smem_u32(raw) & 1023u);
  uint8_t* sG = sA + TERMS * F::A_BYTES;
  const int GST = F::stages(p.K), TABS = F::tables(p.K);
  float* cells = reinterpret_cast<float*>(sG + GST * F::Q_BYTES);
  float* tabs = cells + CELL_BYTES / 4;
  __shared__ uint64_t bars[NBAR];
  __shared__ uint16_t list[MAX_TILES];
  __shared__ int count;
  __shared__ uint32_t slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  uint64_t *a_full = bars, *a_free = bars + 1, *done = bars + 2, *g_full = bars + 3, *g_empty = bars + 5;
  int counts[NBAR];
#pragma unroll
  for (int i = 0; i < NBAR; ++i) counts[i] = i == 0 ? 8 : 1;
  const Frame fr = frame_begin(bars, NBAR, counts, &slot, abort_flag, F::COLS, p.status);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (fr.leave) {
    if (warp == 8) tmem_dealloc(fr.tmem, F::COLS);
    return;
  }
  const int nk = (p.L + ROWS - 1) / ROWS, nt = (p.L + STEP - 1) / STEP;
  const int k0 = (blockIdx.x % nk) * ROWS, h = (blockIdx.x / nk) % p.H, b = blockIdx.x / (nk * p.H);
  const long long plan = ((long long)b * p.H + h) * nt;
  if (warp == 0) {                                         // the query tiles that reach these keys, in order
    int n = 0;
    for (int j0 = 0; j0 < nt; j0 += 32) {
      const int2 r = j0 + tid < nt ? p.ranges[plan + j0 + tid] : make_int2(INT_MAX, -1);
      const bool hit = r.x < k0 + ROWS && r.y >= k0;
      const uint32_t m = __ballot_sync(0xffffffffu, hit);
      if (hit) list[n + __popc(m & ((1u << tid) - 1u))] = (uint16_t)(j0 + tid);
      n += __popc(m);
    }
    if (tid == 0) count = n;
  }
  __syncthreads();
  const int n = count;

  if (warp == 9) {
    if (elect_one_sync()) {
      int st = 0, ph = 1;
      for (int i = 0; i < n; ++i) {
        cta_wait(&g_empty[st], ph, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(&g_full[st], F::Q_BYTES);
        for (int s = 0; s < F::NS; ++s)
          tma_load_3d(sG + st * F::Q_BYTES + s * STEP * 128, &tmG, &g_full[st], h * p.D + s * 64, list[i] * STEP, b);
        if (++st == GST) st = 0, ph ^= 1;
      }
    }
  } else if (warp == 8) {
    const uint32_t idesc = make_idesc(FMT_BF16, FMT_BF16, 1, 1, 128, N);
    const uint64_t ad = make_smem_desc_sw128(smem_u32(sA), STEP * 128, 1024), gd = make_smem_desc_sw128(smem_u32(sG), STEP * 128, 1024);
    int st = 0, ph = 0;
    for (int i = 0; i < n; ++i) {
      cta_wait(&g_full[st], ph, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
      cta_wait(a_full, i & 1, abort_flag, p.status, ERR_WAIT_MISC);
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      tc_fence_after_sync();
      if (elect_one_sync()) {
#pragma unroll
        for (int term = 0; term < TERMS; ++term)
#pragma unroll
          for (int ks = 0; ks < STEP / 16; ++ks)
            tc_mma_f16(fr.tmem, ad + (term * F::A_BYTES + ks * 2048) / 16, gd + (st * F::Q_BYTES + ks * 2048) / 16, idesc, (i | term | ks) != 0);
        if (i + 1 < n) tc_commit(a_free);
        if (i + GST < n) tc_commit(&g_empty[st]);
        if (i + 1 == n) tc_commit(done);
      }
      __syncwarp();
      if (++st == GST) st = 0, ph ^= 1;
    }
  } else {
    const int slot_q = tid & (STEP - 1), seg = tid / STEP, kseg = k0 + seg * SEG;
    float* col = cells + tid;
#pragma unroll
    for (int c = 2; c < SEG + 2; ++c) col[c * BUILDERS] = 0.f;
    Query rec;
    const bool small = p.K == 16 && p.kvec;                // a quarter of a table row for each of a query's threads, loaded a step ahead
    float4 ahead;
    auto fetch = [&](int i) {
      const Query* src = p.queries + (plan + list[i]) * STEP + slot_q;
      rec.a = src->a, rec.b = src->b;
      const int2 k = *reinterpret_cast<const int2*>(&src->kmin);
      rec.kmin = k.x, rec.kmax = k.y;
      if (small) {
        const int l = list[i] * STEP + (__float_as_int(rec.b.w) & 255);
        ahead = l < p.L ? reinterpret_cast<const float4*>(p.kern + (((long long)b * p.L + l) * p.H + h) * p.K)[seg] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    if (n > 0) fetch(0);
    for (int i = 0; i < n; ++i) {
      const int bits = __float_as_int(rec.b.w), q = bits & 255, l = list[i] * STEP + q;
      const bool ok = l < p.L;
      const float expo = rec.b.z;
      float* tab = tabs + (TABS == 2 ? i & 1 : 0) * (p.K + 1) * STEP;
      if (TABS == 1 && i > 0) builders_sync<BUILDERS>();   // nobody reads the last one any more
      const float* krow = p.kern + (((long long)b * p.L + (ok ? l : 0)) * p.H + h) * p.K;
      if (small) {
        float* to = tab + 4 * seg * STEP + slot_q;
        to[0] = ahead.x, to[STEP] = ahead.y, to[2 * STEP] = ahead.z, to[3 * STEP] = ahead.w;
      } else {
        stage_table(tab, krow, ok, slot_q, STEP, seg, 4, p.K, p.kvec);
      }
      if (seg == 3) tab[p.K * STEP + slot_q] = 0.f;        // met with weight zero: the last value is entry K - 1, and nothing of the next
      const Taps t = plan_taps(rec.a, rec.b, rec.kmin, rec.kmax, l);
      if (i + 1 < n) fetch(i + 1);
      builders_sync<BUILDERS>();
      const bool any = __any_sync(0xffffffffu, add_taps(col, t, kseg, p.L, tap_weights(p, tab + slot_q, expo, t.f)));
      if (i >= 1) cta_wait(a_free, (i & 1) ^ 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
      uint8_t* dst = sA + (seg >> 1) * (STEP * 128) + q * 128;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        uint32_t o[TERMS][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float v0 = 0.f, v1 = 0.f;
          if (any) {
            float* c = col + (ch * 8 + 2 * k + 2) * BUILDERS;
            v0 = c[0], v1 = c[BUILDERS];
            c[0] = 0.f, c[BUILDERS] = 0.f;
          }
#pragma unroll
          for (int term = 0; term < TERMS; ++term) o[term][k] = take_term(v0, v1);
        }
        const int at = (((seg & 1) * 4 + ch) ^ (q & 7)) * 16;
#pragma unroll
        for (int term = 0; term < TERMS; ++term)
          *reinterpret_cast<uint4*>(dst + term * F::A_BYTES + at) = make_uint4(o[term][0], o[term][1], o[term][2], o[term][3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(a_full);
    }
    if (n > 0) cta_wait(done, 0, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
    tc_fence_after_sync();
    const int key = k0 + (tid & (ROWS - 1)), part = tid / ROWS;
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    const int cols = p.D >= 32 ? p.D / 2 : p.D, first = part * cols;
    const long long at = (((long long)b * p.L + key) * p.H + h) * p.D;
    for (int c0 = first; c0 < first + cols; c0 += 16) {
      uint32_t v[16];
      tmem_ld_32x32b_x16(fr.tmem + lane_off + c0, v);
      tmem_ld_wait();
      const bool writes = key < p.L && c0 < p.D && !*abort_flag;
      float o[16];
      uint32_t bad = 0;
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        o[k] = n > 0 ? __uint_as_float(v[k]) : 0.f;
        bad |= is_finite(o[k]) ? 0u : 1u << k;
      }
      if (!writes) bad = 0;
      if (builders_any<BUILDERS>(bad != 0)) {
        float g[16];
        gathered_dx(p, b, h, k0, list, n, plan, cells, tabs, reinterpret_cast<uint4*>(sA), c0 - first, cols, bad, g);
#pragma unroll
        for (int k = 0; k < 16; ++k)
          if (bad >> k & 1) o[k] = g[k];
      }
      if (writes) {
        if (sizeof(TO) == 2) {
          uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(p.dx) + at + c0);
#pragma unroll
          for (int k = 0; k < 2; ++k)
            dst[k] = make_uint4(pack_bf16x2(o[8 * k], o[8 * k + 1]), pack_bf16x2(o[8 * k + 2], o[8 * k + 3]), pack_bf16x2(o[8 * k + 4], o[8 * k + 5]),
                                pack_bf16x2(o[8 * k + 6], o[8 * k + 7]));
        } else {
          float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.dx) + at + c0);
#pragma unroll
          for (int k = 0; k < 4; ++k) dst[k] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
        }
      }
    }
  }
  frame_end(fr.tmem, F::COLS, abort_flag);
}

void chk(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}
// Every build is readied for the most it may ever take, once per device: a call of any size readies the others.
template <typename Kern>
void opt_in(Kern k) {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - (int)a.sharedSizeBytes);
  if (e != cudaSuccess) throw std::runtime_error(std::string("telephone: shared memory opt-in: ") + cudaGetErrorString(e));
}
void configure() {
  static PerDeviceOnce cfg;
  int dev = 0;
  if (!cfg.pending(&dev)) return;
  opt_in(tele_band_fwd_kernel<64>);
  opt_in(tele_band_fwd_kernel<128>);
  opt_in(tele_band_rows_kernel<64>);
  opt_in(tele_band_rows_kernel<128>);
  opt_in(tele_band_dx_kernel<64, bf16>);
  opt_in(tele_band_dx_kernel<64, float>);
  opt_in(tele_band_dx_kernel<128, bf16>);
  opt_in(tele_band_dx_kernel<128, float>);
  cfg.done(dev);
}
BP params(const void* x, const float* freq, const float* phase, const float* kern, const float* expo, int L, int H, int D, int K, int half,
          float max_rec, int* status) {
  BP p{};
  p.x = (const bf16*)x;
  p.freq = freq, p.phase = phase, p.kern = kern, p.expo = expo;
  p.L = L, p.H = H, p.K = K, p.half = half, p.D = D;
  p.kvec = K % 4 == 0 && (reinterpret_cast<uintptr_t>(kern) & 15) == 0;
  p.inv_rec = 1.f / max_rec, p.invL = 1.f / (float)L;
  p.status = status;
  return p;
}
CUtensorMap row_map(const void* x, int B, int L, int C) {
  return make_tmap_3d(x, TmapDtype::BF16, (uint64_t)C, (uint64_t)L, (uint64_t)B, (uint64_t)C * 2, (uint64_t)L * C * 2, 64, STEP, true);
}
}  // namespace

// Band products or one gather a tap (fused_taps.cu)? What the operands allow first, then what is faster (times: band, gather).
bool tele_band_takes(const void* x, const void* y, int B, int L, int H, int D, int K, int half, float max_rec, bool backward) {
  if (D != 16 && D != 32 && D != 64 && D != 128) return false;
  if (H * D < 64 || K < 2 || K > 64) return false;
  if (L < 128 || L > MAX_TILES * STEP || half < 1 || half > 128) return false;
  const size_t need = D == 128 ? RowsShape<128>::smem(half) : RowsShape<64>::smem(half);
  if (need > 232448 - 7168) return false;                  // beside the static part; half <= 119 or 120, 16900 tokens at the operator's own tap count
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) != 0) return false;
  if ((long long)B * H * ((L + STEP - 1) / STEP) >= (1ll << 31)) return false;
  // The band grows with the strides, of which max_rec / half is the bound that the caller knows; the gather does not.
  if (!(max_rec > 0.f) || max_rec > (D == 16 ? 22.f : D == 32 ? 32.f : 48.f) * half) return false;
  // What is left by estimates of both times in us, fitted to some 3300 calls of 128 to 20000 tokens, 1 to 16 heads, tables of 2 to 64 values, strides
  // up to 48 (10 to 12 % off, root mean square). A gather takes the taps of a row one after the other, or the time of all rows' taps where there
  // are many. So does a band with its steps of 64 keys, taps and table values: one block of 128 rows, or all of them on 148 multiprocessors
  // (a table of no multiple of four is read value by value). The faster way is missed by 1 to 2 % on average, and among calls of 300 us and more
  // by 23 % at most. Gather and band, backward: 8 x 16384 x 4 heads of 64, table of 64 10130, 4300 us; 1200 tokens, a head of 128, 33 62, 105;
  // 8 x 16384 x 4 of 16, 16 3770, 3350; 6000 x 4 of 16, 33 142, 208.
  const int w = D == 16 ? 0 : D == 32 ? 1 : D == 64 ? 2 : 3, bk = backward;
  static constexpr double START[2][4] = {{7.2, 7.9, 7.8, 9.3}, {19.5, 20.9, 21.6, 23.4}}, TAP[2][4] = {{0.46, 0.34, 0.29, 0.22}, {0.60, 0.47, 0.40, 0.265}};
  static constexpr double ROW_TAP[2][4] = {{12.4e-6, 18.7e-6, 33e-6, 61.2e-6}, {34.4e-6, 50.1e-6, 90e-6, 169e-6}};
  static constexpr double ONE_KEYS[2][4] = {{0.70, 0.70, 0.70, 1.0}, {2.15, 2.15, 2.15, 2.4}}, ALL_KEYS[2][4] = {{0.49, 0.51, 0.54, 0.72}, {1.62, 1.61, 1.69, 2.08}};
  static constexpr double ALL_TABLE[2][4] = {{0.062, 0.062, 0.066, 0.09}, {0.36, 0.38, 0.42, 0.52}};
  const double taps = 2 * half + 1, rows = (double)B * L * H, steps = fmin(128 + 2.0 * max_rec, L) / STEP, table = backward && K % 4 ? 1.8 * K : K;
  const double share = (double)B * H * ((L + ROWS - 1) / ROWS) / 148 * (!backward && half > 118 ? 1.25 : 1.0);      // (above: one block at a time)
  const double gather = START[bk][w] + fmax(TAP[bk][w] * taps, ROW_TAP[bk][w] * rows * taps);
  const double one = ONE_KEYS[bk][w] * steps + (backward ? 0.09 * taps + 0.14 * table : 0.04 * taps + 0.005 * table);
  const double all = share * (ALL_KEYS[bk][w] * steps + (backward ? 0.156 : 0.057) * taps + ALL_TABLE[bk][w] * table);
  return 1.03 * ((backward ? 27.0 : 12.5) + fmax(one, all)) < gather;
}

void tele_band_fwd(const void* x, const float* freq, const float* phase, const float* kern, const float* expo, void* out, int B, int L, int H,
                   int D, int K, int half, float max_rec, int* status, cudaStream_t s) {
  configure();
  BP p = params(x, freq, phase, kern, expo, L, H, D, K, half, max_rec, status);
  p.out = (bf16*)out;
  const CUtensorMap tm = row_map(x, B, L, H * D);
  const unsigned grid = (unsigned)(B * H * ((L + ROWS - 1) / ROWS));
  if (D == 128) tele_band_fwd_kernel<128><<<grid, THREADS, FwdShape<128>::smem(half), s>>>(tm, p);
  else tele_band_fwd_kernel<64><<<grid, THREADS, FwdShape<64>::smem(half), s>>>(tm, p);
  chk("tele_band_fwd");
}

void tele_band_bwd(const void* x, const float* freq, const float* phase, const float* kern, const float* expo, const void* dout, void* dx,
                   bool dx_f32, float* dfreq, float* dphase, float* dkern, float* dexpo_h, void* ranges, void* queries, int B, int L, int H, int D,
                   int K, int half, float max_rec, int* status, cudaStream_t s) {
  configure();
  BP p = params(x, freq, phase, kern, expo, L, H, D, K, half, max_rec, status);
  p.dout = (const bf16*)dout;
  p.dx = dx;
  p.dfreq = dfreq, p.dphase = dphase, p.dkern = dkern, p.dexpo_h = dexpo_h;
  p.kvec = p.kvec && (reinterpret_cast<uintptr_t>(dkern) & 15) == 0;
  p.ranges = (const int2*)ranges, p.queries = (const Query*)queries;
  tele_band_plan_kernel<<<(unsigned)(B * H * ((L + STEP - 1) / STEP)), STEP, 0, s>>>(freq, phase, expo, (int2*)ranges, (Query*)queries, L, H, half);
  chk("tele_band_plan");
  const unsigned grid = (unsigned)(B * H * ((L + ROWS - 1) / ROWS));
  const CUtensorMap tx = row_map(x, B, L, H * D), tg = row_map(dout, B, L, H * D);
  if (D == 128) tele_band_rows_kernel<128><<<grid, RTHREADS, RowsShape<128>::smem(half), s>>>(tx, p);
  else tele_band_rows_kernel<64><<<grid, RTHREADS, RowsShape<64>::smem(half), s>>>(tx, p);
  chk("tele_band_rows");
  if (D == 128 && dx_f32) tele_band_dx_kernel<128, float><<<grid, THREADS, DxShape<128>::smem(K), s>>>(tg, p);
  else if (D == 128) tele_band_dx_kernel<128, bf16><<<grid, THREADS, DxShape<128>::smem(K), s>>>(tg, p);
  else if (dx_f32) tele_band_dx_kernel<64, float><<<grid, THREADS, DxShape<64>::smem(K), s>>>(tg, p);
  else tele_band_dx_kernel<64, bf16><<<grid, THREADS, DxShape<64>::smem(K), s>>>(tg, p);
  chk("tele_band_dx");
}

}  // namespace b200
