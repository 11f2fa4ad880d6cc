// Flash attention forward / backward for sm_100a: every product runs on tcgen05.mma with the
// accumulators in tensor memory, operands are staged by TMA into 128B-swizzled shared memory.
//
// Masking model (the one the GPT trainers need): causal, restricted to the query's document
// (per-token doc_start / doc_end), and a sliding window counted in 128-token blocks.
//
// forward  : persistent, two 128-query tiles of one head per CTA, key/value tiles of 128; S = Q·Kᵀ (K-major
//            operands), P written back to tensor memory as the A operand of P·V, V consumed MN-major straight
//            from its [token][d] tile. The exponentials of one query tile run under the MMAs of the other.
// backward : one CTA = 128 keys x one head, looping over 64-query tiles; Sᵀ = K·Qᵀ and dPᵀ = V·dOᵀ are
//            formed transposed so that Pᵀ / dSᵀ rows are owned by one thread each and feed
//            dV += Pᵀ·dO, dK += dSᵀ·Q (TMEM-resident accumulators) and dQᵀ = Kᵀ·dSᵀ, which is
//            added into an fp32 dQ buffer by TMA reduce-add.
#include "../common/launch.h"
#include "../common/per_device.h"
#include "attn.h"

#include <algorithm>
#include <stdexcept>
#include <string>

#include "../common/ptx.cuh"
#include "../common/tmap.h"

namespace b200 {
namespace {

struct KP {
  int T, H;
  float sl2;    // softmax scale * log2(e)
  float scale;  // softmax scale
  float neg_zero = -0.f;  // addend of products that must not be fused with the sum that follows
  int window_blocks;
  int pairs = 0;          // forward: work items of two query tiles; those after them have one
  const int* doc_start;
  const int* doc_end;
  __nv_bfloat16* o; long long ld_o;
  __nv_bfloat16* dk; long long ld_dk;
  __nv_bfloat16* dv; long long ld_dv;
  float* lse;
  const float* delta;
  int* status;
};

// ------------------------------------------------------------------------------------------------
// forward
// ------------------------------------------------------------------------------------------------
// Persistent, one CTA per SM. A work item is 256 queries x one head: two 128-query tiles (a, b) that walk the same key
// tiles of 128 (a last round of few items is dealt tile by tile). Warps 0-3 / 4-7 are the softmax of tile a / b (thread = query row), warp 8 issues the MMAs, warp 9 the
// TMA loads. Tensor memory holds O and P of both tiles (P as packed bf16: the A operand of P·V, so nothing of a score ever
// touches shared memory) and the scores: two buffers at head_dim 64, one that the tiles use in turn at head_dim 128,
// where O needs the columns. A softmax warp copies its scores to registers and gives the buffer back before it starts
// the exponentials, so S of the next key tile is formed under them. P is handed over in halves of 64 keys, and the P·V of the
// first half runs under the exponentials of the second.
//
// Bound: a 128 x 128 tile costs 16384 exponentials (1024 cycles of the SFU at 16 per clock) and, at head_dim 128, 1024
// cycles of MMA; the two tiles alternate so that one tile's exponentials run under the other's MMAs. Measured, 16384
// tokens x 6 heads of 128, causal: 0.368 ms = 1120 TFLOP/s (0.799 ms with one 128-query tile per CTA and P in shared
// memory); 16 heads of 64: 0.733 ms = 750 TFLOP/s (1.168 ms).
// The output accumulator stays in tensor memory across key tiles. The running maximum is only raised when a block of 64 keys
// exceeds it by more than 2^8, so the TMEM read-scale-write of the accumulator is rare; probabilities are then at most
// 2^8, well inside bf16 / fp32 range.
// What is rounded, and where, is part of the operator: the offset of the exponents is found per 64 keys (absolute positions),
// score * scale and the subtraction of the offset are rounded one after the other, and a row sum adds its 64 terms in order.
// Other offsets are as exact, but move every probability to another place between bf16 values: that changes the gradients
// of a GPT's scalar gains, which nearly cancel, by 2 to 4 %. One offset per 128 keys, a fused multiply-add and pairwise
// sums: 0.345 and 0.677 ms.
constexpr int FQ = 128, FKV = 128;   // queries per tile, keys per tile
constexpr int FWD_THREADS = 384;
// Launched with 168 registers a thread (384 x 168 = 64512); a softmax thread holds 128 scores: 256 x 208 + 128 x 88 = 64512.
constexpr int FWD_REGS_SOFTMAX = 208, FWD_REGS_ISSUE = 88;

template <int D>
struct FwdShape {
  static constexpr int NS = D / 64;                    // 128-byte spans along the head dimension
  static constexpr int Q_BYTES = NS * FQ * 128;        // one query tile
  static constexpr int KV_BYTES = NS * FKV * 128;      // one K or V tile
  static constexpr int NST = D == 128 ? 5 : 8;         // ring of K / V tiles
  static constexpr int SMEM = 2 * Q_BYTES + NST * KV_BYTES + 256 + 1024;
};

// Key range of one query tile in units of the item's key tiles, and what its masking needs.
struct FwdTile {
  int first, last;      // key tiles [first, last); empty when the tile lies past the sequence
  int q0, ds_last;      // first query; document start of the last query
  bool skip;            // no query sees the first 64 keys of tile `first`
};
struct FwdItem {
  int h, lo, n;         // head, first key, number of key tiles of the union
  FwdTile t[2];
};
// First query of tile i of an item; p.T: there is no such tile. MIXED: items from p.pairs on are single tiles.
template <bool MIXED>
__device__ __forceinline__ int fwd_query(const KP& p, int item, int npair, int i) {
  const bool single = MIXED && item >= p.pairs;
  const int u = single ? p.pairs + (item - p.pairs) / 2 : item;
  const int tile = 2 * (npair - 1 - u / p.H) + (single ? (item - p.pairs) & 1 : i);   // late (long-context) pairs first
  return single && i == 1 ? p.T : min(tile * FQ, p.T);
}

template <bool MIXED>
__device__ __forceinline__ FwdItem fwd_item(const KP& p, int item, int npair) {
  FwdItem w;
  w.h = (MIXED && item >= p.pairs ? p.pairs + (item - p.pairs) / 2 : item) % p.H;
  int klo[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int q0 = fwd_query<MIXED>(p, item, npair, i);
    w.t[i].q0 = q0;
    klo[i] = q0 < p.T ? p.doc_start[q0] & ~63 : 0;
    w.t[i].ds_last = q0 < p.T ? p.doc_start[min(q0 + FQ, p.T) - 1] : 0;
    if (p.window_blocks > 0) klo[i] = max(klo[i], (q0 / 128 - p.window_blocks + 1) * 128);
    w.t[i].skip = klo[i] & 64;
    klo[i] = max(klo[i] & ~(FKV - 1), 0);
  }
  w.lo = klo[0];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int q0 = w.t[i].q0;
    w.t[i].first = q0 < p.T ? (klo[i] - w.lo) / FKV : 0;
    w.t[i].last = q0 < p.T ? (min(q0 + FQ, p.T) - w.lo + FKV - 1) / FKV : 0;
  }
  w.n = max(w.t[0].last, w.t[1].last);
  return w;
}
// Items are dealt to the CTAs in rounds, every second round backwards: costs fall along the list, so the sums even out.
__device__ __forceinline__ int fwd_index(int round) {
  const int g = gridDim.x, c = blockIdx.x;
  return round * g + ((round & 1) ? g - 1 - c : c);
}

template <int D, bool MIXED>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const KP p) {
  using F = FwdShape<D>;
  constexpr int NS = F::NS, NST = F::NST;
  constexpr int NSB = D == 128 ? 1 : 2;                          // score buffers
  constexpr uint32_t O_COL = 0, P_COL = 2 * D, S_COL = 2 * D + 128, TMEM_COLS = 512;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
  uint8_t* sQ = smem;
  uint8_t* sKV = sQ + 2 * F::Q_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + NST * F::KV_BYTES);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 1;
  uint64_t* s_full = bars + 2;    // [2] scores of a tile are in TMEM
  uint64_t* p_full = bars + 4;    // [2][2] the probabilities of a half of its keys are, one arrival per warp
  uint64_t* pv_done = bars + 8;   // [2][2] that half of its P·V is accumulated: P may be overwritten, O read
  uint64_t* s_free = bars + 12;   // [NSB] a score buffer has been copied to registers, one arrival per warp
  uint64_t* kv_full = bars + 14;  // [NST]
  uint64_t* kv_empty = kv_full + NST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(kv_empty + NST);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const bool poisoned = status_poisoned(p.status);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int npair = (p.T + 2 * FQ - 1) / (2 * FQ), nitem = MIXED ? p.pairs + 2 * (npair * p.H - p.pairs) : npair * p.H;

  if (tid == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&s_free[i], 4);
      for (int hf = 0; hf < 2; ++hf) { mbar_init(&p_full[2 * i + hf], 4); mbar_init(&pv_done[2 * i + hf], 1); }
    }
    for (int i = 0; i < NST; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 8) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  const bool leave = __syncthreads_or(poisoned);     // all warps or none
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  after_previous();                                  // the set-up has run under the end of the kernel before
  if (leave) {
    if (warp == 8) tmem_dealloc(tmem_base, TMEM_COLS);
    return;
  }
  if (warp >= 8) {
    reg_dealloc<FWD_REGS_ISSUE>();
    if (warp == 9 && elect_one_sync()) {
      // -------------------------------------------------------------- TMA: Q of an item, then K(0), K(1), V(0), K(2), V(1), ...
      uint32_t stage = 0, ph = 0, qph = 0;
      auto load_kv = [&](const CUtensorMap* tm, int key, int h) {
        cta_wait(&kv_empty[stage], ph ^ 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) return;
        mbar_arrive_expect_tx(&kv_full[stage], F::KV_BYTES);
        for (int s = 0; s < NS; ++s)
          tma_load_3d(sKV + stage * F::KV_BYTES + s * FKV * 128, tm, &kv_full[stage], s * 64, key, h);
        if (++stage == NST) stage = 0, ph ^= 1;
      };
      for (int r = 0, it = fwd_index(0); it < nitem; it = fwd_index(++r)) {
        const FwdItem w = fwd_item<MIXED>(p, it, npair);
        if (MIXED && w.n == 0) continue;             // the second tile of a pair that has only one
        cta_wait(q_empty, qph ^ 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) break;
        qph ^= 1;
        const int nq = w.t[1].q0 < p.T ? 2 : 1;
        mbar_arrive_expect_tx(q_full, nq * F::Q_BYTES);
        for (int i = 0; i < nq; ++i)
          for (int s = 0; s < NS; ++s)
            tma_load_3d(sQ + i * F::Q_BYTES + s * FQ * 128, &tmQ, q_full, s * 64, w.t[i].q0, w.h);
        load_kv(&tmK, w.lo, w.h);
        for (int j = 0; j < w.n; ++j) {
          if (j + 1 < w.n) load_kv(&tmK, w.lo + (j + 1) * FKV, w.h);
          load_kv(&tmV, w.lo + j * FKV, w.h);
        }
      }
    } else if (warp == 8) {
      // -------------------------------------------------------------- MMA: per key tile S_a(j+1), P·V_a(j), S_b(j+1), P·V_b(j)
      // The whole warp walks the items, so that descriptors and addresses stay in uniform registers; one elected lane
      // issues. (With a single thread in this branch every MMA was preceded by moves of its operands into them: 99
      // cycles an MMA, where 128 x 128 x 16 takes 64.)
      const uint32_t idesc_s = make_idesc(FMT_BF16, FMT_BF16, 0, 0, 128, FKV);
      const uint32_t idesc_o = make_idesc(FMT_BF16, FMT_BF16, 0, 1, 128, D);
      uint32_t stage = 0, ph = 0, qph = 0, pph[2] = {0, 0}, sph[2] = {1, 1};   // score buffers start free
      auto next_kv = [&]() {      // waits for the next tile of the ring and returns its slot
        const uint32_t slot = stage;
        cta_wait(&kv_full[slot], ph, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
        tc_fence_after_sync();
        if (++stage == NST) stage = 0, ph ^= 1;
        return slot;
      };
      // descriptors differ in their start address only (its unit is 16 bytes)
      const uint64_t qd = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), kd = make_smem_desc_sw128(smem_u32(sKV), 16, 1024);
      const uint64_t vd = make_smem_desc_sw128(smem_u32(sKV), FKV * 128, 1024);
      auto issue_s = [&](int i, uint32_t slot) {
        const int b = NSB == 1 ? 0 : i;
        cta_wait(&s_free[b], sph[b], abort_flag, p.status, ERR_WAIT_TMEM_EMPTY);
        sph[b] ^= 1;
        tc_fence_after_sync();
        const uint64_t ad = qd + i * (F::Q_BYTES / 16), bd = kd + slot * (F::KV_BYTES / 16);
        if (elect_one_sync()) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            tc_mma_f16(tmem_base + S_COL + b * 128, ad + ((ks / 4) * (FQ * 128) + (ks % 4) * 32) / 16,
                       bd + ((ks / 4) * (FKV * 128) + (ks % 4) * 32) / 16, idesc_s, ks != 0);
          tc_commit(&s_full[i]);
        }
        __syncwarp();
      };
      for (int r = 0, it = fwd_index(0); it < nitem; it = fwd_index(++r)) {
        const FwdItem w = fwd_item<MIXED>(p, it, npair);
        if (MIXED && w.n == 0) continue;             // the second tile of a pair that has only one
        cta_wait(q_full, qph, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
        qph ^= 1;
        uint32_t kslot = next_kv();
        if (__any_sync(0xffffffffu, *abort_flag)) break;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (w.t[i].first == 0 && w.t[i].last > 0) issue_s(i, kslot);
        if (elect_one_sync()) {
          tc_commit(&kv_empty[kslot]);
          if (w.n == 1) tc_commit(q_empty);
        }
        __syncwarp();
        for (int j = 0; j < w.n && !__any_sync(0xffffffffu, *abort_flag); ++j) {
          if (j + 1 < w.n) kslot = next_kv();
          const uint32_t vslot = next_kv();
          // Tile b's first scores do not wait for tile a's probabilities where they can be formed at once: with documents of one
          // or two key tiles the two tiles of an item would run one after the other. (8192 x 16 heads of 64, documents of 128:
          // 24.8 us, 31.3 without and in pairs only; later tiles issued in this order as well: 4 % slower on long documents.)
          const bool early = j + 1 == w.t[1].first && (NSB == 2 || j + 1 >= w.t[0].last);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (i == 0 && j + 1 >= w.t[0].first && j + 1 < w.t[0].last) issue_s(0, kslot);
            if ((i == 0) == early) {
              if (j + 1 >= w.t[1].first && j + 1 < w.t[1].last) issue_s(1, kslot);
              if (j + 2 == w.n && elect_one_sync()) tc_commit(q_empty);     // the item's last scores have been issued
            }
            if (j >= w.t[i].first && j < w.t[i].last) {
              const uint64_t bd = vd + vslot * (F::KV_BYTES / 16);
              const bool begin = j == w.t[i].first, skip = begin && w.t[i].skip;
#pragma unroll
              for (int hf = 0; hf < 2; ++hf) {
                cta_wait(&p_full[2 * i + hf], pph[i], abort_flag, p.status, ERR_WAIT_MISC);
                tc_fence_after_sync();
                if (elect_one_sync()) {
                  if (hf == 1 || !skip) {
#pragma unroll
                    for (int ks = 4 * hf; ks < 4 * hf + 4; ++ks)
                      tc_mma_f16_ts(tmem_base + O_COL + i * D, tmem_base + P_COL + i * 64 + ks * 8, bd + ks * (2048 / 16), idesc_o,
                                    (ks != 4 * hf || !(begin && (hf == 0 || skip))) ? 1u : 0u);
                  }
                  // the last report of an item is one that somebody waits for: none may come after the CTA has ended
                  if (hf == 1 && j + 1 == w.n && (i == 1 || w.t[1].last <= j)) tc_commit(&kv_empty[vslot]);
                  tc_commit(&pv_done[2 * i + hf]);
                }
                __syncwarp();
              }
              pph[i] ^= 1;
            }
          }
          if (j + 1 < w.n && elect_one_sync()) {
            tc_commit(&kv_empty[kslot]);
            tc_commit(&kv_empty[vslot]);
          }
          __syncwarp();
        }
        if (__any_sync(0xffffffffu, *abort_flag)) break;
      }
    }
  } else {
    reg_alloc<FWD_REGS_SOFTMAX>();
    // ---------------------------------------------------------------- softmax, epilogue
    const int i = warp >> 2;                       // tile of the pair
    const int row = tid & 127;
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16;
    const int sb = NSB == 1 ? 0 : i;
    const uint32_t s_addr = tmem_base + lane_off + S_COL + sb * 128, p_addr = tmem_base + lane_off + P_COL + i * 64;
    const uint32_t o_addr = tmem_base + lane_off + O_COL + i * D;
    uint32_t sph = 0, vph = 0;
    for (int r = 0, it = fwd_index(0); it < nitem; it = fwd_index(++r)) {
      const FwdItem w = fwd_item<MIXED>(p, it, npair);
      const FwdTile t = i == 0 ? w.t[0] : w.t[1];
      if (t.first >= t.last) continue;
      const int q = t.q0 + row;
      const bool row_ok = q < p.T;
      const int ds = row_ok ? p.doc_start[q] : q;
      float m_run = -INFINITY, l = 0.f;
      for (int j = t.first; j < t.last; ++j) {
        cta_wait(&s_full[i], sph, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
        sph ^= 1;
        tc_fence_after_sync();
        const int kvb = w.lo + j * FKV;
        float v[FKV];
        {
          uint32_t u[FKV / 32][32];
#pragma unroll
          for (int c = 0; c < FKV / 32; ++c) tmem_ld_32x32b_x32(s_addr + c * 32, u[c]);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < FKV; ++c) v[c] = __uint_as_float(u[c / 32][c % 32]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if ((tid & 31) == 0) mbar_arrive(&s_free[sb]);
        // the maximum is taken before the scale is applied where that gives the same value
        if (!(p.sl2 > 0.f)) {
#pragma unroll
          for (int c = 0; c < FKV; ++c) v[c] = __fmul_rn(v[c], p.sl2);
        }
        const float mul = p.sl2 > 0.f ? p.sl2 : 1.f;
        if (kvb + FKV - 1 > t.q0 || kvb < t.ds_last) {
          const int hi = q - kvb, lo = ds - kvb;     // visible columns [lo, hi]
#pragma unroll
          for (int c = 0; c < FKV; ++c) v[c] = (c >= lo && c <= hi) ? v[c] : -INFINITY;
        }
        const uint64_t mul2 = f2_pack(mul, mul), negz = f2_pack(p.neg_zero, p.neg_zero);
        auto maximum = [&](int hf) {
          const float* x = v + 64 * hf;
          float mx[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
          for (int c = 4; c < 60; c += 8) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mx[k] = fmaxf(mx[k], fmaxf(x[c + k], x[c + 4 + k]));
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) mx[k] = fmaxf(mx[k], x[60 + k]);
          return __fmul_rn(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), mul);   // never part of a fused operation
        };
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const float mblk = maximum(hf);
          const bool raise = mblk > m_run + 8.f;
          const bool rescale = raise && m_run != -INFINITY;   // before, the accumulator is zero
          const float alpha = raise ? exp2f(m_run - mblk) : 1.f;
          if (raise) m_run = mblk;
          const float m_use = m_run == -INFINITY ? 0.f : m_run;
          if (hf == 0 && j > t.first) {              // P and O are free once the previous P·V is done
            cta_wait(&pv_done[2 * i + 1], vph ^ 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
            tc_fence_after_sync();
          }
          const uint64_t negm = f2_pack(-m_use, -m_use);
          float sum = 0.f;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t pk[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) {
              const int at = hf * 64 + c * 32 + 2 * k;
              float x, y;
              f2_unpack(f2_add(f2_fma(f2_pack(v[at], v[at + 1]), mul2, negz), negm), x, y);
              x = exp2f(x), y = exp2f(y);
              sum += x;
              sum += y;
              pk[k] = pack_bf16x2(x, y);
            }
            tmem_st_32x32b_x16(p_addr + hf * 32 + c * 16, pk);
          }
          if (__any_sync(0xffffffffu, rescale)) {    // rare (and kept small): bring this warp's accumulator rows to the new maximum
            if (hf == 1) {                           // (the first half's products among them)
              cta_wait(&pv_done[2 * i], vph, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
              tc_fence_after_sync();
            }
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              uint32_t o[32];
              tmem_ld_32x32b_x32(o_addr + c * 32, o);
              tmem_ld_wait();
#pragma unroll
              for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
              tmem_st_32x32b_x32(o_addr + c * 32, o);
            }
          }
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if ((tid & 31) == 0) mbar_arrive(&p_full[2 * i + hf]);
          l = fmaf(l, alpha, sum);
        }
        vph ^= 1;
      }
      cta_wait(&pv_done[2 * i + 1], vph ^ 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* orow = p.o + (long long)q * p.ld_o + w.h * D;
#pragma unroll
      for (int c = 0; c < D / 32; ++c) {
        uint32_t v[32];
        tmem_ld_32x32b_x32(o_addr + c * 32, v);
        tmem_ld_wait();
        if (row_ok) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint4 u = make_uint4(pack_bf16x2(__uint_as_float(v[8 * k]) * inv, __uint_as_float(v[8 * k + 1]) * inv),
                                 pack_bf16x2(__uint_as_float(v[8 * k + 2]) * inv, __uint_as_float(v[8 * k + 3]) * inv),
                                 pack_bf16x2(__uint_as_float(v[8 * k + 4]) * inv, __uint_as_float(v[8 * k + 5]) * inv),
                                 pack_bf16x2(__uint_as_float(v[8 * k + 6]) * inv, __uint_as_float(v[8 * k + 7]) * inv));
            reinterpret_cast<uint4*>(orow + c * 32)[k] = u;
          }
        }
      }
      if (row_ok) p.lse[(long long)w.h * p.T + q] = m_run + log2f(l);
    }
  }
  __syncwarp();
  if (*abort_flag && tid == 0) {  // let loads still in flight land before shared memory is released
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 8) tmem_dealloc(tmem_base, TMEM_COLS);
}

// ------------------------------------------------------------------------------------------------
// delta[h][t] = sum_d O[t,h,d] * dO[t,h,d]
// ------------------------------------------------------------------------------------------------
template <int D>
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, long long ld_o,
                                  const __nv_bfloat16* __restrict__ d_o, long long ld_do, float* __restrict__ delta,
                                  int T, int H) {
  // one warp per (t, h)
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= T * H) return;
  const int t = gw / H, h = gw % H;
  const __nv_bfloat16* a = o + (long long)t * ld_o + h * D;
  const __nv_bfloat16* b = d_o + (long long)t * ld_do + h * D;
  float acc = 0.f;
  for (int i = lane * 2; i < D; i += 64) {
    float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(a + i));
    float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(b + i));
    acc += x.x * y.x + x.y * y.y;
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (lane == 0) delta[(long long)h * T + t] = acc;
}

// Same with 16-byte loads: D / 8 adjacent lanes own a row, a warp covers 32 / (D / 8) rows (needs 16-byte aligned rows).
template <int D>
__global__ void attn_delta_vec_kernel(const __nv_bfloat16* __restrict__ o, long long ld_o,
                                      const __nv_bfloat16* __restrict__ d_o, long long ld_do,
                                      float* __restrict__ delta, int T, int H) {
  let_next_start();
  after_previous();
  o = fresh(o), d_o = fresh(d_o);
  constexpr int LPR = D / 8;
  const long long row = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
  const int sub = threadIdx.x % LPR;
  float acc = 0.f;
  int t = 0, h = 0;
  const bool on = row < (long long)T * H;
  if (on) {
    t = (int)(row / H), h = (int)(row % H);
    const uint4 ua = *reinterpret_cast<const uint4*>(o + (long long)t * ld_o + h * D + sub * 8);
    const uint4 ub = *reinterpret_cast<const uint4*>(d_o + (long long)t * ld_do + h * D + sub * 8);
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&ua);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&ub);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pb[i]);
      acc = fmaf(x.x, y.x, fmaf(x.y, y.y, acc));
    }
  }
#pragma unroll
  for (int s = LPR / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (on && sub == 0) delta[(long long)h * T + t] = acc;
}

// ------------------------------------------------------------------------------------------------
// backward
// ------------------------------------------------------------------------------------------------
// Head_dim 128. Warps 0-7 compute (warps w and w+4 share TMEM lane quarter (w & 3) and split the columns of S and dP), four warps
// drain dQ, one issues the MMAs, one the TMA loads. The tensor pipe runs the products in issue order, per query tile `it`:
//   S, dP of tile it+1   as soon as every warp has copied tile it's S / dP out of TMEM: under the exponentials of tile it;
//   dQ of tile it        right behind the exponentials, on its own barrier, drained by warps that do nothing else;
//   dV, dK of tile it    their barrier is waited for before P / dS are overwritten.
// Pᵀ and dSᵀ are the A operands of dV / dK from tensor memory; dSᵀ is in shared memory too, for dQ.
// Bound: shared memory, 288 KB a tile of 128 keys x 64 queries (S, dP and dQ read 6 KB of operands per MMA, dQ is staged, Q and dO
// arrive): 2300 cycles at 128 bytes a clock, of 2600. Measured, 16384 tokens causal, 6 heads: 0.965 ms = 1070 TFLOP/s (1.28 ms with dQ
// drained by the compute warps, whose copy, fence and barrier were 900 cycles a tile with nothing to run under them, and shared
// memory behind generic addresses); documents of 1024, 49152 tokens: 0.360 ms (0.433 ms). Four warps a lane quarter: 0.98 ms.
constexpr int BWD_PARTS = 2, BWD_WARPS = 4 * BWD_PARTS, BWD_COMPUTE = 32 * BWD_WARPS, BWD_THREADS = BWD_COMPUTE + 128 + 64;
constexpr int BWD64_QB = 6;
constexpr int BWD_MMA = BWD_WARPS + 4, BWD_TMA = BWD_MMA + 1;   // the warps after the four that drain dQ

__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd128_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdQ, const KP p) {
  constexpr int D = 128, NS = D / 64;
  constexpr int BKV = 128, BQ = 64;
  constexpr int KV_BYTES = NS * BKV * 128;  // K or V tile
  constexpr int Q_BYTES = NS * BQ * 128;    // Q or dO tile
  constexpr int DS_BYTES = BKV * 128;       // dSᵀ: 128 key rows x 64 queries
  constexpr int DQ_BYTES = BQ * D * 4;      // fp32 staging of one dQ tile
  constexpr uint32_t ST_COL = 0, DPT_COL = 64, DV_COL = 128, DK_COL = 128 + D, DQT_COL = 128 + 2 * D;
  constexpr uint32_t P16_COL = DQT_COL + 64, DS16_COL = P16_COL + 32;   // Pᵀ and dSᵀ as packed bf16: A operands of dV, dK
  constexpr uint32_t TMEM_COLS = 512;
  static_assert(DS16_COL + 32 <= TMEM_COLS, "tensor memory");

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
  uint8_t* sK = smem;
  uint8_t* sV = sK + KV_BYTES;
  constexpr int NQB = 3;              // Q / dO buffers
  uint8_t* sQ = sV + KV_BYTES;
  uint8_t* sdO = sQ + NQB * Q_BYTES;
  uint8_t* sdST = sdO + NQB * Q_BYTES;
  float* sdQ = reinterpret_cast<float*>(sdST + DS_BYTES);
  float2* s_ld_all = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(sdQ) + DQ_BYTES);  // [2][64] {lse, delta}, double-buffered over query tiles
  int* s_ds_all = reinterpret_cast<int*>(s_ld_all + 2 * BQ);      // [2][64] document start of each query
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_ds_all + 2 * BQ);
  uint64_t* bar_kv = bars;
  uint64_t* bar_m1 = bars + 1;     // S / dP of a tile are in TMEM
  uint64_t* bar_m2 = bars + 2;     // dV / dK of a tile are accumulated: P and dS may be overwritten
  uint64_t* bar_dq = bars + 3;     // dQ of a tile is in TMEM
  uint64_t* bar_sfree = bars + 4;  // S / dP of a tile are in registers, one arrival per compute warp
  uint64_t* bar_pds = bars + 5;    // P / dS of a tile are in place, one arrival per compute warp
  uint64_t* bar_dqfree = bars + 6; // dQ of a tile is in registers, one arrival per drain warp
  uint64_t* bar_q = bars + 7;      // [3] a Q / dO buffer is full
  uint64_t* bar_qe = bars + 10;    // [3] and empty again
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 13);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  after_previous();
  const bool poisoned = status_poisoned(p.status);
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int quarter = warp & 3;
  const int part = (warp >> 2) & (BWD_PARTS - 1);   // its columns: CQ queries, D / BWD_PARTS of the head dimension
  constexpr int CQ = BQ / BWD_PARTS, CD = D / BWD_PARTS;
  const int r = quarter * 32 + lane;  // accumulator row owned by this thread
  const int jb = blockIdx.x;
  const int h = blockIdx.y;
  const int kv0 = jb * BKV;
  const int kv = kv0 + r;

  // query range that can see any key of this tile
  const int last_kv = min(kv0 + BKV, p.T) - 1;
  int q_hi = p.doc_end[last_kv];
  if (p.window_blocks > 0) q_hi = min(q_hi, (jb + p.window_blocks) * 128);
  q_hi = min(q_hi, p.T);
  const int q_lo = kv0;
  const int ntile = (q_hi - q_lo + BQ - 1) / BQ;
  // per-query scalars (lse, delta, document start) are loaded two tiles ahead and stored one tile ahead; those of the
  // first two tiles are on their way during the set-up
  auto scalars = [&](int q0, float2& ld, int& ds) {
    const int qq = q0 + tid;
    const bool okq = tid < BQ && qq < p.T;
    ld = make_float2(okq ? p.lse[(long long)h * p.T + qq] : INFINITY, okq ? p.delta[(long long)h * p.T + qq] : 0.f);
    ds = okq ? p.doc_start[qq] : 0x7fffffff;
  };
  float2 nxt_ld, far_ld;
  int nxt_ds, far_ds;
  scalars(q_lo, nxt_ld, nxt_ds);
  scalars(q_lo + BQ, far_ld, far_ds);

  if (tid == 0) {
    mbar_init(bar_kv, 1);
    mbar_init(bar_m1, 1);
    mbar_init(bar_m2, 1);
    mbar_init(bar_dq, 1);
    mbar_init(bar_sfree, BWD_WARPS);
    mbar_init(bar_pds, BWD_WARPS);
    mbar_init(bar_dqfree, 4);
    for (int i = 0; i < NQB; ++i) { mbar_init(&bar_q[i], 1); mbar_init(&bar_qe[i], 1); }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == BWD_MMA) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  const bool leave = __syncthreads_or(poisoned);     // all warps or none
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  if (leave) {
    if (warp == BWD_MMA) tmem_dealloc(tmem_base, TMEM_COLS);
    return;
  }
  const uint32_t lane_off = uint32_t(quarter * 32) << 16;

  if (warp == BWD_TMA) {
    if (elect_one_sync()) {
      mbar_arrive_expect_tx(bar_kv, 2 * KV_BYTES);
      for (int s = 0; s < NS; ++s) {
        tma_load_3d(sK + s * BKV * 128, &tmK, bar_kv, s * 64, kv0, h);
        tma_load_3d(sV + s * BKV * 128, &tmV, bar_kv, s * 64, kv0, h);
      }
      for (int it = 0; it < ntile; ++it) {
        const int buf = it % NQB;
        if (it >= NQB) cta_wait(&bar_qe[buf], (it / NQB - 1) & 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(&bar_q[buf], 2 * Q_BYTES);
        for (int s = 0; s < NS; ++s) {
          tma_load_3d(sQ + buf * Q_BYTES + s * BQ * 128, &tmQ, &bar_q[buf], s * 64, q_lo + it * BQ, h);
          tma_load_3d(sdO + buf * Q_BYTES + s * BQ * 128, &tmdO, &bar_q[buf], s * 64, q_lo + it * BQ, h);
        }
      }
    }
  } else if (warp == BWD_MMA) {
    // the whole warp walks the tiles and one elected lane issues: operands stay in uniform registers (see the forward)
    const uint32_t idesc_st = make_idesc(FMT_BF16, FMT_BF16, 0, 0, 128, BQ);   // K·Qᵀ, V·dOᵀ
    const uint32_t idesc_dv = make_idesc(FMT_BF16, FMT_BF16, 0, 1, 128, D);    // Pᵀ·dO, dSᵀ·Q   (B MN-major)
    const uint32_t idesc_dq = make_idesc(FMT_BF16, FMT_BF16, 1, 1, 128, BQ);   // Kᵀ·dSᵀ         (A, B MN-major)
    // descriptors differ in their start address only (its unit is 16 bytes)
    const uint64_t kd = make_smem_desc_sw128(smem_u32(sK), 16, 1024), vd = make_smem_desc_sw128(smem_u32(sV), 16, 1024);
    const uint64_t qd = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), dod = make_smem_desc_sw128(smem_u32(sdO), 16, 1024);
    const uint64_t kmn = make_smem_desc_sw128(smem_u32(sK), BKV * 128, 1024), dsmn = make_smem_desc_sw128(smem_u32(sdST), BKV * 128, 1024);
    const uint64_t qmn = make_smem_desc_sw128(smem_u32(sQ), BQ * 128, 1024), domn = make_smem_desc_sw128(smem_u32(sdO), BQ * 128, 1024);
    auto issue_s_dp = [&](int it) {
      const int buf = it % NQB;
      cta_wait(&bar_q[buf], (it / NQB) & 1, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
      tc_fence_after_sync();
      const uint64_t off = buf * (Q_BYTES / 16);
      if (elect_one_sync()) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint64_t bd = qd + off + ((ks / 4) * (BQ * 128) + (ks % 4) * 32) / 16;
          tc_mma_f16(tmem_base + ST_COL, kd + ((ks / 4) * (BKV * 128) + (ks % 4) * 32) / 16, bd, idesc_st, ks != 0);
        }
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint64_t bd = dod + off + ((ks / 4) * (BQ * 128) + (ks % 4) * 32) / 16;
          tc_mma_f16(tmem_base + DPT_COL, vd + ((ks / 4) * (BKV * 128) + (ks % 4) * 32) / 16, bd, idesc_st, ks != 0);
        }
        tc_commit(bar_m1);
      }
      __syncwarp();
    };
    cta_wait(bar_kv, 0, abort_flag, p.status, ERR_WAIT_SMEM_FULL);     // also when no query tile reads them
    tc_fence_after_sync();
    if (ntile > 0) issue_s_dp(0);
    for (int it = 0; it < ntile; ++it) {
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      const int buf = it % NQB;
      if (it + 1 < ntile) {
        cta_wait(bar_sfree, it & 1, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY);
        tc_fence_after_sync();
        issue_s_dp(it + 1);
      }
      cta_wait(bar_pds, it & 1, abort_flag, p.status, ERR_WAIT_MISC);
      if (it > 0) cta_wait(bar_dqfree, (it - 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY);
      tc_fence_after_sync();
      const uint64_t off = buf * (Q_BYTES / 16);
      if (elect_one_sync()) {
#pragma unroll
        for (int ks = 0; ks < BKV / 16; ++ks)  // dQᵀ = Kᵀ · dSᵀ
          tc_mma_f16(tmem_base + DQT_COL, kmn + ks * (2048 / 16), dsmn + ks * (2048 / 16), idesc_dq, ks != 0);
        tc_commit(bar_dq);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks) { // dV += Pᵀ · dO
          const uint64_t bd = domn + off + ks * (2048 / 16);
          tc_mma_f16_ts(tmem_base + DV_COL, tmem_base + P16_COL + ks * 8, bd, idesc_dv, (it | ks) != 0);
        }
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks) { // dK += dSᵀ · Q
          const uint64_t bd = qmn + off + ks * (2048 / 16);
          tc_mma_f16_ts(tmem_base + DK_COL, tmem_base + DS16_COL + ks * 8, bd, idesc_dv, (it | ks) != 0);
        }
        tc_commit(&bar_qe[buf]);
        tc_commit(bar_m2);        // the last one is waited for: no report may come after the CTA has ended
      }
      __syncwarp();
    }
  } else if (warp >= BWD_WARPS) {
    // dQᵀ of a tile (row = head-dim index r) -> staging[q][r], then one bulk reduce-add into the fp32 accumulator (reductions
    // issued element by element from registers measured 25 % slower). Warps of their own: in the compute warps this copy, its
    // fence and its barrier were 900 of 2850 cycles a tile, with nothing to run under them.
    const bool issue_red = tid == BWD_COMPUTE;
    auto drain_sync = [] { asm volatile("bar.sync 2, 128;" ::: "memory"); };
    for (int it = 0; it < ntile; ++it) {
      cta_wait(bar_dq, it & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      uint32_t v[2][32];
      if (r < D) {
        tmem_ld_32x32b_x32(tmem_base + lane_off + DQT_COL, v[0]);
        tmem_ld_32x32b_x32(tmem_base + lane_off + DQT_COL + 32, v[1]);
        tmem_ld_wait();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_dqfree);
      if (issue_red) tma_store_wait_read<0>();   // the last reduce-add has drained the staging buffer
      drain_sync();
      if (r < D) {
#pragma unroll
        for (int i = 0; i < BQ; ++i) sdQ[i * D + r] = __uint_as_float(v[i / 32][i % 32]) * p.scale;
      }
      fence_proxy_async_smem();
      drain_sync();                              // the staged tile is complete
      if (issue_red) {
        tma_reduce_add_3d(&tmdQ, sdQ, 0, q_lo + it * BQ, h);
        tma_store_commit();
      }
    }
    if (issue_red) tma_store_wait_read<0>();     // shared memory may be given back
  } else {
    auto compute_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(BWD_COMPUTE) : "memory"); };
    if (tid < BQ) {
      s_ld_all[tid] = nxt_ld;
      s_ds_all[tid] = nxt_ds;
    }
    compute_sync();
    for (int it = 0; it < ntile; ++it) {
      const int qt0 = q_lo + it * BQ;
      const float2* s_ld = s_ld_all + (it & 1) * BQ;
      const int* s_ds = s_ds_all + (it & 1) * BQ;
      nxt_ld = far_ld, nxt_ds = far_ds;
      if (it + 2 < ntile) scalars(qt0 + 2 * BQ, far_ld, far_ds);
      cta_wait(bar_m1, it & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      uint32_t sv[CQ], dv_[CQ];
      tmem_ld_32x32b_x32(tmem_base + lane_off + ST_COL + part * CQ, sv);
      tmem_ld_32x32b_x32(tmem_base + lane_off + DPT_COL + part * CQ, dv_);
      tmem_ld_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_sfree);

      // masks are needed only where the tile touches the causal diagonal, a document boundary or the sequence end
      const bool need_mask = (qt0 < kv0 + BKV) || (s_ds[BQ - 1] > kv0) || (kv0 + BKV > p.T) || (qt0 + BQ > p.T);
      // probabilities, then the mask in a loop of its own: a branch per element would serialise the latencies of the others
#pragma unroll
      for (int i = 0; i < CQ; i += 2) {
        const float4 ld = *reinterpret_cast<const float4*>(&s_ld[part * CQ + i]);   // {lse, delta} of two queries
        sv[i] = __float_as_uint(exp2f(fmaf(__uint_as_float(sv[i]), p.sl2, -ld.x)));
        sv[i + 1] = __float_as_uint(exp2f(fmaf(__uint_as_float(sv[i + 1]), p.sl2, -ld.z)));
        dv_[i] = __float_as_uint(__uint_as_float(dv_[i]) - ld.y);
        dv_[i + 1] = __float_as_uint(__uint_as_float(dv_[i + 1]) - ld.w);
      }
      if (need_mask) {
        // queries [lo, hi) of this thread's see its key: from the key itself to the last query whose document has begun at
        // or before it (document starts never fall, so that is a search for the first later one)
        const int lo = kv - qt0 - part * CQ;
        int hi = CQ;
        if (s_ds[part * CQ + CQ - 1] > kv) {
          hi = 0;
#pragma unroll
          for (int step = CQ / 2; step > 0; step >>= 1)
            if (s_ds[part * CQ + hi + step - 1] <= kv) hi += step;
        }
        if (kv >= p.T) hi = 0;
#pragma unroll
        for (int i = 0; i < CQ; ++i)
          if (i < lo || i >= hi) sv[i] = 0u;
      }
      uint32_t pp[CQ / 2], dd[CQ / 2];
#pragma unroll
      for (int i = 0; i < CQ; i += 2) {
        const float p0 = __uint_as_float(sv[i]), p1 = __uint_as_float(sv[i + 1]);
        pp[i >> 1] = pack_bf16x2(p0, p1);
        dd[i >> 1] = pack_bf16x2(p0 * __uint_as_float(dv_[i]), p1 * __uint_as_float(dv_[i + 1]));
      }
      if (tid < BQ && it + 1 < ntile) {
        s_ld_all[((it + 1) & 1) * BQ + tid] = nxt_ld;
        s_ds_all[((it + 1) & 1) * BQ + tid] = nxt_ds;
      }
      compute_sync();                            // the next tile's scalars are visible
      if (it > 0) {
        cta_wait(bar_m2, (it - 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);   // P / dS of the last tile are free
        tc_fence_after_sync();
      }
      tmem_st_32x32b_x16(tmem_base + lane_off + P16_COL + part * (CQ / 2), pp);
      tmem_st_32x32b_x16(tmem_base + lane_off + DS16_COL + part * (CQ / 2), dd);
#pragma unroll
      for (int j = 0; j < CQ / 8; ++j) {
        const int at = r * 128 + (((part * (CQ / 8) + j) ^ (r & 7)) << 4);
        *reinterpret_cast<uint4*>(sdST + at) = make_uint4(dd[4 * j], dd[4 * j + 1], dd[4 * j + 2], dd[4 * j + 3]);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_pds);
    }
    // final: dV, dK rows; each warp writes its part of the head dimension
    if (ntile > 0) cta_wait(bar_m2, (ntile - 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
    tc_fence_after_sync();
    __nv_bfloat16* dvrow = p.dv + (long long)kv * p.ld_dv + h * D + part * CD;
    __nv_bfloat16* dkrow = p.dk + (long long)kv * p.ld_dk + h * D + part * CD;
    if (ntile > 0) {
      auto write = [&](uint32_t col, __nv_bfloat16* row, float mul) {
#pragma unroll
        for (int c = 0; c < CD; c += 16) {
          uint32_t v[16];
          tmem_ld_32x32b_x16(tmem_base + lane_off + col + part * CD + c, v);
          tmem_ld_wait();
          if (kv < p.T) {
#pragma unroll
            for (int j = 0; j < 2; ++j)
              reinterpret_cast<uint4*>(row + c)[j] =
                  make_uint4(pack_bf16x2(__uint_as_float(v[8 * j]) * mul, __uint_as_float(v[8 * j + 1]) * mul),
                             pack_bf16x2(__uint_as_float(v[8 * j + 2]) * mul, __uint_as_float(v[8 * j + 3]) * mul),
                             pack_bf16x2(__uint_as_float(v[8 * j + 4]) * mul, __uint_as_float(v[8 * j + 5]) * mul),
                             pack_bf16x2(__uint_as_float(v[8 * j + 6]) * mul, __uint_as_float(v[8 * j + 7]) * mul));
          }
        }
      };
      write(DV_COL, dvrow, 1.f);
      write(DK_COL, dkrow, p.scale);
    } else if (kv < p.T) {
      // no query tile attends this key tile: its gradients are zero (the caller does not pre-zero dk / dv)
#pragma unroll
      for (int j = 0; j < CD / 8; ++j) {
        reinterpret_cast<uint4*>(dvrow)[j] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(dkrow)[j] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
  __syncwarp();
  if (tid == 0) {
    if (*abort_flag) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == BWD_MMA) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Head_dim 64. Two groups of four compute warps take the query tiles in turn (warp w of a group: TMEM lane quarter w & 3, thread = key),
// four warps drain dQ, one issues the MMAs, one the TMA loads. Tensor memory holds three buffers of 128 columns, tile it in buffer
// it % 3: its S | dP, then Pᵀ | dSᵀ as packed bf16 (A operands of dV, dK) over S and dQᵀ over dP; a buffer is free again when
// the tile's products are done (they run in issue order) and its dQᵀ has been copied. So the scores of a group's next tile are
// ready when it has finished one, and it waits for nothing else. dSᵀ is in shared memory too, for dQ.
// The tensor pipe runs, per query tile `it`: S, dP of tile it+2; then, behind the group that has tile it, dQ, dV and dK of tile it.
// Measured, 16384 tokens causal, 16 heads: 1.76 ms = 780 TFLOP/s (3.00 ms with all eight warps on one tile and its scores behind
// the copy of its own; 2.00 with two buffers; 2.13 with one group and K and V, as A operands, in tensor memory); documents of about
// 5000: 0.67 ms (1.07), of 700, 20011 tokens: 0.28 ms (0.39). A group needs some 2100 cycles a tile (64 exponentials a thread, one warp
// a scheduler), two tiles at a time.
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd64_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const __grid_constant__ CUtensorMap tmdQ, const KP p) {
  constexpr int D = 64;
  constexpr int BKV = 128, BQ = 64;
  constexpr int KV_BYTES = BKV * 128;       // K or V tile
  constexpr int Q_BYTES = BQ * 128;         // Q or dO tile
  constexpr int DS_BYTES = BKV * 128;       // dSᵀ: 128 key rows x 64 queries, one for each buffer
  constexpr int DQ_BYTES = BQ * D * 4;      // fp32 staging of one dQ tile
  constexpr int NB = 3;                     // buffers in tensor memory, and of dSᵀ
  constexpr uint32_t BUF = 128, DP_COL = 64, P16_COL = 0, DS16_COL = 32, DQT_COL = 64;     // in a buffer
  constexpr uint32_t DV_COL = NB * BUF, DK_COL = DV_COL + D;
  constexpr uint32_t TMEM_COLS = 512;
  static_assert(DK_COL + D <= TMEM_COLS, "tensor memory");

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
  uint8_t* sK = smem;
  uint8_t* sV = sK + KV_BYTES;
  constexpr int NQB = BWD64_QB;       // Q / dO buffers: tiles it to it+2 are in use, the others on their way
  uint8_t* sQ = sV + KV_BYTES;
  uint8_t* sdO = sQ + NQB * Q_BYTES;
  uint8_t* sdST = sdO + NQB * Q_BYTES;
  float* sdQ = reinterpret_cast<float*>(sdST + NB * DS_BYTES);
  float2* s_ld_all = reinterpret_cast<float2*>(reinterpret_cast<uint8_t*>(sdQ) + DQ_BYTES);  // [group][2][64] {lse, delta}, for its tiles in turn
  int* s_ds_all = reinterpret_cast<int*>(s_ld_all + 4 * BQ);      // [group][2][64] document start of each query
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_ds_all + 4 * BQ);
  uint64_t* bar_m1 = bars;              // [NB] S / dP of a tile are in TMEM
  uint64_t* bar_pds = bars + NB;        // [NB] P / dS of a tile are in place, one arrival per warp of the group
  uint64_t* bar_dq = bars + 2 * NB;     // [NB] dQ of a tile is in TMEM
  uint64_t* bar_dqfree = bars + 3 * NB; // [NB] and in registers, one arrival per drain warp
  uint64_t* bar_q = bars + 4 * NB;      // [NQB] a Q / dO buffer is full
  uint64_t* bar_qe = bar_q + NQB;       // [NQB] and empty again
  uint64_t* bar_kv = bar_qe + NQB;
  uint64_t* bar_done = bar_kv + 1;      // dV and dK are complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  after_previous();
  const bool poisoned = status_poisoned(p.status);
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const int quarter = warp & 3;
  const int group = (warp >> 2) & 1;
  const int r = quarter * 32 + lane;  // accumulator row of this thread
  const int jb = blockIdx.x;
  const int h = blockIdx.y;
  const int kv0 = jb * BKV;
  const int kv = kv0 + r;

  // query range that can see any key of this tile
  const int last_kv = min(kv0 + BKV, p.T) - 1;
  int q_hi = p.doc_end[last_kv];
  if (p.window_blocks > 0) q_hi = min(q_hi, (jb + p.window_blocks) * 128);
  q_hi = min(q_hi, p.T);
  const int q_lo = kv0;
  const int ntile = (q_hi - q_lo + BQ - 1) / BQ;
  // per-query scalars (lse, delta, document start) of a group's next tile are loaded while it works on a tile; those of the first are
  // on their way during the set-up
  float2 nxt_ld;
  int nxt_ds;
  auto scalars = [&](int it) {
    const int qq = q_lo + it * BQ + r;
    const bool okq = r < BQ && it < ntile && qq < p.T;
    nxt_ld = make_float2(okq ? p.lse[(long long)h * p.T + qq] : INFINITY, okq ? p.delta[(long long)h * p.T + qq] : 0.f);
    nxt_ds = okq ? p.doc_start[qq] : 0x7fffffff;
  };
  scalars(group);

  if (tid == 0) {
    for (int i = 0; i < NB; ++i) {
      mbar_init(&bar_m1[i], 1);
      mbar_init(&bar_pds[i], 4);
      mbar_init(&bar_dq[i], 1);
      mbar_init(&bar_dqfree[i], 4);
    }
    for (int i = 0; i < NQB; ++i) { mbar_init(&bar_q[i], 1); mbar_init(&bar_qe[i], 1); }
    mbar_init(bar_kv, 1);
    mbar_init(bar_done, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == BWD_MMA) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  const bool leave = __syncthreads_or(poisoned);     // all warps or none
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  if (leave) {
    if (warp == BWD_MMA) tmem_dealloc(tmem_base, TMEM_COLS);
    return;
  }
  const uint32_t lane_off = uint32_t(quarter * 32) << 16;

  if (warp == BWD_TMA) {
    if (elect_one_sync()) {
      mbar_arrive_expect_tx(bar_kv, 2 * KV_BYTES);
      tma_load_3d(sK, &tmK, bar_kv, 0, kv0, h);
      tma_load_3d(sV, &tmV, bar_kv, 0, kv0, h);
      for (int it = 0; it < ntile; ++it) {
        const int buf = it % NQB;
        if (it >= NQB) cta_wait(&bar_qe[buf], (it / NQB - 1) & 1, abort_flag, p.status, ERR_WAIT_SMEM_EMPTY);
        if (*abort_flag) break;
        mbar_arrive_expect_tx(&bar_q[buf], 2 * Q_BYTES);
        tma_load_3d(sQ + buf * Q_BYTES, &tmQ, &bar_q[buf], 0, q_lo + it * BQ, h);
        tma_load_3d(sdO + buf * Q_BYTES, &tmdO, &bar_q[buf], 0, q_lo + it * BQ, h);
      }
    }
  } else if (warp == BWD_MMA) {
    // the whole warp walks the tiles and one elected lane issues: operands stay in uniform registers (see the forward)
    const uint32_t idesc_st = make_idesc(FMT_BF16, FMT_BF16, 0, 0, 128, BQ);   // K·Qᵀ, V·dOᵀ
    const uint32_t idesc_dv = make_idesc(FMT_BF16, FMT_BF16, 0, 1, 128, D);    // Pᵀ·dO, dSᵀ·Q   (B MN-major)
    const uint32_t idesc_dq = make_idesc(FMT_BF16, FMT_BF16, 1, 1, 128, BQ);   // Kᵀ·dSᵀ         (A, B MN-major)
    // descriptors differ in their start address only (its unit is 16 bytes)
    const uint64_t kd = make_smem_desc_sw128(smem_u32(sK), 16, 1024), vd = make_smem_desc_sw128(smem_u32(sV), 16, 1024);
    const uint64_t qd = make_smem_desc_sw128(smem_u32(sQ), 16, 1024), dod = make_smem_desc_sw128(smem_u32(sdO), 16, 1024);
    const uint64_t kmn = make_smem_desc_sw128(smem_u32(sK), BKV * 128, 1024), dsmn = make_smem_desc_sw128(smem_u32(sdST), BKV * 128, 1024);
    const uint64_t qmn = make_smem_desc_sw128(smem_u32(sQ), BQ * 128, 1024), domn = make_smem_desc_sw128(smem_u32(sdO), BQ * 128, 1024);
    auto issue_s_dp = [&](int it) {
      const int buf = it % NQB, b = it % NB;
      cta_wait(&bar_q[buf], (it / NQB) & 1, abort_flag, p.status, ERR_WAIT_SMEM_FULL);
      if (it >= NB) cta_wait(&bar_dqfree[b], (it / NB - 1) & 1, abort_flag, p.status, ERR_WAIT_TMEM_EMPTY);
      tc_fence_after_sync();
      const uint64_t off = buf * (Q_BYTES / 16);
      const uint32_t s_col = tmem_base + b * BUF;
      if (elect_one_sync()) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) tc_mma_f16(s_col, kd + ks * 2, qd + off + ks * 2, idesc_st, ks != 0);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) tc_mma_f16(s_col + DP_COL, vd + ks * 2, dod + off + ks * 2, idesc_st, ks != 0);
        tc_commit(&bar_m1[b]);
      }
      __syncwarp();
    };
    cta_wait(bar_kv, 0, abort_flag, p.status, ERR_WAIT_SMEM_FULL);     // also when no query tile reads them
    tc_fence_after_sync();
    if (ntile > 0) issue_s_dp(0);
    if (ntile > 1) issue_s_dp(1);
    for (int it = 0; it < ntile; ++it) {
      if (__any_sync(0xffffffffu, *abort_flag)) break;
      const int buf = it % NQB, b = it % NB;
      if (it + 2 < ntile) issue_s_dp(it + 2);
      cta_wait(&bar_pds[b], (it / NB) & 1, abort_flag, p.status, ERR_WAIT_MISC);
      tc_fence_after_sync();
      const uint64_t off = buf * (Q_BYTES / 16), ds = dsmn + b * (DS_BYTES / 16);
      const uint32_t base = tmem_base + b * BUF;
      if (elect_one_sync()) {
#pragma unroll
        for (int ks = 0; ks < BKV / 16; ++ks)  // dQᵀ = Kᵀ · dSᵀ
          tc_mma_f16(base + DQT_COL, kmn + ks * (2048 / 16), ds + ks * (2048 / 16), idesc_dq, ks != 0);
        tc_commit(&bar_dq[b]);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)   // dV += Pᵀ · dO
          tc_mma_f16_ts(tmem_base + DV_COL, base + P16_COL + ks * 8, domn + off + ks * (2048 / 16), idesc_dv, (it | ks) != 0);
#pragma unroll
        for (int ks = 0; ks < BQ / 16; ++ks)   // dK += dSᵀ · Q
          tc_mma_f16_ts(tmem_base + DK_COL, base + DS16_COL + ks * 8, qmn + off + ks * (2048 / 16), idesc_dv, (it | ks) != 0);
        // only what somebody waits for is reported: nothing may come after the CTA has ended
        if (it + NQB < ntile) tc_commit(&bar_qe[buf]);
        if (it + 1 == ntile) tc_commit(bar_done);
      }
      __syncwarp();
    }
  } else if (warp >= BWD_WARPS) {
    // dQᵀ of a tile (row = head-dim index r) -> staging[q][r], then one bulk reduce-add into the fp32 accumulator (reductions
    // issued element by element from registers measured 25 % slower). Warps of their own: in the compute warps this copy, its
    // fence and its barrier were 900 of 2850 cycles a tile, with nothing to run under them.
    const bool issue_red = tid == BWD_COMPUTE;
    auto drain_sync = [] { asm volatile("bar.sync 3, 128;" ::: "memory"); };
    for (int it = 0; it < ntile; ++it) {
      const int b = it % NB;
      cta_wait(&bar_dq[b], (it / NB) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      uint32_t v[2][32];
      if (r < D) {
        tmem_ld_32x32b_x32(tmem_base + lane_off + b * BUF + DQT_COL, v[0]);
        tmem_ld_32x32b_x32(tmem_base + lane_off + b * BUF + DQT_COL + 32, v[1]);
        tmem_ld_wait();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_dqfree[b]);
      if (issue_red) tma_store_wait_read<0>();   // the last reduce-add has drained the staging buffer
      drain_sync();
      if (r < D) {
#pragma unroll
        for (int i = 0; i < BQ; ++i) sdQ[i * D + r] = __uint_as_float(v[i / 32][i % 32]) * p.scale;
      }
      fence_proxy_async_smem();
      drain_sync();                              // the staged tile is complete
      if (issue_red) {
        tma_reduce_add_3d(&tmdQ, sdQ, 0, q_lo + it * BQ, h);
        tma_store_commit();
      }
    }
    if (issue_red) tma_store_wait_read<0>();     // shared memory may be given back
  } else {
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
    for (int it = group; it < ntile; it += 2) {
      const int qt0 = q_lo + it * BQ, b = it % NB;
      float2* s_ld = s_ld_all + (it & 3) * BQ;     // (a slower warp may still read those of the group's last tile)
      int* s_ds = s_ds_all + (it & 3) * BQ;
      const uint32_t base = tmem_base + lane_off + b * BUF;
      uint8_t* ds_row = sdST + b * DS_BYTES + r * 128;
      if (r < BQ) {
        s_ld[r] = nxt_ld;
        s_ds[r] = nxt_ds;
      }
      group_sync();
      scalars(it + 2);
      cta_wait(&bar_m1[b], (it / NB) & 1, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
      tc_fence_after_sync();
      uint32_t sv[64], dp[32];
      {
        uint32_t a[32], c[32];
        tmem_ld_32x32b_x32(base, a);
        tmem_ld_32x32b_x32(base + 32, c);
        tmem_ld_32x32b_x32(base + DP_COL, dp);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) sv[i] = a[i], sv[32 + i] = c[i];
      }
      // masks are needed only where the tile touches the causal diagonal, a document boundary or the sequence end
      const bool need_mask = (qt0 < kv0 + BKV) || (s_ds[BQ - 1] > kv0) || (kv0 + BKV > p.T) || (qt0 + BQ > p.T);
      // probabilities, then the mask in a loop of its own: a branch per element would serialise the latencies of the others
#pragma unroll
      for (int i = 0; i < 64; i += 2) {
        const float4 ld = *reinterpret_cast<const float4*>(&s_ld[i]);   // {lse, delta} of two queries
        sv[i] = __float_as_uint(exp2f(fmaf(__uint_as_float(sv[i]), p.sl2, -ld.x)));
        sv[i + 1] = __float_as_uint(exp2f(fmaf(__uint_as_float(sv[i + 1]), p.sl2, -ld.z)));
      }
      if (need_mask) {
        // queries [lo, hi) see this thread's key: from the key itself to the last query whose document has begun at
        // or before it (document starts never fall, so that is a search for the first later one)
        const int lo = kv - qt0;
        int hi = 64;
        if (s_ds[63] > kv) {
          hi = 0;
#pragma unroll
          for (int step = 32; step > 0; step >>= 1)
            if (s_ds[hi + step - 1] <= kv) hi += step;
        }
        if (kv >= p.T) hi = 0;
#pragma unroll
        for (int i = 0; i < 64; ++i)
          if (i < lo || i >= hi) sv[i] = 0u;
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {          // over S, which this thread, the only reader of its row, has read as a whole
        uint32_t pp[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) pp[i] = pack_bf16x2(__uint_as_float(sv[32 * c + 2 * i]), __uint_as_float(sv[32 * c + 2 * i + 1]));
        tmem_st_32x32b_x16(base + P16_COL + c * 16, pp);
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        if (c == 1) {
          tmem_ld_32x32b_x32(base + DP_COL + 32, dp);
          tmem_ld_wait();
        }
        uint32_t dd[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float4 ld = *reinterpret_cast<const float4*>(&s_ld[32 * c + i]);
          dd[i >> 1] = pack_bf16x2(__uint_as_float(sv[32 * c + i]) * (__uint_as_float(dp[i]) - ld.y),
                                   __uint_as_float(sv[32 * c + i + 1]) * (__uint_as_float(dp[i + 1]) - ld.w));
        }
        tmem_st_32x32b_x16(base + DS16_COL + c * 16, dd);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<uint4*>(ds_row + (((c * 4 + j) ^ (r & 7)) << 4)) = make_uint4(dd[4 * j], dd[4 * j + 1], dd[4 * j + 2], dd[4 * j + 3]);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_pds[b]);
    }

    // final: dV, dK rows; each group writes half of the head dimension
    constexpr int CD = D / 2;
    if (ntile > 0) cta_wait(bar_done, 0, abort_flag, p.status, ERR_WAIT_TMEM_FULL);
    tc_fence_after_sync();
    __nv_bfloat16* dvrow = p.dv + (long long)kv * p.ld_dv + h * D + group * CD;
    __nv_bfloat16* dkrow = p.dk + (long long)kv * p.ld_dk + h * D + group * CD;
    if (ntile > 0) {
      auto write = [&](uint32_t col, __nv_bfloat16* row, float mul) {
#pragma unroll
        for (int c = 0; c < CD; c += 32) {
          uint32_t v[32];
          tmem_ld_32x32b_x32(tmem_base + lane_off + col + group * CD + c, v);
          tmem_ld_wait();
          if (kv < p.T) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              reinterpret_cast<uint4*>(row + c)[j] =
                  make_uint4(pack_bf16x2(__uint_as_float(v[8 * j]) * mul, __uint_as_float(v[8 * j + 1]) * mul),
                             pack_bf16x2(__uint_as_float(v[8 * j + 2]) * mul, __uint_as_float(v[8 * j + 3]) * mul),
                             pack_bf16x2(__uint_as_float(v[8 * j + 4]) * mul, __uint_as_float(v[8 * j + 5]) * mul),
                             pack_bf16x2(__uint_as_float(v[8 * j + 6]) * mul, __uint_as_float(v[8 * j + 7]) * mul));
          }
        }
      };
      write(DV_COL, dvrow, 1.f);
      write(DK_COL, dkrow, p.scale);
    } else if (kv < p.T) {
      // no query tile attends this key tile: its gradients are zero (the caller does not pre-zero dk / dv)
#pragma unroll
      for (int j = 0; j < CD / 8; ++j) {
        reinterpret_cast<uint4*>(dvrow)[j] = make_uint4(0u, 0u, 0u, 0u);
        reinterpret_cast<uint4*>(dkrow)[j] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }
  __syncwarp();
  if (tid == 0) {
    if (*abort_flag) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == BWD_MMA) tmem_dealloc(tmem_base, TMEM_COLS);
}

CUtensorMap qkv_map(const void* base, int T, int H, int D, long long ld, int rows) {
  return make_tmap_3d(base, TmapDtype::BF16, (uint64_t)D, (uint64_t)T, (uint64_t)H, (uint64_t)ld * 2, (uint64_t)D * 2, 64,
                      (uint32_t)rows, true);
}

KP make_kp(const AttnArgs& a) {
  KP p;
  p.T = a.T; p.H = a.H;
  p.scale = a.scale;
  p.sl2 = a.scale * 1.4426950408889634f;
  p.window_blocks = a.window_blocks;
  p.doc_start = a.doc_start; p.doc_end = a.doc_end;
  p.o = reinterpret_cast<__nv_bfloat16*>(a.o); p.ld_o = a.ld_o;
  p.dk = reinterpret_cast<__nv_bfloat16*>(a.dk); p.ld_dk = a.ld_dk;
  p.dv = reinterpret_cast<__nv_bfloat16*>(a.dv); p.ld_dv = a.ld_dv;
  p.lse = a.lse; p.delta = a.delta;
  p.status = a.status;
  return p;
}

void check_common(const AttnArgs& a) {
  if (a.D != 64 && a.D != 128) throw std::runtime_error("attention: head_dim must be 64 or 128");
  if (a.T <= 0 || a.H <= 0) throw std::runtime_error("attention: empty problem");
  if (!a.doc_start || !a.doc_end) throw std::runtime_error("attention: doc_start / doc_end are required");
}

template <typename K>
void set_smem(K kern, int bytes) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) throw std::runtime_error(std::string("attention: cudaFuncSetAttribute: ") + cudaGetErrorString(e));
}

void check_launch(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

template <int D, bool MIXED>
void fwd_configure() {
  auto kern = attn_fwd_kernel<D, MIXED>;
  set_smem(kern, FwdShape<D>::SMEM);
  cudaFuncAttributes attr;  // how many registers a thread is launched with is the compiler's choice
  const cudaError_t e = cudaFuncGetAttributes(&attr, kern);
  if (e != cudaSuccess) throw std::runtime_error(std::string("attention: cudaFuncGetAttributes: ") + cudaGetErrorString(e));
  if (!register_split_fits(attr.numRegs, FWD_THREADS, 256 * FWD_REGS_SOFTMAX + 128 * FWD_REGS_ISSUE))
    throw std::runtime_error("attention: the forward was built with " + std::to_string(attr.numRegs) +
                             " registers a thread, too few for its register split");
}

template <int D, bool MIXED>
void fwd_launch(const AttnArgs& a, const KP& p, int items) {
  using F = FwdShape<D>;
  CUtensorMap tq = qkv_map(a.q, a.T, a.H, D, a.ld_q, FQ);
  CUtensorMap tk = qkv_map(a.k, a.T, a.H, D, a.ld_k, FKV);
  CUtensorMap tv = qkv_map(a.v, a.T, a.H, D, a.ld_v, FKV);
  auto kern = attn_fwd_kernel<D, MIXED>;
  const int grid = std::min(p.pairs + 2 * (items - p.pairs), sm_count());
  launch_early(kern, grid, FWD_THREADS, F::SMEM, a.stream, tq, tk, tv, p);
  check_launch("attn_fwd launch");
}

template <int D>
void fwd_impl(const AttnArgs& a) {
  static PerDeviceOnce cfg;   // function attributes are per device
  int dev = 0;
  if (cfg.pending(&dev)) {    // every build at once: a call of any size readies the others, for a capture say
    fwd_configure<D, true>();
    if constexpr (D == 128) fwd_configure<D, false>();
    cfg.done(dev);
  }
  // The last round of items is dealt in single tiles where there is a CTA for each: two tiles on one multiprocessor share its
  // exponentials, which only pays while the other multiprocessors have work as well. 2048 x 6 heads of 128: 27.7 us (37.3 in
  // pairs, 53.9 with one tile per CTA and P in shared memory); 333 x 16 heads of 64 in documents of 128: 7.0 (8.8, 7.0).
  const int items = (a.T + 2 * FQ - 1) / (2 * FQ) * a.H, sms = sm_count(), rest = items % sms;
  KP p = make_kp(a);
  p.pairs = 2 * rest <= sms ? items - rest : items;
  // A build that knows pairs only is 6 % faster at head_dim 128 (16384 x 6 heads: 368 us, 392 with both kinds), 6 % slower at 64
  // (16 heads: 780, 733).
  if constexpr (D == 128) {
    if (p.pairs == items) return fwd_launch<D, false>(a, p, items);
  }
  fwd_launch<D, true>(a, p, items);
}

template <int D>
void bwd_impl(const AttnArgs& a) {
  const int smem = (D == 128 ? 2 * 2 * 128 * 128 + 6 * 2 * 64 * 128 + 128 * 128 : 2 * 128 * 128 + 2 * BWD64_QB * 64 * 128 + 3 * 128 * 128) +
                   64 * D * 4 + 12 * 64 * 4 + 256 + 1024;
  CUtensorMap tq = qkv_map(a.q, a.T, a.H, D, a.ld_q, 64);
  CUtensorMap tk = qkv_map(a.k, a.T, a.H, D, a.ld_k, 128);
  CUtensorMap tv = qkv_map(a.v, a.T, a.H, D, a.ld_v, 128);
  CUtensorMap tdo = qkv_map(a.d_o, a.T, a.H, D, a.ld_do, 64);
  CUtensorMap tdq = make_tmap_3d(a.dq_acc, TmapDtype::F32, (uint64_t)D, (uint64_t)a.T, (uint64_t)a.H,
                                 (uint64_t)a.ld_dq * 4, (uint64_t)D * 4, (uint32_t)D, 64, false);
  auto kern = D == 128 ? attn_bwd128_kernel : attn_bwd64_kernel;
  static PerDeviceOnce cfg;   // the shared-memory opt-in is a per-device attribute
  int dev = 0;
  if (cfg.pending(&dev)) { set_smem(kern, smem); cfg.done(dev); }
  dim3 grid((a.T + 127) / 128, a.H);
  launch_early(kern, grid, BWD_THREADS, smem, a.stream, tq, tk, tv, tdo, tdq, make_kp(a));
  check_launch("attn_bwd launch");
}

}  // namespace

void attn_fwd_sm100(const AttnArgs& a) {
  check_common(a);
  if (a.D == 128) fwd_impl<128>(a); else fwd_impl<64>(a);
}

void attn_delta_sm100(const AttnArgs& a) {
  check_common(a);
  const long long warps = (long long)a.T * a.H;
  const int threads = 256;
  const int blocks = (int)((warps * 32 + threads - 1) / threads);
  auto* o = reinterpret_cast<const __nv_bfloat16*>(a.o);
  auto* d_o = reinterpret_cast<const __nv_bfloat16*>(a.d_o);
  const bool aligned = (((uintptr_t)o | (uintptr_t)d_o) & 15) == 0 && a.ld_o % 8 == 0 && a.ld_do % 8 == 0;
  if (aligned) {
    const long long lanes = warps * (a.D / 8);
    const int vblocks = (int)((lanes + threads - 1) / threads);
    if (a.D == 128) launch_early(attn_delta_vec_kernel<128>, vblocks, threads, 0, a.stream, o, a.ld_o, d_o, a.ld_do, a.delta, a.T, a.H);
    else            launch_early(attn_delta_vec_kernel<64>, vblocks, threads, 0, a.stream, o, a.ld_o, d_o, a.ld_do, a.delta, a.T, a.H);
  } else if (a.D == 128) {
    attn_delta_kernel<128><<<blocks, threads, 0, a.stream>>>(o, a.ld_o, d_o, a.ld_do, a.delta, a.T, a.H);
  } else {
    attn_delta_kernel<64><<<blocks, threads, 0, a.stream>>>(o, a.ld_o, d_o, a.ld_do, a.delta, a.T, a.H);
  }
  check_launch("attn_delta launch");
}

void attn_bwd_sm100(const AttnArgs& a) {
  check_common(a);
  // dQᵀ = Kᵀ·dSᵀ puts the head dimension on the MMA M axis, always issued at M = 128. With head_dim 64 the upper 64
  // rows of the A operand fall on the V tile that follows K in shared memory; their accumulator rows are never read.
  if (a.D == 128) bwd_impl<128>(a); else bwd_impl<64>(a);
}

}  // namespace b200

// ------------------------------------------------------------------------------------------------
// Allocation-free entry point (see attn_noalloc.h): the delta scratch is a fixed array in the library image.
// ------------------------------------------------------------------------------------------------
#include "attn_noalloc.h"

static __device__ __align__(256) float g_noalloc_delta[B200_ATTN_NOALLOC_MAX_HT];

namespace {
thread_local std::string t_noalloc_error;
// Device address of the scratch array, per device ordinal. Two host threads that make the first call on one device
// both store the same value.
std::atomic<float*> g_noalloc_delta_addr[64];
}  // namespace

extern "C" const char* b200_attn_bwd_noalloc_error(void) { return t_noalloc_error.c_str(); }

extern "C" int b200_attn_bwd_noalloc(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                     const float* lse, float* dq_acc, void* dk, void* dv, const int* doc_start,
                                     const int* doc_end, int T, int H, int D, long long ld_q, long long ld_k,
                                     long long ld_v, long long ld_o, long long ld_do, long long ld_dq, long long ld_dk,
                                     long long ld_dv, float scale, int window_blocks, int* status,
                                     cudaStream_t stream) {
  try {
    if (!q || !k || !v || !o || !d_o || !lse || !dq_acc || !dk || !dv || !doc_start || !doc_end || T <= 0 || H <= 0) {
      t_noalloc_error = "null pointer or empty problem";
      return -1;
    }
    if (D != 128 && D != 64) {
      t_noalloc_error = "head_dim must be 64 or 128";
      return -1;
    }
    if ((long long)T * H > (long long)B200_ATTN_NOALLOC_MAX_HT) {
      t_noalloc_error = "H * T exceeds the built-in scratch (B200_ATTN_NOALLOC_MAX_HT floats)";
      return -2;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) {
      t_noalloc_error = "cannot determine the current device";
      return -3;
    }
    float* scratch = g_noalloc_delta_addr[dev].load(std::memory_order_acquire);
    if (scratch == nullptr) {
      // Once per device, with that device current: in host code the array's name is only a handle, the address a
      // kernel can use has to be asked for.
      void* ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, g_noalloc_delta);
      if (e != cudaSuccess || ptr == nullptr) {
        t_noalloc_error = std::string("cudaGetSymbolAddress failed: ") + cudaGetErrorString(e);
        return -3;
      }
      scratch = static_cast<float*>(ptr);
      g_noalloc_delta_addr[dev].store(scratch, std::memory_order_release);
    }
    b200::AttnArgs a;
    a.q = q; a.k = k; a.v = v; a.o = const_cast<void*>(o); a.d_o = d_o;
    a.dq_acc = dq_acc; a.dk = dk; a.dv = dv;
    a.lse = const_cast<float*>(lse);
    a.delta = scratch;
    a.doc_start = doc_start; a.doc_end = doc_end;
    a.T = T; a.H = H; a.D = D;
    a.ld_q = ld_q; a.ld_k = ld_k; a.ld_v = ld_v; a.ld_o = ld_o; a.ld_do = ld_do; a.ld_dq = ld_dq; a.ld_dk = ld_dk;
    a.ld_dv = ld_dv;
    a.scale = scale; a.window_blocks = window_blocks; a.status = status; a.stream = stream;
    b200::attn_delta_sm100(a);
    b200::attn_bwd_sm100(a);
    return 0;
  } catch (const std::exception& ex) {
    t_noalloc_error = ex.what();
    return -3;
  }
}
