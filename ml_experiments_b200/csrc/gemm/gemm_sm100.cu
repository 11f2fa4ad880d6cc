// Persistent, warp-specialised GEMM for sm_100a.
//
//   warp 0      : TMA producer  (cp.async.bulk.tensor -> 128B-swizzled shared-memory stages)
//   warp 1      : MMA issuer    (one thread issues tcgen05.mma; accumulators live in tensor memory)
//   the others  : epilogue      (tcgen05.ld -> fused epilogue -> swizzled staging -> TMA store / reduce-add)
//
// Two TMEM accumulators (2 x BN columns) let the epilogue of tile i overlap the main loop of tile
// i+1. Operands may be K-major or MN-major (selected per operand through the shared-memory
// descriptor and the instruction descriptor), so forward (A·Wᵀ), data-gradient (dY·W) and
// weight-gradient (dYᵀ·X) products all run without a transpose pass. bf16 and fp8 (e4m3/e5m2)
// inputs, fp32 accumulation, bf16 or fp32 output, batched, optional split-K by TMA reduce-add.
#include "../common/per_device.h"
#include "gemm.h"

#include <stdexcept>
#include <string>

#include "../common/ptx.cuh"
#include "../common/tmap.h"

namespace b200 {

namespace {

constexpr int BM = 128;
// Epilogue warps: a pair has two for each quarter of the rows, which share its columns. (The squared-ReLU backward reads an aux
// tile and takes a square root per element: with four warps 49152 x 3072 x 768 took 308 us where the product alone takes 176.)
constexpr int epi_warps(int pair) { return pair ? 8 : 4; }
constexpr int threads(int pair) { return 64 + 32 * epi_warps(pair); }

struct KParams {
  int M, N, K;
  int batch, splits;
  int k_per_split;  // multiple of the stage depth
  int tiles_m, tiles_n, total_tiles;
  uint32_t idesc;
  int epi;
  int out_f32;
  int reduce_add;
  float alpha, beta;
  const __nv_bfloat16* aux;
  long long ld_aux, stride_aux;
  int* status;
};

template <int BN, int STAGES, int PAIR>
struct SmemLayout {
  static constexpr int kABytes = BM * 128;
  static constexpr int kBBytes = BN / (PAIR + 1) * 128;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStagingBytes = epi_warps(PAIR) * 2 * 4096;   // each 2 buffers x (32 rows x 128 B)
  static constexpr int kBarOffset = STAGES * kStageBytes + kStagingBytes;
  static constexpr int kTotal = kBarOffset + (2 * STAGES + 4 + 2 * epi_warps(PAIR)) * 8 + 16 + 1024;  // + alignment slack
};

// PAIR: two CTAs work on one tile of 256 x BN. Each loads and keeps its own 128 rows of A and half of B, which the tensor cores of
// both read: 64 bytes per clock and SM out of L2 at the full rate of the tensor cores where a CTA of its own, with 128 x 256, needs 96.
template <int BN, int STAGES, int AMN, int BMN, int ESZ, int PAIR>
__global__ void __launch_bounds__(threads(PAIR), 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmAux, const KParams p) {
  using L = SmemLayout<BN, STAGES, PAIR>;
  constexpr int TM = BM * (PAIR + 1), BROWS = BN / (PAIR + 1);   // rows of a tile, rows of B in this CTA
  constexpr int BK = 128 / ESZ;         // elements along K per stage (one 128-byte swizzle span)
  constexpr int UMMA_K = 32 / ESZ;      // elements along K per tcgen05.mma
  constexpr int KSTEPS = BK / UMMA_K;   // 4
  constexpr int MN_SPAN = 128 / ESZ;    // elements per 128-byte span along M/N (MN-major operands)
  constexpr int CHUNK_BYTES = BK * 128; // one MN-major box: BK k-rows x 128 B
  constexpr uint32_t TMEM_COLS = 2 * BN;
  constexpr int EW = epi_warps(PAIR), ECOLS = BN * 4 / EW;   // columns of an epilogue warp

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + (-smem_u32(smem_raw) & 1023u);
  uint8_t* staging = smem + STAGES * L::kStageBytes;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint64_t* aux_bar = tempty_bar + 2;  // [epilogue warps][2 staging buffers]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aux_bar + 2 * EW);

  const int rank = PAIR ? (int)cluster_rank() : 0, unit = blockIdx.x / (PAIR + 1), units = gridDim.x / (PAIR + 1);
  const bool poisoned = status_poisoned(p.status);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], EW * (PAIR + 1));
    }
    for (int a = 0; a < 2 * EW; ++a) mbar_init(&aux_bar[a], 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
    tma_prefetch_desc(&tmAux);
  }
  if (PAIR && threadIdx.x == 0) tmem_slot[1] = poisoned;
  if (warp == 1) {
    if (PAIR) {
      tmem_alloc_pair(tmem_slot, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  bool leave = __syncthreads_or(poisoned);           // all warps or none
  if (PAIR) {                                        // of both CTAs: the first one's word decides
    cluster_sync();                                  // (barriers are ready in both)
    leave = cluster_load(cluster_addr(&tmem_slot[1], 0)) != 0;
  }
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  let_next_start();
  after_previous();                                  // the set-up above has run under the end of the kernel before
  if (leave) {
    if (PAIR) cluster_sync();                        // the word has been read
    if (warp == 1) {
      if (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
      else tmem_dealloc(tmem_base, TMEM_COLS);
    }
    return;
  }

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // As the MMA issuer below: the warp walks the tiles, one elected lane issues, coordinates and addresses stay in uniform registers.
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    const uint32_t full0 = PAIR ? cluster_addr(full_bar, 0) : smem_u32(full_bar);   // of a pair, the loads of both report to the CTA that issues
    const uint32_t smem0 = smem_u32(smem);
    for (int t = unit; t < p.total_tiles && ok; t += units) {
      int r = t;
      const int nt = r % p.tiles_n; r /= p.tiles_n;  // N fastest: concurrent CTAs share one A panel through L2
      const int mt = r % p.tiles_m; r /= p.tiles_m;
      const int sp = r % p.splits;
      const int b = r / p.splits;
      const int m0 = mt * TM + rank * BM, n0 = nt * BN + rank * BROWS;
      const int kbeg = sp * p.k_per_split;
      const int kend = min(p.K, kbeg + p.k_per_split);
      const int nkb = (kend - kbeg + BK - 1) / BK;
      for (int kb = 0; kb < nkb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ERR_WAIT_SMEM_EMPTY));
        if (!ok) break;
        if (elect_one_sync()) {
          const uint32_t sA = smem0 + stage * L::kStageBytes, sB = sA + L::kABytes, bar = full0 + stage * 8;
          const int k0 = kbeg + kb * BK;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[stage], L::kStageBytes * (PAIR + 1));
          if (AMN == 0) {
            tma_load_3d_at<PAIR>(sA, &tmA, bar, k0, m0, b);
          } else {
#pragma unroll
            for (int c = 0; c < BM / MN_SPAN; ++c) tma_load_3d_at<PAIR>(sA + c * CHUNK_BYTES, &tmA, bar, m0 + c * MN_SPAN, k0, b);
          }
          if (BMN == 0) {
            tma_load_3d_at<PAIR>(sB, &tmB, bar, k0, n0, b);
          } else {
#pragma unroll
            for (int c = 0; c < BROWS / MN_SPAN; ++c) tma_load_3d_at<PAIR>(sB + c * CHUNK_BYTES, &tmB, bar, n0 + c * MN_SPAN, k0, b);
          }
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    if (PAIR && ok) {      // the reports of the last stages: none may come after this CTA has ended
      for (int i = 0; i < STAGES && ok; ++i) {
        ok = __all_sync(0xffffffffu, mbar_wait(&empty_bar[stage], phase ^ 1, p.status, ERR_WAIT_SMEM_EMPTY));
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    if (!ok && lane == 0) {
      // Give loads that are still in flight a bounded time (1 ms) to land before shared memory is released.
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 1000000ull) __nanosleep(1000);
    }
  } else if (warp == 1 && rank == 0) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the tiles and one elected lane issues: descriptors and addresses then stay in uniform registers
    // (from a single-thread branch they are moved there for every MMA, 99 cycles each; 128 x 128 x 16 takes 64).
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    // descriptors differ in their start address only (its unit is 16 bytes)
    const uint64_t a_desc = make_smem_desc_sw128(smem_u32(smem), AMN ? CHUNK_BYTES : 16, 1024);
    const uint64_t b_desc = make_smem_desc_sw128(smem_u32(smem + L::kABytes), BMN ? CHUNK_BYTES : 16, 1024);
    constexpr int A_STEP = (AMN ? UMMA_K * 128 : 32) / 16, B_STEP = (BMN ? UMMA_K * 128 : 32) / 16;
    for (int t = unit; t < p.total_tiles && ok; t += units) {
      int r = t / (p.tiles_m * p.tiles_n);
      const int sp = r % p.splits;
      const int kbeg = sp * p.k_per_split;
      const int kend = min(p.K, kbeg + p.k_per_split);
      const int nkb = (kend - kbeg + BK - 1) / BK;
      ok = __all_sync(0xffffffffu, mbar_wait(&tempty_bar[acc], acc_phase ^ 1, p.status, ERR_WAIT_TMEM_EMPTY));
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t d_tmem = tmem_base + acc * BN;
      for (int kb = 0; kb < nkb; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, p.status, ERR_WAIT_SMEM_FULL));
        if (!ok) break;
        tc_fence_after_sync();
        if (elect_one_sync()) {
          const uint64_t ad = a_desc + stage * (L::kStageBytes / 16), bd = b_desc + stage * (L::kStageBytes / 16);
#pragma unroll
          for (int ks = 0; ks < KSTEPS; ++ks) {
            if (PAIR) tc_mma_pair<ESZ == 1>(d_tmem, ad + ks * A_STEP, bd + ks * B_STEP, p.idesc, (kb | ks) != 0);
            else if (ESZ == 2) tc_mma_f16(d_tmem, ad + ks * A_STEP, bd + ks * B_STEP, p.idesc, (kb | ks) != 0);
            else tc_mma_f8(d_tmem, ad + ks * A_STEP, bd + ks * B_STEP, p.idesc, (kb | ks) != 0);
          }
          auto commit = [](uint64_t* bar) {
            if (PAIR) tc_commit_pair(bar);
            else tc_commit(bar);
          };
          commit(&empty_bar[stage]);                     // frees the stage once these MMAs have read it
          if (kb == nkb - 1) commit(&tfull_bar[acc]);    // accumulator complete
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
  } else if (warp >= 2) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    const int cbeg = EW == 4 ? 0 : (warp - 2) / 4 * ECOLS;          // first of its columns of the tile
    uint8_t* my_staging = staging + (warp - 2) * 8192;
    auto give_back = [&](int a) {                      // the accumulator has been read
      if (PAIR) cluster_arrive(cluster_addr(&tempty_bar[a], 0));
      else mbar_arrive(&tempty_bar[a]);
    };
    int buf = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    const int out_cols_per_buf = p.out_f32 ? 32 : 64;
    // bf16 output with an aux operand: the aux tile is brought by TMA into the (swizzled) staging buffer, combined in
    // place by the thread that owns the row, and the same buffer is then stored - no uncoalesced per-row global loads.
    const bool aux_tma = (p.epi == EPI_AXPBY || p.epi == EPI_RELU2_BWD) && !p.out_f32 && !p.reduce_add;
    uint64_t* my_aux_bar = aux_bar + (warp - 2) * 2;
    uint32_t aux_phase0 = 0, aux_phase1 = 0;
    for (int t = unit; t < p.total_tiles && ok; t += units) {
      int r = t;
      const int nt = r % p.tiles_n; r /= p.tiles_n;
      const int mt = r % p.tiles_m; r /= p.tiles_m;
      const int b = r / p.splits;
      const int m0 = mt * TM + rank * BM, n0 = nt * BN;
      const int row = m0 + q * 32 + lane;
      const int ngroups = max(0, min(ECOLS / 64, (p.N - n0 - cbeg + 63) / 64));
      auto issue_aux = [&](int g, int bsel) {
        if (lane == 0) {
          tma_store_wait_read<0>();  // the store that last used this buffer has drained it
          mbar_arrive_expect_tx(&my_aux_bar[bsel], 4096);
          tma_load_3d(my_staging + bsel * 4096, &tmAux, &my_aux_bar[bsel], n0 + cbeg + g * 64, m0 + q * 32, b);
        }
      };
      constexpr int AHEAD = ECOLS / 64 <= 2 ? 2 : 1;
      if (aux_tma) {                 // the first aux tiles are on their way while the product is formed
#pragma unroll
        for (int g = 0; g < AHEAD; ++g)
          if (g < ngroups) issue_aux(g, buf ^ g);
      }
      if (!mbar_wait(&tfull_bar[acc], acc_phase, p.status, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after_sync();
      if (aux_tma) {
        for (int g = 0; g < ngroups && ok; ++g) {
          if (AHEAD == 1 && g + 1 < ngroups) issue_aux(g + 1, buf ^ 1);
          uint32_t v0[32], v1[32];
          tmem_ld_32x32b_x32(tmem_base + (uint32_t(q * 32) << 16) + acc * BN + cbeg + g * 64, v0);
          tmem_ld_32x32b_x32(tmem_base + (uint32_t(q * 32) << 16) + acc * BN + cbeg + g * 64 + 32, v1);
          tmem_ld_wait();
          const uint32_t ph = buf ? aux_phase1 : aux_phase0;
          if (!mbar_wait(&my_aux_bar[buf], ph, p.status, ERR_WAIT_SMEM_FULL)) { ok = false; break; }
          if (buf) aux_phase1 ^= 1; else aux_phase0 ^= 1;
          uint8_t* rowp = my_staging + buf * 4096 + lane * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint4* cell = reinterpret_cast<uint4*>(rowp + ((j ^ (lane & 7)) << 4));
            const uint4 u = *cell;
            float a[8], f[8];
            float2 x0 = unpack_bf16x2(u.x), x1 = unpack_bf16x2(u.y), x2 = unpack_bf16x2(u.z), x3 = unpack_bf16x2(u.w);
            a[0] = x0.x; a[1] = x0.y; a[2] = x1.x; a[3] = x1.y; a[4] = x2.x; a[5] = x2.y; a[6] = x3.x; a[7] = x3.y;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float accv = __uint_as_float(j < 4 ? v0[8 * j + i] : v1[8 * (j - 4) + i]) * p.alpha;
              f[i] = (p.epi == EPI_AXPBY) ? fmaf(p.beta, a[i], accv) : accv * 2.f * sqrtf(a[i]);
            }
            *cell = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmC, my_staging + buf * 4096, n0 + cbeg + g * 64, m0 + q * 32, b);
            tma_store_commit();
          }
          buf ^= 1;
        }
        if (AHEAD == 2) buf = 0;     // (groups and buffers go together)
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) give_back(acc);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
        continue;
      }
      const __nv_bfloat16* aux_row =
          p.aux ? p.aux + (long long)b * p.stride_aux + (long long)row * p.ld_aux : nullptr;
      int filled = 0;      // columns written into the current staging buffer
      int buf_col0 = n0 + cbeg;   // first output column of the current staging buffer
      const bool use_aux = (p.epi == EPI_AXPBY || p.epi == EPI_RELU2_BWD);
      const bool aux_vec = use_aux && row < p.M && ((p.ld_aux & 7) == 0);
      uint4 aux_next[4];
      auto fetch_aux = [&](int c) {  // 32 bf16 of this thread's row, columns n0+c .. n0+c+31
        const int col = n0 + c;
        if (aux_vec && col + 32 <= p.N) {
          const uint4* src = reinterpret_cast<const uint4*>(aux_row + col);
#pragma unroll
          for (int i = 0; i < 4; ++i) aux_next[i] = __ldg(src + i);
        } else {
          __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(aux_next);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            e[i] = (row < p.M && col + i < p.N) ? aux_row[col + i] : __float2bfloat16(0.f);
        }
      };
      if (use_aux) fetch_aux(cbeg);
      for (int c = cbeg; c < cbeg + ECOLS; c += 32) {
        if (n0 + c >= p.N) break;
        uint32_t v[32];
        tmem_ld_32x32b_x32(tmem_base + (uint32_t(q * 32) << 16) + acc * BN + c, v);
        uint4 aux_cur[4];
        if (use_aux) {
#pragma unroll
          for (int i = 0; i < 4; ++i) aux_cur[i] = aux_next[i];
          if (c + 32 < cbeg + ECOLS && n0 + c + 32 < p.N) fetch_aux(c + 32);  // in flight while this chunk is processed
        }
        tmem_ld_wait();
        float f[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(v[i]) * p.alpha;
        if (p.epi == EPI_RELU2) {
#pragma unroll
          for (int i = 0; i < 32; ++i) { float rr = fmaxf(f[i], 0.f); f[i] = rr * rr; }
        } else if (use_aux) {
          float a[32];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 u = aux_cur[i];
            float2 x0 = unpack_bf16x2(u.x), x1 = unpack_bf16x2(u.y), x2 = unpack_bf16x2(u.z), x3 = unpack_bf16x2(u.w);
            a[8 * i + 0] = x0.x; a[8 * i + 1] = x0.y; a[8 * i + 2] = x1.x; a[8 * i + 3] = x1.y;
            a[8 * i + 4] = x2.x; a[8 * i + 5] = x2.y; a[8 * i + 6] = x3.x; a[8 * i + 7] = x3.y;
          }
          if (p.epi == EPI_AXPBY) {
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = fmaf(p.beta, a[i], f[i]);
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = f[i] * 2.f * sqrtf(a[i]);
          }
        }
        // ---- stage into 128B-swizzled shared memory (row = lane, 16-byte chunk j stored at j ^ (lane & 7))
        if (filled == 0) {
          if (lane == 0) tma_store_wait_read<1>();  // the store that last used this buffer has drained it
          __syncwarp();
          buf_col0 = n0 + c;
        }
        uint8_t* rowp = my_staging + buf * 4096 + lane * 128;
        if (p.out_f32) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            uint4 u = make_uint4(__float_as_uint(f[4 * j]), __float_as_uint(f[4 * j + 1]),
                                 __float_as_uint(f[4 * j + 2]), __float_as_uint(f[4 * j + 3]));
            *reinterpret_cast<uint4*>(rowp + ((j ^ (lane & 7)) << 4)) = u;
          }
        } else {
          const int h = filled >> 5;  // 0 or 1: which half of the 64-column buffer
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 u = make_uint4(pack_bf16x2(f[8 * j], f[8 * j + 1]), pack_bf16x2(f[8 * j + 2], f[8 * j + 3]),
                                 pack_bf16x2(f[8 * j + 4], f[8 * j + 5]), pack_bf16x2(f[8 * j + 6], f[8 * j + 7]));
            *reinterpret_cast<uint4*>(rowp + (((h * 4 + j) ^ (lane & 7)) << 4)) = u;
          }
        }
        filled += 32;
        if (filled == out_cols_per_buf) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (p.reduce_add) tma_reduce_add_3d(&tmC, my_staging + buf * 4096, buf_col0, m0 + q * 32, b);
            else              tma_store_3d(&tmC, my_staging + buf * 4096, buf_col0, m0 + q * 32, b);
            tma_store_commit();
          }
          buf ^= 1;
          filled = 0;
        }
      }
      // accumulator fully read: hand it back to the MMA warp
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) give_back(acc);
      if (filled != 0) {  // partially filled buffer at a ragged N edge (columns beyond N are clipped by TMA)
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (p.reduce_add) tma_reduce_add_3d(&tmC, my_staging + buf * 4096, buf_col0, m0 + q * 32, b);
          else              tma_store_3d(&tmC, my_staging + buf * 4096, buf_col0, m0 + q * 32, b);
          tma_store_commit();
        }
        buf ^= 1;
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (lane == 0) tma_store_wait_all<0>();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync();     // neither ends while the other's operands, accumulator or barriers are in use
  tc_fence_after_sync();
  if (warp == 1) {
    if (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int BN, int STAGES, int AMN, int BMN, int ESZ, int PAIR>
void launch(const GemmArgs& a, const KParams& kp, const CUtensorMap& tA, const CUtensorMap& tB,
            const CUtensorMap& tC, const CUtensorMap& tX, int grid) {
  using L = SmemLayout<BN, STAGES, PAIR>;
  auto kern = gemm_kernel<BN, STAGES, AMN, BMN, ESZ, PAIR>;
  static PerDeviceOnce configured;   // the shared-memory opt-in is a per-device attribute
  int dev = 0;
  if (configured.pending(&dev)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotal);
    if (e != cudaSuccess) throw std::runtime_error(std::string("gemm: cudaFuncSetAttribute: ") + cudaGetErrorString(e));
    configured.done(dev);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads(PAIR));
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = a.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = PAIR + 1;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = PAIR ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tA, tB, tC, tX, kp);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) throw std::runtime_error(std::string("gemm launch: ") + cudaGetErrorString(e));
}

template <int BN, int STAGES, int ESZ, int PAIR>
void dispatch_major(const GemmArgs& a, const KParams& kp, const CUtensorMap& tA, const CUtensorMap& tB,
                    const CUtensorMap& tC, const CUtensorMap& tX, int grid) {
  if (!a.a_mn && !a.b_mn) launch<BN, STAGES, 0, 0, ESZ, PAIR>(a, kp, tA, tB, tC, tX, grid);
  else if (!a.a_mn && a.b_mn) launch<BN, STAGES, 0, 1, ESZ, PAIR>(a, kp, tA, tB, tC, tX, grid);
  else if (a.a_mn && !a.b_mn) launch<BN, STAGES, 1, 0, ESZ, PAIR>(a, kp, tA, tB, tC, tX, grid);
  else if constexpr (!PAIR) launch<BN, STAGES, 1, 1, ESZ, 0>(a, kp, tA, tB, tC, tX, grid);      // (by_pairs: never pairs)
}

}  // namespace

// A pair's set-up and end (clusters, their barriers) take time, and its tiles of 256 rows may leave more of the machine without work in
// the last round. Weight gradients (both operands MN-major, K long) gain nothing from it: 3072 x 768 x 49152 163, 159 us.
// Pair, single: 8 of 3072 x 768 x 768 (29 GFLOP) 29.2, 27.5 us; 10007 x 3072 x 768 (47) 39.8, 41.3; 16 of 768 x 768 x
// 3072 (58) 47.4, 49.5; 20011 x 3072 x 768 72, 77; 49152 x 3072 x 768 173, 186. Nor has a pair enough work in a tile whose K ends after a few
// stages of 128 bytes, where its epilogue, twice as long, is not hidden: bf16, 49152 x 3072 x 256 119, 92, x 512 133, 127; fp8, 49152 x 50304 x 768 2550, 1910.
// From 11 stages on it is the faster one (bf16: 704 0.97, 640 1.0 of the single's time, means of five sizes and five epilogues).
static bool by_pairs(int M, int N, int K, int batch, bool both_mn, int esz, int splits, int sms) {
  if (N <= 128 || sms < 2 || M <= BM || 2.0 * M * N * K * batch < 4e10 || both_mn) return false;
  if ((K + splits - 1) / splits * esz <= 10 * 128) return false;
  auto rounds = [&](int rows, int at_once) {
    const long long tiles = (long long)((M + rows - 1) / rows) * ((N + 255) / 256) * splits * batch;
    return (double)((tiles + at_once - 1) / at_once);
  };
  return 0.9 * rounds(2 * BM, sms / 2) <= rounds(BM, sms);
}
bool gemm_by_pairs(int M, int N, int K, int batch, bool both_mn, int element_bytes, int splits) {
  return by_pairs(M, N, K, batch, both_mn, element_bytes, splits, sm_count());
}

void gemm_sm100(const GemmArgs& a) {
  const int esz = (a.a_dtype == GEMM_BF16) ? 2 : 1;
  const int esz_b = (a.b_dtype == GEMM_BF16) ? 2 : 1;
  if (esz != esz_b) throw std::runtime_error("gemm: A and B must both be bf16 or both be fp8");
  if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.batch <= 0) throw std::runtime_error("gemm: empty problem");
  if (a.c_dtype != GEMM_BF16 && a.c_dtype != GEMM_F32) throw std::runtime_error("gemm: C must be bf16 or fp32");
  const int splits = a.split_k < 1 ? 1 : a.split_k;
  const bool reduce_add = (splits > 1) || a.accumulate;
  if (reduce_add && a.c_dtype != GEMM_F32) throw std::runtime_error("gemm: split-K / accumulate needs fp32 C");
  if (splits > 1 && !a.accumulate && a.ldc != a.N) throw std::runtime_error("gemm: split-K needs a dense C (ldc == N)");
  if (splits > 1 && a.epilogue != EPI_NONE) throw std::runtime_error("gemm: split-K supports only the plain epilogue");
  if ((a.epilogue == EPI_AXPBY || a.epilogue == EPI_RELU2_BWD) && a.aux == nullptr)
    throw std::runtime_error("gemm: this epilogue needs aux");

  const int BN = a.N > 128 ? 256 : 128;
  const int sms = a.max_ctas > 0 ? a.max_ctas : sm_count();
  const bool pair = by_pairs(a.M, a.N, a.K, a.batch, a.a_mn && a.b_mn, esz, splits, sms);
  const int TM = pair ? 2 * BM : BM, brows = pair ? BN / 2 : BN;
  const int BK = 128 / esz;
  const int span = 128 / esz;
  const TmapDtype in_dt = esz == 2 ? TmapDtype::BF16 : TmapDtype::U8;
  const uint64_t nb = (uint64_t)a.batch;

  CUtensorMap tA, tB, tC;
  if (!a.a_mn) tA = make_tmap_3d(a.A, in_dt, a.K, a.M, nb, a.lda * esz, a.stride_a * esz, BK, BM, true);
  else         tA = make_tmap_3d(a.A, in_dt, a.M, a.K, nb, a.lda * esz, a.stride_a * esz, span, BK, true);
  if (!a.b_mn) tB = make_tmap_3d(a.B, in_dt, a.K, a.N, nb, a.ldb * esz, a.stride_b * esz, BK, brows, true);
  else         tB = make_tmap_3d(a.B, in_dt, a.N, a.K, nb, a.ldb * esz, a.stride_b * esz, span, BK, true);
  const int osz = a.c_dtype == GEMM_F32 ? 4 : 2;
  tC = make_tmap_3d(a.C, a.c_dtype == GEMM_F32 ? TmapDtype::F32 : TmapDtype::BF16, a.N, a.M, nb, a.ldc * osz,
                    a.stride_c * osz, 128 / osz, 32, true);

  CUtensorMap tX = tC;  // aux tile map (bf16 [batch][M][N]); only dereferenced by the aux epilogues
  if (a.aux != nullptr && (a.ldaux % 8) == 0)
    tX = make_tmap_3d(a.aux, TmapDtype::BF16, a.N, a.M, nb, a.ldaux * 2, a.stride_aux * 2, 64, 32, true);
  else if (a.aux != nullptr)
    throw std::runtime_error("gemm: aux row pitch must be a multiple of 8 elements");

  KParams kp;
  kp.M = a.M; kp.N = a.N; kp.K = a.K;
  kp.batch = a.batch; kp.splits = splits;
  int kps = (a.K + splits - 1) / splits;
  kps = (kps + BK - 1) / BK * BK;
  kp.k_per_split = kps;
  // drop splits that would start beyond K
  while (kp.splits > 1 && (long long)(kp.splits - 1) * kps >= a.K) kp.splits--;
  kp.tiles_m = (a.M + TM - 1) / TM;
  kp.tiles_n = (a.N + BN - 1) / BN;
  kp.total_tiles = kp.tiles_m * kp.tiles_n * kp.splits * a.batch;
  auto fmt = [](int dt) -> uint32_t { return dt == GEMM_BF16 ? FMT_BF16 : (dt == GEMM_E4M3 ? FMT_E4M3 : FMT_E5M2); };
  kp.idesc = make_idesc(fmt(a.a_dtype), fmt(a.b_dtype), a.a_mn ? 1 : 0, a.b_mn ? 1 : 0, TM, BN);
  kp.epi = a.epilogue;
  kp.out_f32 = a.c_dtype == GEMM_F32;
  kp.reduce_add = reduce_add ? 1 : 0;
  kp.alpha = a.alpha; kp.beta = a.beta;
  kp.aux = reinterpret_cast<const __nv_bfloat16*>(a.aux);
  kp.ld_aux = a.ldaux; kp.stride_aux = a.stride_aux;
  kp.status = a.status;

  if (splits > 1 && !a.accumulate) {
    // split-K partial sums are combined by reduce-add into C, which therefore starts from zero
    if (a.batch == 1 || a.stride_c == (long long)a.M * a.ldc) {
      cudaMemsetAsync(a.C, 0, (size_t)a.batch * a.M * a.ldc * osz, a.stream);
    } else {
      for (int b = 0; b < a.batch; ++b)
        cudaMemsetAsync((char*)a.C + (size_t)b * a.stride_c * osz, 0, (size_t)a.M * a.ldc * osz, a.stream);
    }
  }

  int grid = pair ? sms & ~1 : sms;
  const int wanted = kp.total_tiles * (pair ? 2 : 1);
  if (grid > wanted) grid = wanted;

  if (esz == 2) {
    if (pair) dispatch_major<256, 5, 2, 1>(a, kp, tA, tB, tC, tX, grid);
    else if (BN == 256) dispatch_major<256, 4, 2, 0>(a, kp, tA, tB, tC, tX, grid);
    else dispatch_major<128, 6, 2, 0>(a, kp, tA, tB, tC, tX, grid);
  } else {
    if (pair) dispatch_major<256, 5, 1, 1>(a, kp, tA, tB, tC, tX, grid);
    else if (BN == 256) dispatch_major<256, 4, 1, 0>(a, kp, tA, tB, tC, tX, grid);
    else dispatch_major<128, 6, 1, 0>(a, kp, tA, tB, tC, tX, grid);
  }
}

}  // namespace b200
