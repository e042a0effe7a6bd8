// Grouped bf16 GEMMs of the mixture-of-experts MLP for sm_100a.
//
// Token rows arrive grouped by (source rank, local expert); group g occupies
// rows [g_start[g], g_start[g] + g_len[g]) of a row buffer, with g_len a
// multiple of 128 (segments are padded with zero rows) and expert(g) =
// g % experts.  Three products share one kernel template:
//
//   kGroupedFwd    Y[rows, N]  = X[rows, K]  * W[e][N, K]^T      (forward)
//   kGroupedDgrad  dX[rows, K] = dY[rows, N] * W[e][N, K]        (input gradient)
//   kGroupedWgrad  dW[e][N, K] += dY[rows_e, N]^T * X[rows_e, K] (weight gradient,
//                  contraction over all row segments of expert e)
//
// The structure is that of the dense kernel (gemm_sm100.cu): persistent CTAs, alone or in pairs on two SMs that share
// one tcgen05.mma, a TMA producer warp, an MMA warp, two TMEM accumulators and eight epilogue warps.  The first CTA's
// producer resolves the tiles that it draws from a counter, from the group table (the row counts are produced by the
// router on the GPU), and hands their coordinates to the other warps and to the other CTA.  Expert weights are read
// through a 3-D tensor map (k, n, expert).  No multicast; bounded waits.
//
// Forward and input gradient are computed transposed: the weights are the M operand (128 rows per CTA, 256 per pair), the
// tokens the N operand, 256 or, at the end of a segment, 128 at a time.  What bounds these products is the fill of
// shared memory from L2, some 65 bytes per cycle and SM.  With tokens as M a tile is 128 tokens (segments are whole
// numbers of 128 rows, often odd ones) x 256 weights, 48 KiB of operands per 512 cycles of MMA; a pair with weights as M
// loads 32 KiB per SM for them.
#include "gemm_sm100.h"

#include <algorithm>

#include "ptx.cuh"

namespace piper {
namespace {

constexpr int BM = 128;              // M rows of a CTA
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int PAD = 128;             // row segments are multiples of this
constexpr int A_STAGE_BYTES = BM * BK * 2;
constexpr int BOX_BYTES = 64 * BK * 2;         // one 64 x 64 box
constexpr int MAX_STAGES = 6;
constexpr int NUM_THREADS = 384;     // TMA, MMA, TMEM-allocation and table warp, then eight epilogue warps
constexpr int MAX_GROUPS = 1024;
constexpr int EPI_WARPS = 8;
// Tiles handed out ahead.  Nothing tells the producer that a slot has been read: every tile has at least one k-block, so
// it waits for a stage before the next one, and is at most the stages + 2 accumulators + 1 ahead of the slowest warp.
constexpr int RING = 16;

template <int MODE, int CTAS>
struct Cfg {
  static constexpr int STAGE_BYTES = A_STAGE_BYTES + BN / CTAS * BK * 2;
  // per epilogue warp: 32 tokens x 32 features, or 32 rows x 128 bytes of a weight gradient
  static constexpr int C_BYTES = MODE == kGroupedWgrad ? 4096 : 2048;
  static constexpr int STAGES = CTAS == 2 ? (MODE == kGroupedWgrad ? 5 : 6) : (MODE == kGroupedWgrad ? 3 : 4);
  static constexpr int C_OFF = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFF = C_OFF + EPI_WARPS * C_BYTES;
  static constexpr int TABLE_OFF = BAR_OFF + 768;       // table[MAX_GROUPS + 1], start[], len[]
  static constexpr int SMEM_BYTES = TABLE_OFF + (3 * MAX_GROUPS + 4) * 4 + 1024;
  static_assert(STAGES <= MAX_STAGES && STAGES + 3 < RING && SMEM_BYTES <= 232448, "shared memory");
};

// What a tile is, as its producer hands it on.
struct __align__(16) Tile {
  int m0;           // first weight row (forward), weight column (input gradient), or row of dW
  int n0;           // first token row, or column of dW
  int expert;       // -1: no more tiles
  int count;        // tokens of the tile, or k-blocks of a weight gradient
};

struct Barriers {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t tile_full[RING];
  Tile tile[RING];
  uint32_t tmem_base;
  int first;         // the first tile of this CTA (or pair)
};
static_assert(sizeof(Barriers) <= 768, "barriers");

struct GroupedParams {
  const int* g_start;    // [G] first row of each group
  const int* g_len;      // [G] padded row count (multiple of 128)
  int num_groups;        // G = sources * experts
  int experts;           // local experts
  int N, K;              // weight shape per expert [N, K]
  int accumulate;
  void* out;
  int* status;
  int* sched;            // next tile, finished CTAs
};

// Measured at 4096 tokens, 128 experts, top 8, 2048 x 768 (two projections each), in tiles of 128 tokens by single CTAs and
// in this form: forward 363 and 314 us, input gradient 360 and 314 us, weight gradient into bf16 479 and 391 us (its
// bytes take 265 us); 777 tokens, 32 experts, top 4, 1024 x 512: 47, 41, 37 and 39, 36, 36 us.
// OUT_BF16 selects the element type of a weight gradient (fp32 buckets accumulate; a bf16 result is stored).
template <int MODE, int CTAS, bool OUT_BF16>
__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const GroupedParams p) {
  using L = Cfg<MODE, CTAS>;
  constexpr int STAGES = L::STAGES;
  constexpr bool A_MN = MODE != kGroupedFwd;           // input gradient: W[e] read along its columns
  constexpr bool B_MN = MODE == kGroupedWgrad;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  Barriers* bars = reinterpret_cast<Barriers*>(smem + L::BAR_OFF);
  // Token tiles before each segment and, behind them, of all; for a weight gradient the experts with rows from the front,
  // those without from the back ([experts - 1] first), and the number with rows in [num_groups].
  int* table = reinterpret_cast<int*>(smem + L::TABLE_OFF);
  int* g_start = table + MAX_GROUPS + 1;
  int* g_len = g_start + MAX_GROUPS;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int rank = CTAS == 2 ? static_cast<int>(cluster_rank()) : 0;
  const int m_size = MODE == kGroupedDgrad ? p.K : p.N;
  const int tiles_m = (m_size + BM * CTAS - 1) / (BM * CTAS);
  const int sources = p.num_groups / p.experts;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bars->acc_full[a], 1);
      mbar_init(&bars->acc_empty[a], EPI_WARPS * CTAS);
    }
    for (int i = 0; i < RING; ++i) mbar_init(&bars->tile_full[i], 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_c);
  }
  if (warp == 3) {
    grid_wait();
    // Token tiles before each segment, in the order q = expert * sources + source (group = source * experts + expert):
    // a warp scan, since one thread walking the table pays a memory latency per group in front of every launch.
    int acc = 0;
#pragma unroll 4
    for (int q0 = 0; q0 < p.num_groups; q0 += 32) {
      const int q = q0 + lane;
      const bool in = q < p.num_groups;
      const int grp = in ? (q % sources) * p.experts + q / sources : 0;
      const int len = in ? p.g_len[grp] / PAD * PAD : 0;
      const int start = in ? p.g_start[grp] : 0;
      const int n = (len + BN - 1) / BN;
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (in) {
        if (MODE != kGroupedWgrad) table[q] = acc + inc - n;
        g_start[grp] = start;
        g_len[grp] = len;
      }
      acc += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (MODE == kGroupedWgrad) {
      __syncwarp();
      acc = 0;
      for (int e0 = 0; e0 < p.experts; e0 += 32) {
        const int e = e0 + lane;
        bool rows = false;
        if (e < p.experts)
          for (int src = 0; src < sources; ++src) rows = rows || g_len[src * p.experts + e] > 0;
        const uint32_t mask = __ballot_sync(0xffffffffu, rows);
        const int before = acc + __popc(mask & ((1u << lane) - 1));
        if (e < p.experts) table[rows ? before : p.experts - 1 - (e - before)] = e;
        acc += __popc(mask);
      }
    }
    if (lane == 0) table[p.num_groups] = acc;
  }
  if (warp == 2) {
    // tiles come from a counter, as in the dense kernel; the first one is drawn beside the table
    tmem_alloc_n<CTAS>(&bars->tmem_base, 512);
    tmem_relinquish_n<CTAS>();
    grid_wait();
    int first = static_cast<int>(blockIdx.x) / CTAS;
    if (rank == 0 && lane == 0 && p.sched != nullptr) first = atomicAdd(&p.sched[0], 1);
    if (lane == 0) bars->first = first;
  }
  grid_wait();
  tc_fence_before();
  if (CTAS == 2) cluster_sync();
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

  // The n-th tile of this CTA (or pair).
  auto tile_at = [&](uint32_t n, Tile& t) -> bool {
    if (!__all_sync(0xffffffffu, mbar_wait(&bars->tile_full[n % RING], (n / RING) & 1, p.status))) return false;
    const int4 v = *reinterpret_cast<const int4*>(&bars->tile[n % RING]);
    t = {v.x, v.y, v.z, v.w};
    return true;
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer (both CTAs of a pair load their own halves)
    const int tiles_n = (p.K + BN - 1) / BN;           // weight gradient
    const int num_tiles = tiles_m * table[p.num_groups] * (MODE == kGroupedWgrad ? tiles_n : 1);
    const int contract_blocks = ((MODE == kGroupedFwd ? p.K : p.N) + BK - 1) / BK;
    uint32_t n = 0, fills = 0, ph = 0;
    int s = 0;
    bool ok = true;
    for (;; ++n) {
      if (rank == 0 && elect_one()) {
        const int units = static_cast<int>(gridDim.x) / CTAS;
        const int i = n > 0 && p.sched != nullptr && num_tiles > units ? atomicAdd(&p.sched[0], 1)
                                                                       : bars->first + static_cast<int>(n) * units;
        Tile t = {0, 0, -1, 0};
        if (i < num_tiles) {
          if (MODE == kGroupedWgrad) {
            // column tiles fastest: the CTAs that run at the same time write whole rows of dW
            const int u = i / tiles_n;
            t.n0 = (i - u * tiles_n) * BN;
            const int j = u / tiles_m;
            t.m0 = (u - j * tiles_m) * BM * CTAS;
            t.expert = table[j];
            for (int src = 0; src < sources; ++src) t.count += g_len[src * p.experts + t.expert] / BK;
          } else {
            const int u = i / tiles_m;
            t.m0 = (i - u * tiles_m) * BM * CTAS;
            // Weight tiles of one token tile are consecutive, and token tiles are walked expert by expert (all sources
            // of an expert together): the CTAs that run at the same time share their tokens and a few experts'
            // weights through L2, so both stream from DRAM once.
            int lo = 0, hi = p.num_groups;             // largest q with table[q] <= u
            while (hi - lo > 1) {
              const int mid = (lo + hi) >> 1;
              if (table[mid] <= u) lo = mid; else hi = mid;
            }
            t.expert = lo / sources;                   // the table is ordered (expert, source)
            const int grp = (lo - t.expert * sources) * p.experts + t.expert;
            const int r0 = (u - table[lo]) * BN;
            t.n0 = g_start[grp] + r0;
            t.count = min(BN, g_len[grp] - r0);
          }
        }
        bars->tile[n % RING] = t;
        if (CTAS == 2)
          st_async_v4(mapa_u32(smem_u32(&bars->tile[n % RING]), 1), mapa_u32(smem_u32(&bars->tile_full[n % RING]), 1),
                      t.m0, t.n0, t.expert, t.count);
        mbar_arrive(&bars->tile_full[n % RING]);
      } else if (rank == 1 && elect_one()) {
        mbar_arrive_expect_tx(&bars->tile_full[n % RING], 16);
      }
      __syncwarp();
      Tile t;
      if (!(ok = tile_at(n, t)) || t.expert < 0) break;
      const int m0 = t.m0 + rank * BM;
      const int b_rows = (MODE == kGroupedWgrad ? BN : t.count) / CTAS;      // tokens (or dW columns) this CTA loads
      const int n0 = t.n0 + rank * b_rows;
      const uint32_t bytes = CTAS * (A_STAGE_BYTES + b_rows * BK * 2);
      int seg = 0, seg_row = 0;                        // weight gradient: current segment and row in it
      const int blocks = MODE == kGroupedWgrad ? t.count : contract_blocks;
      for (int kb = 0; kb < blocks; ++kb) {
        if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->empty[s], ph ^ 1, p.status)))) break;
        int k0 = kb * BK;
        if (MODE == kGroupedWgrad) {
          while (seg_row >= g_len[seg * p.experts + t.expert]) {
            ++seg;
            seg_row = 0;
          }
          k0 = g_start[seg * p.experts + t.expert] + seg_row;
          seg_row += BK;
        }
        if (elect_one()) {
          uint8_t* sa = smem + s * L::STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(&bars->full[s], bytes);
          if (MODE == kGroupedFwd) {
            tma_load_3d_n<CTAS>(sa, &tmap_a, &bars->full[s], k0, m0, t.expert);
          } else if (MODE == kGroupedDgrad) {
            tma_load_3d_n<CTAS>(sa, &tmap_a, &bars->full[s], m0, k0, t.expert);
            tma_load_3d_n<CTAS>(sa + BOX_BYTES, &tmap_a, &bars->full[s], m0 + 64, k0, t.expert);
          } else {
            tma_load_2d_n<CTAS>(sa, &tmap_a, &bars->full[s], m0, k0);
            tma_load_2d_n<CTAS>(sa + BOX_BYTES, &tmap_a, &bars->full[s], m0 + 64, k0);
          }
          for (int j = 0; j < b_rows / 64; ++j)
            tma_load_2d_n<CTAS>(sb + j * BOX_BYTES, &tmap_b, &bars->full[s], B_MN ? n0 + 64 * j : k0,
                                B_MN ? k0 : n0 + 64 * j);
        }
        __syncwarp();
        ++fills;
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (!ok) break;
    }
    grid_launch();                                     // the last loads are on their way
    if (ok) {
      // every stage handed back before the CTA may leave: no commit is still on its way to these barriers
      for (int i = 0; i < STAGES && ok; ++i) {
        ok = mbar_wait(&bars->empty[s], ph ^ 1, p.status);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    } else if (rank == 0) {
      for (int i = 0; i < STAGES; ++i) {               // let the copies already issued land
        if (fills <= static_cast<uint32_t>(i)) continue;
        mbar_wait(&bars->full[i], ((fills - 1 - i) / STAGES) & 1, nullptr);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer (first CTA of a pair, for both)
    // uniform control flow, one elected lane issues
    if (rank == 0) {
      const uint64_t da0 = umma_desc_sw128(smem_u32(smem), A_MN ? BOX_BYTES : 16, 1024);
      const uint64_t db0 = umma_desc_sw128(smem_u32(smem) + A_STAGE_BYTES, B_MN ? BOX_BYTES : 16, 1024);
      constexpr int a_step = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      constexpr int b_step = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      const int contract_blocks = ((MODE == kGroupedFwd ? p.K : p.N) + BK - 1) / BK;
      uint32_t ph = 0;
      int s = 0;
      bool ok = true;
      for (uint32_t n = 0; ok; ++n) {
        Tile t;
        if (!(ok = tile_at(n, t)) || t.expert < 0) break;
        const int blocks = MODE == kGroupedWgrad ? t.count : contract_blocks;
        const uint32_t idesc = umma_idesc_bf16(BM * CTAS, MODE == kGroupedWgrad ? BN : t.count, A_MN, B_MN);
        const uint32_t acc = n & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_empty[acc], ((n >> 1) & 1) ^ 1, p.status));
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = 0; kb < blocks && ok; ++kb) {
          if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->full[s], ph, p.status)))) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t da = da0 + (s * L::STAGE_BYTES >> 4), db = db0 + (s * L::STAGE_BYTES >> 4);
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16_ss_n<CTAS>(tmem_d, da + k * a_step, db + k * b_step, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit_n<CTAS>(&bars->empty[s]);
            if (kb == blocks - 1) umma_commit_n<CTAS>(&bars->acc_full[acc]);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------- epilogue
    const int q = warp & 3;                     // TMEM lanes [32q, 32q + 32)
    const int half = (warp - 4) >> 2;           // odd or even column chunks
    uint8_t* const blk = smem + L::C_OFF + (warp - 4) * L::C_BYTES;
    for (uint32_t n = 0;; ++n) {
      Tile t;
      if (!tile_at(n, t) || t.expert < 0) break;
      const int row0 = t.m0 + rank * BM + q * 32;
      const uint32_t acc = n & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->acc_full[acc], (n >> 1) & 1, p.status))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
      if (MODE == kGroupedWgrad) {
        // a warp's 32 rows x 128 bytes at a time through a swizzled block and a TMA store (fp32 accumulation: a TMA
        // reduce-add, C is never read by the SM); the tensor map clips ragged edges
        constexpr int COLS = OUT_BF16 ? 64 : 32;
#pragma unroll 1
        for (int c = half; c < BN / COLS; c += 2) {
          const int col0 = t.n0 + c * COLS;
          if (col0 >= p.K || row0 >= p.N) break;
          uint4 v16[8];
#pragma unroll
          for (int h = 0; h < COLS / 32; ++h) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + c * COLS + h * 32, r);
            tmem_ld_wait();
            if (OUT_BF16) {
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                uint32_t* o = reinterpret_cast<uint32_t*>(&v16[h * 4 + v]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  o[i] = pack_bf16x2(__uint_as_float(r[8 * v + 2 * i]), __uint_as_float(r[8 * v + 2 * i + 1]));
              }
            } else {
#pragma unroll
              for (int v = 0; v < 8; ++v) v16[v] = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
            }
          }
          if (lane == 0) bulk_wait_group_read<0>();      // the previous block has left the buffer
          __syncwarp();
#pragma unroll
          for (int v = 0; v < 8; ++v) reinterpret_cast<uint4*>(blk + lane * 128)[v ^ (lane & 7)] = v16[v];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (p.accumulate) tma_reduce_add_3d_bulk(&tmap_c, blk, col0, row0, t.expert);
            else tma_store_3d_bulk(&tmap_c, blk, col0, row0, t.expert);
            bulk_commit_group();
          }
        }
      } else if (row0 < m_size) {
        // Lanes are features, registers tokens: a feature is stored per lane, a token's 32 features as one 64-byte row
        // of the block (no bank conflicts), and the block leaves as a TMA store that clips the last features.
#pragma unroll 1
        for (int c = half; c < t.count / 32; c += 2) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
          if (lane == 0) bulk_wait_group_read<0>();      // the previous block has left the buffer
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            reinterpret_cast<__nv_bfloat16*>(blk)[i * 32 + lane] = __float2bfloat16(__uint_as_float(r[i]));
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d_bulk(&tmap_c, blk, row0, t.n0 + c * 32, 0);
            bulk_commit_group();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTAS == 2) mbar_arrive_cluster(mapa_u32(smem_u32(&bars->acc_empty[acc]), 0));
        else mbar_arrive(&bars->acc_empty[acc]);
      }
    }
    if (lane == 0) bulk_wait_group<0>();         // staged blocks leave before the CTA does
  } else if (MODE == kGroupedWgrad && !p.accumulate) {
    // -------------------------------- experts without rows: their gradients are zero, written beside the other tiles
    const long long vecs = static_cast<long long>(p.N) * p.K * (OUT_BF16 ? 2 : 4) / 16;      // K is a multiple of 8
    for (int j = table[p.num_groups]; j < p.experts; ++j) {
      uint4* dst = static_cast<uint4*>(p.out) + table[j] * vecs;
      for (long long i = (blockIdx.x * 2 + warp - 2) * 32 + lane; i < vecs; i += gridDim.x * 64)
        dst[i] = make_uint4(0, 0, 0, 0);
    }
  }

  tc_fence_before();
  if (CTAS == 2) cluster_sync();
  else __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_n<CTAS>(tmem_base, 512);
  }
  if (p.sched != nullptr && threadIdx.x == 0) {
    if (atomicAdd(&p.sched[1], 1) == static_cast<int>(gridDim.x) - 1) {   // last CTA rearms the scheduler slot
      p.sched[0] = 0;
      p.sched[1] = 0;
      __threadfence();
    }
  }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

int make_tmap_3d(CUtensorMap* out, const void* base, uint64_t d0, uint64_t d1, uint64_t d2,
                 uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1,
                 CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                 CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  static EncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return -1;
    fn = reinterpret_cast<EncodeFn>(ptr);
  }
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(nullptr);
    ctx_bound = true;
  }
  const cuuint64_t dims[3] = {d0, d1, d2};
  const cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
  const cuuint32_t box[3] = {b0, b1, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r =
      fn(out, type, 3, const_cast<void*>(base), dims, strides, box, estr,
         CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

template <int MODE, int CTAS, bool OUT_BF16>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GroupedParams& p, int num_sms,
           cudaStream_t st) {
  auto kern = grouped_gemm_kernel<MODE, CTAS, OUT_BF16>;
  constexpr int smem = Cfg<MODE, CTAS>::SMEM_BYTES;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -2;
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(num_sms / CTAS * CTAS));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = CTAS;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = CTAS > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, ta, tb, tc, p) == cudaSuccess ? 0 : -3;
}

}  // namespace

// CTAs per tile: pairs wherever the tiles go round them (the launch knows the row buffer's size, not the segments'), single
// CTAs below, which cover twice as many SMs.  One and two per tile at 4096 tokens, 64 experts, top 8, 2048 x 768: forward 304
// and 273 us, weight gradient 350 and 296 us; at 4096 tokens, 8 experts, top 2, 256 x 256: 15.4 and 16.7 us, 27.0 and 28.1 us.
static bool by_pairs(const GroupedGemmArgs& g, int num_sms) {
  const long long m_tiles = ((g.mode == kGroupedDgrad ? g.K : g.N) + 2 * BM - 1) / (2 * BM);
  const long long rows = std::max<long long>(g.num_groups, g.rows_capacity / BN);
  const long long n_tiles = g.mode == kGroupedWgrad ? static_cast<long long>(g.experts) * ((g.K + BN - 1) / BN) : rows;
  return num_sms >= 2 && m_tiles * n_tiles >= num_sms / 2;
}

int grouped_gemm_launch(const GroupedGemmArgs& g, int num_sms, cudaStream_t st) {
  if (g.num_groups <= 0 || g.num_groups > MAX_GROUPS || g.experts <= 0 || g.num_groups % g.experts != 0) return -11;
  if (g.N % 8 != 0 || g.K % 8 != 0 || g.rows_capacity < 0) return -12;
  if (g.rows_capacity == 0) {
    // A rank can receive no rows at all (every token routed to experts of other ranks): nothing to multiply.
    // The weight gradient of such a step is zero.
    if (g.mode == kGroupedWgrad && !g.accumulate) {
      const size_t bytes = static_cast<size_t>(g.experts) * g.N * g.K * (g.out_bf16 ? 2 : 4);
      if (cudaMemsetAsync(g.out, 0, bytes, st) != cudaSuccess) return -3;
    }
    return 0;
  }
  GroupedParams p;
  p.g_start = g.g_start;
  p.g_len = g.g_len;
  p.num_groups = g.num_groups;
  p.experts = g.experts;
  p.N = g.N;
  p.K = g.K;
  p.accumulate = g.accumulate;
  p.out = g.out;
  p.status = g.status;
  p.sched = gemm_sched_slot();
  CUtensorMap ta, tb, tc;
  int rc;
  const uint64_t R = static_cast<uint64_t>(g.rows_capacity);
  const uint64_t N = g.N, K = g.K, E = g.experts;
  const bool pair = by_pairs(g, num_sms);
  if (g.mode == kGroupedFwd) {
    // A = W [E, N, K] K-major; B = X [R, K] K-major; C = Y [R, N]
    if ((rc = make_tmap_3d(&ta, g.w, K, N, E, K * 2, N * K * 2, BK, BM)) != 0) return rc;
    if ((rc = make_tmap_2d_bf16(&tb, g.x, K, R, K * 2, BK, 64)) != 0) return rc;
    if ((rc = make_tmap_3d(&tc, g.out, N, R, 1, N * 2, R * N * 2, 32, 32, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                           CU_TENSOR_MAP_SWIZZLE_NONE)) != 0)
      return rc;
    return pair ? launch<kGroupedFwd, 2, true>(ta, tb, tc, p, num_sms, st)
                : launch<kGroupedFwd, 1, true>(ta, tb, tc, p, num_sms, st);
  }
  if (g.mode == kGroupedDgrad) {
    // A = W [E, N, K] read MN-major (rows along K, contraction over N); B = dY [R, N] K-major; C = dX [R, K]
    if ((rc = make_tmap_3d(&ta, g.w, K, N, E, K * 2, N * K * 2, 64, BK)) != 0) return rc;
    if ((rc = make_tmap_2d_bf16(&tb, g.dy, N, R, N * 2, BK, 64)) != 0) return rc;
    if ((rc = make_tmap_3d(&tc, g.out, K, R, 1, K * 2, R * K * 2, 32, 32, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                           CU_TENSOR_MAP_SWIZZLE_NONE)) != 0)
      return rc;
    return pair ? launch<kGroupedDgrad, 2, true>(ta, tb, tc, p, num_sms, st)
                : launch<kGroupedDgrad, 1, true>(ta, tb, tc, p, num_sms, st);
  }
  // wgrad: A = dY [R, N] MN-major, B = X [R, K] MN-major, C = dW [E, N, K] fp32 or bf16
  if ((rc = make_tmap_2d_bf16(&ta, g.dy, N, R, N * 2, 64, BK)) != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&tb, g.x, K, R, K * 2, 64, BK)) != 0) return rc;
  const uint64_t es = g.out_bf16 ? 2 : 4;
  if ((rc = make_tmap_3d(&tc, g.out, K, N, E, K * es, N * K * es, 128 / es, 32,
                         g.out_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32)) != 0)
    return rc;
  if (g.out_bf16)
    return pair ? launch<kGroupedWgrad, 2, true>(ta, tb, tc, p, num_sms, st)
                : launch<kGroupedWgrad, 1, true>(ta, tb, tc, p, num_sms, st);
  return pair ? launch<kGroupedWgrad, 2, false>(ta, tb, tc, p, num_sms, st)
              : launch<kGroupedWgrad, 1, false>(ta, tb, tc, p, num_sms, st);
}

}  // namespace piper
