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
// The structure is that of the dense kernel (gemm_sm100.cu): persistent
// CTAs, TMA producer warp, tcgen05.mma issued by one elected lane of a warp
// that walks the loop uniformly, two TMEM accumulators, eight epilogue warps;
// the tile -> coordinate mapping is computed on the device from the group
// table, because the row counts are produced by the router on the GPU.  Expert weights are read
// through a 3-D tensor map (k, n, expert).  No multicast; bounded waits.
#include "gemm_sm100.h"
#include "ptx.cuh"

namespace piper {
namespace {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;
constexpr int B_STAGE_BYTES = BN * BK * 2;
constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
constexpr int MN_BOX_BYTES = 64 * BK * 2;
constexpr int NUM_THREADS = 384;     // TMA, MMA, TMEM-allocation and one idle warp, then eight epilogue warps
constexpr int MAX_GROUPS = 1024;
constexpr int EPI_WARPS = 8;
constexpr int C_STAGE_BYTES = 4096;  // weight gradients: one 32-row x 128-byte block per epilogue warp

// The weight gradient contracts over few rows (a few k-blocks per tile) and writes far more than it reads, so it
// trades one operand stage for staging blocks that leave as TMA stores.
template <int MODE>
struct Cfg {
  static constexpr int STAGES = MODE == kGroupedWgrad ? 3 : 4;
  static constexpr int C_OFF = STAGES * STAGE_BYTES;
  static constexpr int BAR_OFF = C_OFF + (MODE == kGroupedWgrad ? EPI_WARPS * C_STAGE_BYTES : 0);
  static constexpr int TABLE_OFF = BAR_OFF + 256;       // tile_prefix[MAX_GROUPS + 1], start[], len[]
  static constexpr int SMEM_BYTES = TABLE_OFF + (3 * MAX_GROUPS + 4) * 4 + 1024;
};

struct Barriers {
  uint64_t full[4];
  uint64_t empty[4];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
};

struct GroupedParams {
  const int* g_start;    // [G] first row of each group
  const int* g_len;      // [G] padded row count (multiple of 128)
  int num_groups;        // G = sources * experts
  int experts;           // local experts
  int N, K;              // weight shape per expert [N, K]
  void* c;               // output (fwd / dgrad)
  long long ldc;
  int accumulate;
  int* status;
};

// Tile descriptor resolved from a linear tile index.
struct Tile {
  int m0, n0;       // output coordinates (rows / weight-N for wgrad, cols)
  int expert;
  int group;        // row group (fwd/dgrad)
  bool valid;
};

template <int MODE>
__device__ __forceinline__ Tile resolve_tile(int t, const int* tile_prefix, const GroupedParams& p,
                                             const int* start, int tiles_n) {
  Tile r;
  r.valid = true;
  if (MODE == kGroupedWgrad) {
    const int tiles_m = (p.N + BM - 1) / BM;
    const int per_expert = tiles_m * tiles_n;
    r.expert = t / per_expert;
    const int rem = t % per_expert;
    r.m0 = (rem % tiles_m) * BM;
    r.n0 = (rem / tiles_m) * BN;
    r.group = 0;
    return r;
  }
  // Column tiles of one row tile are consecutive, and row tiles are walked expert by expert (all sources of an
  // expert together): the CTAs of a wave share their A tiles and a few experts' weights through L2, so both
  // operands stream from DRAM once.  (Row tiles fastest re-read every row once per column tile.)
  const int mt = t / tiles_n;
  r.n0 = (t % tiles_n) * BN;
  int lo = 0, hi = p.num_groups;          // largest q with tile_prefix[q] <= mt
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_prefix[mid] <= mt) lo = mid; else hi = mid;
  }
  const int sources = p.num_groups / p.experts;
  r.expert = lo / sources;                 // tile_prefix is ordered (expert, source)
  r.group = (lo % sources) * p.experts + r.expert;
  r.m0 = start[r.group] + (mt - tile_prefix[lo]) * BM;
  return r;
}

// Measured at 4096 tokens, 128 experts, top 8, 2048 x 768 (two projections each): forward 378 -> 361 us and input
// gradient 377 -> 357 us with the group table scanned by a warp; weight gradient 473 us into bf16, against 1206 us for
// direct fp32 stores plus 836 us that cleared and converted the fp32 tensor.  No unit is above 62 % busy (64 experts,
// top 4); what fills the rest has not been measured.
// OUT_BF16 selects the element type of a weight gradient (fp32 buckets accumulate; a bf16 result is stored).
template <int MODE, bool OUT_BF16>
__global__ void __launch_bounds__(NUM_THREADS, 1)
grouped_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const GroupedParams p) {
  constexpr int STAGES = Cfg<MODE>::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  Barriers* bars = reinterpret_cast<Barriers*>(smem + Cfg<MODE>::BAR_OFF);
  int* tile_prefix = reinterpret_cast<int*>(smem + Cfg<MODE>::TABLE_OFF);
  int* g_start = tile_prefix + MAX_GROUPS + 1;
  int* g_len = g_start + MAX_GROUPS;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  constexpr bool A_MN = (MODE == kGroupedWgrad);
  constexpr bool B_MN = (MODE != kGroupedFwd);
  const int out_cols = (MODE == kGroupedFwd) ? p.N : p.K;       // columns of the output matrix
  const int contract = (MODE == kGroupedFwd) ? p.K : p.N;       // contraction length (fwd / dgrad)
  const int tiles_n = (out_cols + BN - 1) / BN;
  const int sources = p.num_groups / p.experts;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bars->full[s], 1);
      mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bars->acc_full[a], 1);
      mbar_init(&bars->acc_empty[a], 8);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 3) {
    // Row tiles before each segment, in the order q = expert * sources + source (group = source * experts + expert):
    // a warp scan, since one thread walking the table pays a memory latency per group in front of every launch.
    int acc = 0;
#pragma unroll 4
    for (int q0 = 0; q0 < p.num_groups; q0 += 32) {
      const int q = q0 + lane;
      const bool in = q < p.num_groups;
      const int grp = in ? (q % sources) * p.experts + q / sources : 0;
      const int len = in ? p.g_len[grp] : 0;
      const int start = in ? p.g_start[grp] : 0;
      const int n = len / BM;
      int inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (in) {
        tile_prefix[q] = acc + inc - n;
        g_start[grp] = start;
        g_len[grp] = len;
      }
      acc += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) tile_prefix[p.num_groups] = acc;
  }
  if (warp == 2) {
    tmem_alloc(&bars->tmem_base, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  const int total_m_tiles = tile_prefix[p.num_groups];
  const int num_tiles = (MODE == kGroupedWgrad) ? p.experts * ((p.N + BM - 1) / BM) * tiles_n
                                                : total_m_tiles * tiles_n;

  // Number of 64-deep k-blocks of a tile.
  auto k_blocks_of = [&](const Tile& t) -> int {
    if (MODE != kGroupedWgrad) return (contract + BK - 1) / BK;
    int n = 0;
    for (int s = 0; s < sources; ++s) n += g_len[s * p.experts + t.expert] / BK;
    return n;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int ti = blockIdx.x; ti < num_tiles && ok; ti += gridDim.x) {
        const Tile t = resolve_tile<MODE>(ti, tile_prefix, p, g_start, tiles_n);
        auto issue = [&](int a_x, int a_y, int b_x, int b_y) -> bool {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&bars->empty[s], ph ^ 1, p.status)) return false;
          uint8_t* sa = smem + s * STAGE_BYTES;
          uint8_t* sb = sa + A_STAGE_BYTES;
          mbar_arrive_expect_tx(&bars->full[s], STAGE_BYTES);
          if (A_MN) {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              tma_load_2d(sa + j * MN_BOX_BYTES, &tmap_a, &bars->full[s], a_x + 64 * j, a_y);
          } else {
            tma_load_2d(sa, &tmap_a, &bars->full[s], a_x, a_y);
          }
          if (MODE == kGroupedFwd) {
            tma_load_3d(sb, &tmap_b, &bars->full[s], b_x, b_y, t.expert);
          } else if (MODE == kGroupedDgrad) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_3d(sb + j * MN_BOX_BYTES, &tmap_b, &bars->full[s], b_x + 64 * j, b_y, t.expert);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_2d(sb + j * MN_BOX_BYTES, &tmap_b, &bars->full[s], b_x + 64 * j, b_y);
          }
          ++it;
          return true;
        };
        if (MODE == kGroupedWgrad) {
          for (int s = 0; s < sources && ok; ++s) {
            const int g = s * p.experts + t.expert;
            const int r0 = g_start[g], len = g_len[g];
            for (int r = 0; r < len && ok; r += BK) ok = issue(t.m0, r0 + r, t.n0, r0 + r);
          }
        } else {
          const int kb = (contract + BK - 1) / BK;
          for (int k = 0; k < kb && ok; ++k) {
            // fwd:   A[x=k, y=row], B[x=k, y=n, z=e]
            // dgrad: A[x=k(contraction over N), y=row], B[x=out col, y=k, z=e]
            ok = (MODE == kGroupedFwd) ? issue(k * BK, t.m0, k * BK, t.n0) : issue(k * BK, t.m0, t.n0, k * BK);
          }
        }
      }
      if (!ok) {
        for (int s = 0; s < STAGES; ++s) {
          if (it <= static_cast<uint32_t>(s)) continue;
          const uint32_t fills = (it - 1 - s) / STAGES + 1;
          mbar_wait(&bars->full[s], (fills - 1) & 1, nullptr);
        }
      }
    }
  } else if (warp == 1) {
    // uniform control flow, one elected lane issues
    constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, A_MN, B_MN);
    const uint64_t da0 = A_MN ? umma_desc_sw128(smem_u32(smem), MN_BOX_BYTES, 1024)
                              : umma_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t db0 = B_MN ? umma_desc_sw128(smem_u32(smem) + A_STAGE_BYTES, MN_BOX_BYTES, 1024)
                              : umma_desc_sw128(smem_u32(smem) + A_STAGE_BYTES, 16, 1024);
    constexpr int a_step = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
    constexpr int b_step = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
    uint32_t local_tile = 0, ph = 0;
    int s = 0;
    bool ok = true;
    for (int ti = blockIdx.x; ti < num_tiles && ok; ti += gridDim.x) {
      const Tile t = resolve_tile<MODE>(ti, tile_prefix, p, g_start, tiles_n);
      const int kb_total = k_blocks_of(t);
      if (kb_total == 0) continue;
      const int acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      ++local_tile;
      ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_empty[acc], acc_ph ^ 1, p.status));
      const uint32_t tmem_d = tmem_base + acc * BN;
      for (int kb = 0; kb < kb_total && ok; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bars->full[s], ph, p.status));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t da = da0 + (s * STAGE_BYTES >> 4), db = db0 + (s * STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_ss(tmem_d, da + k * a_step, db + k * b_step, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit(&bars->empty[s]);
          if (kb == kb_total - 1) umma_commit(&bars->acc_full[acc]);
        }
        __syncwarp();
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3;                     // TMEM lanes [32q, 32q + 32)
    const int ch = (warp - 4) >> 2;             // columns [128ch, 128ch + 128) of the tile
    uint32_t local_tile = 0;
    bool ok = true;
    for (int ti = blockIdx.x; ti < num_tiles && ok; ti += gridDim.x) {
      const Tile t = resolve_tile<MODE>(ti, tile_prefix, p, g_start, tiles_n);
      const int kb_total = k_blocks_of(t);
      const int row = t.m0 + q * 32 + lane;
      // expert without rows: nothing to add; a non-accumulating output tile is zero
      if (kb_total == 0 && (MODE != kGroupedWgrad || p.accumulate)) continue;
      const int acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      if (kb_total > 0) {
        ++local_tile;
        if (!__all_sync(0xffffffffu, mbar_wait(&bars->acc_full[acc], acc_ph, p.status))) { ok = false; break; }
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN + ch * 128;
      if (MODE == kGroupedWgrad) {
        // a warp's 32 rows x 128 bytes at a time through a swizzled block and a TMA store (fp32 accumulation: a TMA
        // reduce-add, C is never read by the SM); the tensor map clips ragged edges
        uint8_t* cbuf = smem + Cfg<MODE>::C_OFF + (warp - 4) * C_STAGE_BYTES;
        constexpr int COLS = OUT_BF16 ? 64 : 32;
#pragma unroll 1
        for (int c = 0; c < 128 / COLS; ++c) {
          const int col0 = t.n0 + ch * 128 + c * COLS;
          if (col0 >= out_cols || t.m0 + q * 32 >= p.N) break;
          uint4 blk[8];
#pragma unroll
          for (int h = 0; h < COLS / 32; ++h) {
            uint32_t r[32];
            if (kb_total > 0) {
              tmem_ld_32x32(taddr + c * COLS + h * 32, r);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = 0;
            }
            if (OUT_BF16) {
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                uint32_t* o = reinterpret_cast<uint32_t*>(&blk[h * 4 + v]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  o[i] = pack_bf16x2(__uint_as_float(r[8 * v + 2 * i]), __uint_as_float(r[8 * v + 2 * i + 1]));
              }
            } else {
#pragma unroll
              for (int v = 0; v < 8; ++v) blk[v] = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
            }
          }
          if (lane == 0) bulk_wait_group_read<0>();      // the previous block has left the buffer
          __syncwarp();
#pragma unroll
          for (int v = 0; v < 8; ++v) reinterpret_cast<uint4*>(cbuf + lane * 128)[v ^ (lane & 7)] = blk[v];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (p.accumulate) tma_reduce_add_3d_bulk(&tmap_c, cbuf, col0, t.m0 + q * 32, t.expert);
            else tma_store_3d_bulk(&tmap_c, cbuf, col0, t.m0 + q * 32, t.expert);
            bulk_commit_group();
          }
        }
        if (kb_total == 0) continue;
      } else {
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
          const int col0 = t.n0 + ch * 128 + c * 32;
          if (col0 >= out_cols) continue;
          __nv_bfloat16* crow = reinterpret_cast<__nv_bfloat16*>(p.c) + row * p.ldc + col0;
          if (col0 + 32 <= out_cols) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(r[8 * v + 0]), __uint_as_float(r[8 * v + 1]));
              o.y = pack_bf16x2(__uint_as_float(r[8 * v + 2]), __uint_as_float(r[8 * v + 3]));
              o.z = pack_bf16x2(__uint_as_float(r[8 * v + 4]), __uint_as_float(r[8 * v + 5]));
              o.w = pack_bf16x2(__uint_as_float(r[8 * v + 6]), __uint_as_float(r[8 * v + 7]));
              reinterpret_cast<uint4*>(crow)[v] = o;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)        // constant indices keep r[] in registers
              if (col0 + j < out_cols) crow[j] = __float2bfloat16(__uint_as_float(r[j]));
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->acc_empty[acc]);
    }
    if (MODE == kGroupedWgrad && lane == 0) bulk_wait_group<0>();   // staged blocks leave before the CTA does
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

int make_tmap_3d(CUtensorMap* out, const void* base, uint64_t d0, uint64_t d1, uint64_t d2,
                      uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1,
                      CUtensorMapDataType type = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16) {
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
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

template <int MODE, bool OUT_BF16>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GroupedParams& p, int num_sms,
           cudaStream_t st) {
  auto kern = grouped_gemm_kernel<MODE, OUT_BF16>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<MODE>::SMEM_BYTES) != cudaSuccess)
      return -2;
    configured = true;
  }
  kern<<<num_sms, NUM_THREADS, Cfg<MODE>::SMEM_BYTES, st>>>(ta, tb, tc, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace

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
  p.c = g.out;
  p.accumulate = g.accumulate;
  p.status = g.status;
  CUtensorMap ta, tb;
  int rc;
  const uint64_t R = static_cast<uint64_t>(g.rows_capacity);
  const uint64_t N = g.N, K = g.K, E = g.experts;
  if (g.mode == kGroupedFwd) {
    // A = X [R, K] K-major; B = W [E, N, K] K-major; C = Y [R, N]
    if ((rc = make_tmap_2d_bf16(&ta, g.x, K, R, K * 2, BK, BM)) != 0) return rc;
    if ((rc = make_tmap_3d(&tb, g.w, K, N, E, K * 2, N * K * 2, BK, BN)) != 0) return rc;
    p.ldc = g.N;
    return launch<kGroupedFwd, true>(ta, tb, ta, p, num_sms, st);
  }
  if (g.mode == kGroupedDgrad) {
    // A = dY [R, N] K-major (contraction N); B = W [E, N, K] read MN-major; C = dX [R, K]
    if ((rc = make_tmap_2d_bf16(&ta, g.dy, N, R, N * 2, BK, BM)) != 0) return rc;
    if ((rc = make_tmap_3d(&tb, g.w, K, N, E, K * 2, N * K * 2, 64, BK)) != 0) return rc;
    p.ldc = g.K;
    return launch<kGroupedDgrad, true>(ta, tb, ta, p, num_sms, st);
  }
  // wgrad: A = dY [R, N] MN-major, B = X [R, K] MN-major, C = dW [E, N, K] fp32 or bf16
  if ((rc = make_tmap_2d_bf16(&ta, g.dy, N, R, N * 2, 64, BK)) != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&tb, g.x, K, R, K * 2, 64, BK)) != 0) return rc;
  CUtensorMap tc;
  const uint64_t es = g.out_bf16 ? 2 : 4;
  if ((rc = make_tmap_3d(&tc, g.out, K, N, E, K * es, N * K * es, 128 / es, 32,
                         g.out_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32)) != 0)
    return rc;
  p.ldc = g.K;
  return g.out_bf16 ? launch<kGroupedWgrad, true>(ta, tb, tc, p, num_sms, st)
                    : launch<kGroupedWgrad, false>(ta, tb, tc, p, num_sms, st);
}

}  // namespace piper
