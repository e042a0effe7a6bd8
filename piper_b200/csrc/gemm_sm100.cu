// Dense bf16 GEMM for sm_100a: C[M,N] = A[M,K] * B[N,K]^T with fp32
// accumulation in tensor memory.
//
// Persistent CTAs walk output tiles of 128 rows and a width chosen per launch (32 to 256 columns), either each CTA
// by itself or in pairs on two neighbouring SMs (tcgen05 cta_group::2: 256-row tiles, each CTA holds 128 rows of A and
// half of B's rows in shared memory, its tensor memory takes its 128 rows of C).  Roles by warp:
//   warp 0      TMA producer: fills a ring of shared-memory stages with 128-byte-swizzled operand tiles
//               (cp.async.bulk.tensor, no multicast); the first CTA of a pair also hands out the tiles.
//   warp 1      MMA issuer (first CTA of a pair, for both): tcgen05.mma into one of two 256-column accumulators.
//               The warp walks the loop uniformly and one elected lane issues: in a single-lane branch every descriptor
//               has to be moved into uniform registers, about 100 cycles per MMA.
//   warp 2      TMEM allocator / deallocator.
//   warps 4-11  epilogue: tcgen05.ld of the finished accumulator, conversion, staging in shared memory, TMA store (or
//               TMA reduce-add), while the MMAs of the next tile run in the other accumulator.
//
// What bounds it: an SM fills shared memory from L2 at about 65 bytes per cycle while it multiplies (see gemm_cost).  A
// k-block of a 128 x w tile is (128 + w) x 128 bytes for 2w cycles of MMA, 756 cycles of fill against 512 at w = 256; in a
// pair each SM loads half of B's rows, (128 + w / 2) x 128 bytes, 504 cycles of fill, and reads half as much of B from
// shared memory.
//
// Each operand can be K-major (contraction index contiguous in memory) or
// MN-major (row index contiguous), which covers forward (X W^T), input
// gradient (dY W) and weight gradient (dY^T X) of a linear layer without any
// transposed copy.  The epilogue either stores bf16 or adds into an fp32
// buffer (gradient accumulation into the flat fp32 bucket).  Every output element is the sum of the same products in
// the same order whatever the tile shape, so results do not depend on it, except where a gradient's contraction is split
// (gemm_split_shape).
//
// All mbarrier waits are bounded; on expiry the kernel records a status code,
// drains its TMA copies, frees TMEM and returns.
#include "gemm_sm100.h"

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdlib>

#include "ptx.cuh"

namespace piper {
namespace {

constexpr int BM = 128;                        // rows of a CTA
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;
constexpr int MN_BOX_BYTES = 64 * BK * 2;
constexpr int MAX_STAGES = 8;
constexpr int OPERAND_BYTES = 196608;          // 4 stages of 128 x 256 operands, 6 of a CTA pair
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 128 + 32 * EPI_WARPS;
constexpr int C_STAGE_BYTES = 4096;            // per epilogue warp: two bf16 or one fp32 block of 32 x 32
constexpr int BAR_OFF = OPERAND_BYTES + EPI_WARPS * C_STAGE_BYTES;
constexpr int SMEM_BYTES = BAR_OFF + 768 + 1024;
constexpr int RING = 16;                       // tiles handed out ahead: at most the stages + 2 accumulators + 1

struct Bars {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t tile_full[RING];
  int tile[RING][4];         // the tile's number in the first word
  uint32_t tmem_base;
  int first;                 // the first tile of this CTA (or pair)
};
static_assert(sizeof(Bars) <= 768 && offsetof(Bars, tile) % 16 == 0 && SMEM_BYTES <= 232448, "shared memory");

struct Params {
  int M, N, K;
  int width;          // columns of a tile
  int stages;
  int accumulate;
  int c_bufs;         // staging buffers per epilogue warp; the second ones take the room of operand stages
  int band;           // tiles of the faster dimension that are walked together
  int splits;         // parts of the contraction, each a tile of its own
  int k_per;          // k-blocks of a part
  int split_rows;     // rows between the parts' outputs
  int* status;
  int* sched;
};

template <int CTAS, bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                 const __grid_constant__ CUtensorMap tmap_c, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  Bars* bars = reinterpret_cast<Bars*>(smem + BAR_OFF);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const uint32_t rank = CTAS == 2 ? cluster_rank() : 0;
  const int width = p.width;
  const int b_rows = width / CTAS;                                       // rows of B that this CTA loads
  const int b_boxes = (b_rows + 63) / 64;
  const int stage_bytes = A_STAGE_BYTES + (B_MN ? b_boxes * MN_BOX_BYTES : b_rows * BK * 2);
  const int stages = p.stages;
  const int tiles_m = (p.M + BM * CTAS - 1) / (BM * CTAS);
  const int tiles_n = (p.N + width - 1) / width;
  const int out_tiles = tiles_m * tiles_n;
  const int num_tiles = out_tiles * p.splits;
  const int k_blocks = (p.K + BK - 1) / BK;
  const bool n_fast = tiles_n < tiles_m;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_STAGES; ++s) {
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
  if (warp == 2) {
    tmem_alloc_n<CTAS>(&bars->tmem_base, 512);
    tmem_relinquish_n<CTAS>();
  }
  // Tiles come from a counter, so that none waits for a CTA that finds no SM until others are done: beside a kernel that
  // holds 16 SMs, with the CTA's own number as the first tile and so, 4096 x 8192 x 1024 65.3 and 58.9 us, 4096 x 14336 x 4096 297 and
  // 289 us; alone 54.6 and 54.4, 254 and 253 us.  The first draw runs beside the allocation, but behind the wait, as every access
  // to global memory does (in front of it no pass is faster by more than its runs differ).  In a launch of one round a CTA
  // that comes late has as much to do as one that draws twice; there every CTA takes its number (512 x 256 x 688 6.5 us, with
  // the counter 6.9).
  const int units = static_cast<int>(gridDim.x) / CTAS;
  const bool draws = p.sched != nullptr && num_tiles > units;
  grid_wait();
  if (warp == 3 && rank == 0 && lane == 0)
    bars->first = draws ? atomicAdd(&p.sched[0], 1) : static_cast<int>(blockIdx.x) / CTAS;
  tc_fence_before();
  if (CTAS == 2) cluster_sync(); else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);

  // Tiles that run at the same time share operands: the dimension with fewer tiles is walked fastest, so that a wave
  // covers all of it and the operand of the other dimension streams through L2 once; in bands, where the operand of the
  // faster dimension would not stay in L2 from one wave to the next.
  // The parts of a split contraction follow one another.
  auto coords = [&](int tile, int& tm, int& tn, int& part) {
    part = p.splits > 1 ? tile / out_tiles : 0;
    tile -= part * out_tiles;
    const int fast = n_fast ? tiles_n : tiles_m, slow = n_fast ? tiles_m : tiles_n;
    const int b = tile / (p.band * slow), f0 = b * p.band;
    const int bw = min(p.band, fast - f0), r = tile - f0 * slow;
    const int f = f0 + r % bw, sl = r / bw;
    tm = n_fast ? sl : f;
    tn = n_fast ? f : sl;
  };
  // The n-th tile of this CTA (or pair), -1 behind the last one.
  auto tile_at = [&](uint32_t n, int& tile) -> bool {
    if (!__all_sync(0xffffffffu, mbar_wait(&bars->tile_full[n % RING], (n / RING) & 1, p.status))) return false;
    tile = *reinterpret_cast<volatile int*>(&bars->tile[n % RING]);
    return true;
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer (both CTAs of a pair load their own halves)
    uint32_t n = 0;
    int s = 0;
    uint32_t ph = 0, fills = 0;
    bool ok = true;
    for (;; ++n) {
      if (rank == 0 && elect_one()) {
        int next = n > 0 && draws ? atomicAdd(&p.sched[0], 1) : bars->first + static_cast<int>(n) * units;
        if (next >= num_tiles) next = -1;
        bars->tile[n % RING][0] = next;
        if (CTAS == 2)
          st_async_v4(mapa_u32(smem_u32(&bars->tile[n % RING]), 1), mapa_u32(smem_u32(&bars->tile_full[n % RING]), 1),
                      next, 0, 0, 0);
        mbar_arrive(&bars->tile_full[n % RING]);
      } else if (rank == 1 && elect_one()) {
        mbar_arrive_expect_tx(&bars->tile_full[n % RING], 16);
      }
      __syncwarp();
      int tile;
      if (!(ok = tile_at(n, tile)) || tile < 0) break;
      int tm, tn, part;
      coords(tile, tm, tn, part);
      const int kb1 = min(k_blocks, (part + 1) * p.k_per);
      const int m0 = tm * (BM * CTAS) + static_cast<int>(rank) * BM;
      const int n0 = tn * width + static_cast<int>(rank) * b_rows;
      for (int kb = part * p.k_per; kb < kb1; ++kb) {
        if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->empty[s], ph ^ 1, p.status)))) break;
        if (elect_one()) {
          uint8_t* sa = smem + s * stage_bytes;
          uint8_t* sb = sa + A_STAGE_BYTES;
          if (rank == 0) mbar_arrive_expect_tx(&bars->full[s], CTAS * stage_bytes);
          const int k0 = kb * BK;
          if (A_MN) {
            tma_load_2d_n<CTAS>(sa, &tmap_a, &bars->full[s], m0, k0);
            tma_load_2d_n<CTAS>(sa + MN_BOX_BYTES, &tmap_a, &bars->full[s], m0 + 64, k0);
          } else {
            tma_load_2d_n<CTAS>(sa, &tmap_a, &bars->full[s], k0, m0);
          }
          if (B_MN) {
            for (int j = 0; j < b_boxes; ++j)
              tma_load_2d_n<CTAS>(sb + j * MN_BOX_BYTES, &tmap_b, &bars->full[s], n0 + 64 * j, k0);
          } else {
            tma_load_2d_n<CTAS>(sb, &tmap_b, &bars->full[s], k0, n0);
          }
        }
        __syncwarp();
        ++fills;
        if (++s == stages) { s = 0; ph ^= 1; }
      }
      if (!ok) break;
    }
    grid_launch();                               // the last loads are on their way
    if (ok) {
      // every stage handed back before the CTA may leave: no commit is still on its way to these barriers
      for (int i = 0; i < stages && ok; ++i) {
        ok = mbar_wait(&bars->empty[s], ph ^ 1, p.status);
        if (++s == stages) { s = 0; ph ^= 1; }
      }
    } else if (rank == 0) {
      for (int i = 0; i < stages; ++i) {         // let the copies already issued land
        if (fills <= static_cast<uint32_t>(i)) continue;
        mbar_wait(&bars->full[i], ((fills - 1 - i) / stages) & 1, nullptr);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer (first CTA of a pair, for both)
    if (rank == 0) {
      const uint32_t idesc = umma_idesc_bf16(BM * CTAS, width, A_MN, B_MN);
      const uint64_t da0 = umma_desc_sw128(smem_u32(smem), A_MN ? MN_BOX_BYTES : 16, 1024);
      const uint64_t db0 = umma_desc_sw128(smem_u32(smem) + A_STAGE_BYTES, B_MN ? MN_BOX_BYTES : 16, 1024);
      constexpr int a_step = (A_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      constexpr int b_step = (B_MN ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (uint32_t n = 0; ok; ++n) {
        int tile;
        if (!(ok = tile_at(n, tile)) || tile < 0) break;
        const uint32_t acc = n & 1;
        if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->acc_empty[acc], ((n >> 1) & 1) ^ 1, p.status)))) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * 256;
        const int part = p.splits > 1 ? tile / out_tiles : 0;
        const int kb0 = part * p.k_per, kb1 = min(k_blocks, kb0 + p.k_per);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->full[s], ph, p.status)))) break;
          tc_fence_after();
          if (elect_one()) {
            const uint64_t da = da0 + (static_cast<uint32_t>(s * stage_bytes) >> 4);
            const uint64_t db = db0 + (static_cast<uint32_t>(s * stage_bytes) >> 4);
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_bf16_ss_n<CTAS>(tmem_d, da + k * a_step, db + k * b_step, idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            umma_commit_n<CTAS>(&bars->empty[s]);
            if (kb == kb1 - 1) umma_commit_n<CTAS>(&bars->acc_full[acc]);
          }
          __syncwarp();
          if (++s == stages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------- epilogue
    const int q = warp & 3;                     // TMEM lanes [32q, 32q + 32)
    const int half = (warp - 4) >> 2;           // odd or even 32-column chunks
    uint8_t* const stage0 = smem + BAR_OFF - (warp - 3) * C_STAGE_BYTES * p.c_bufs;
    uint8_t* stage = stage0;
    for (uint32_t n = 0;; ++n) {
      int tile;
      if (!tile_at(n, tile) || tile < 0) break;
      const uint32_t acc = n & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&bars->acc_full[acc], (n >> 1) & 1, p.status))) break;
      int tm, tn, part;
      coords(tile, tm, tn, part);
      const int row0 = tm * (BM * CTAS) + static_cast<int>(rank) * BM + q * 32;
      const int n0 = tn * width;
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * 256;
      // chunks of 32 columns: two in flight for bf16 (2 KiB staged each), one for fp32 (4 KiB)
      constexpr int CHUNKS = EPI == kEpiStoreBf16 ? 2 : 1;
      constexpr int BLOCK = C_STAGE_BYTES / CHUNKS;
#pragma unroll 1
      for (int c = half; c < width / 32; c += 2 * CHUNKS) {
        if (row0 >= p.M || n0 + c * 32 >= p.N) break;
        uint32_t r[CHUNKS][32];
#pragma unroll
        for (int j = 0; j < CHUNKS; ++j)
          if (j == 0 || c + 2 * j < width / 32) tmem_ld_32x32(taddr + (c + 2 * j) * 32, r[j]);
        tmem_ld_wait();
        if (lane == 0) {                               // the previous blocks have left the buffer
          if (p.c_bufs == 2) bulk_wait_group_read<1>();
          else bulk_wait_group_read<0>();
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < CHUNKS; ++j) {
          uint8_t* blk = stage + j * BLOCK;
          if (EPI == kEpiStoreBf16) {
            // 64-byte rows, 16-byte chunks XOR-swizzled by the row pair
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const uint32_t* x = &r[j][8 * v];
              uint4 o;
              o.x = pack_bf16x2(__uint_as_float(x[0]), __uint_as_float(x[1]));
              o.y = pack_bf16x2(__uint_as_float(x[2]), __uint_as_float(x[3]));
              o.z = pack_bf16x2(__uint_as_float(x[4]), __uint_as_float(x[5]));
              o.w = pack_bf16x2(__uint_as_float(x[6]), __uint_as_float(x[7]));
              reinterpret_cast<uint4*>(blk + lane * 64)[v ^ ((lane >> 1) & 3)] = o;
            }
          } else {
            // 128-byte rows, 16-byte chunks XOR-swizzled by row
#pragma unroll
            for (int v = 0; v < 8; ++v)
              reinterpret_cast<uint4*>(blk + lane * 128)[v ^ (lane & 7)] =
                  make_uint4(r[j][4 * v], r[j][4 * v + 1], r[j][4 * v + 2], r[j][4 * v + 3]);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // the tensor map clips ragged edges; a reduce-add never reads C into the SM
#pragma unroll
          for (int j = 0; j < CHUNKS; ++j) {
            const int col0 = n0 + (c + 2 * j) * 32;
            if (j > 0 && (c + 2 * j >= width / 32 || col0 >= p.N)) continue;
            if (EPI == kEpiAccumF32 && p.accumulate) tma_reduce_add_2d_bulk(&tmap_c, stage + j * BLOCK, col0, row0);
            else tma_store_2d_bulk(&tmap_c, stage + j * BLOCK, col0, row0 + part * p.split_rows);
          }
          bulk_commit_group();
        }
        if (p.c_bufs == 2) stage = stage == stage0 ? stage0 + C_STAGE_BYTES : stage0;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CTAS == 2) mbar_arrive_cluster(mapa_u32(smem_u32(&bars->acc_empty[acc]), 0));
        else mbar_arrive(&bars->acc_empty[acc]);
      }
    }
    if (lane == 0) bulk_wait_group<0>();         // staged blocks must leave before the CTA does
  }

  tc_fence_before();
  if (CTAS == 2) cluster_sync(); else __syncthreads();
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

// C[m, n] = sum of the parts of a split contraction, in their order, rounded to bf16 once.  parts [splits][rows][ld]; a thread
// has eight neighbouring columns, which the scratch holds for every row (ld is a multiple of eight).
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ parts, __nv_bfloat16* __restrict__ c, int M, int N, int rows, int ld, long long ldc,
                 int splits) {
  grid_begin(parts);
  const int vecs = ld / 8;
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= static_cast<long long>(M) * vecs) return;
  const int m = static_cast<int>(i / vecs), n = static_cast<int>(i - static_cast<long long>(m) * vecs) * 8;
  const float4* src = reinterpret_cast<const float4*>(parts + static_cast<long long>(m) * ld + n);
  const long long step = static_cast<long long>(rows) * ld / 4;
  float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float4 a = __ldcs(src + s * step), b = __ldcs(src + s * step + 1);
    lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
    hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
  }
  const uint4 o = make_uint4(pack_bf16x2(lo.x, lo.y), pack_bf16x2(lo.z, lo.w), pack_bf16x2(hi.x, hi.y), pack_bf16x2(hi.z, hi.w));
  __nv_bfloat16* dst = c + m * ldc + n;
  if (n + 8 <= N) {
    *reinterpret_cast<uint4*>(dst) = o;
  } else {
    const uint32_t w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (n + j < N) dst[j] = reinterpret_cast<const __nv_bfloat16*>(w)[j];
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point, so the
// library does not link against libcuda directly.
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

EncodeFn get_encode_fn() {
  static EncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeFn>(p);
  }
  return fn;
}

}  // namespace

// Pool of tile-scheduler slots (next tile, finished CTAs), one slot per dense or grouped launch in rotation; the launch 4,096
// before, whose last CTA rearms the slot, has to have ended on its stream by then.  It is the only device memory this library
// allocates by itself: 32 KiB, once per process.
constexpr int kSchedSlots = 4096;

int* gemm_sched_slot() {
  static int* const pool = []() -> int* {
    const char* env = getenv("PIPER_GEMM_STATIC_TILES");
    if (env != nullptr && env[0] == '1') return nullptr;
    int* p = nullptr;
    if (cudaMalloc(&p, kSchedSlots * 2 * sizeof(int)) != cudaSuccess ||
        cudaMemset(p, 0, kSchedSlots * 2 * sizeof(int)) != cudaSuccess)
      return nullptr;
    return p;
  }();
  static std::atomic<unsigned long long> counter{0};
  return pool == nullptr ? nullptr : pool + 2 * (counter++ % kSchedSlots);
}

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                      uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer) {
  EncodeFn fn = get_encode_fn();
  if (fn == nullptr) return -1;
  // The driver entry point needs a current context on the calling thread;
  // autograd's backward threads have only used the runtime API lazily.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) {
    cudaFree(nullptr);
    ctx_bound = true;
  }
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {row_stride_bytes};
  const cuuint32_t box[2] = {box_inner, box_outer};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r =
      fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

// fp32 tensor map of C with 32x32 boxes and 128-byte swizzle (epilogue staging layout).
int make_tmap_c_f32(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t row_stride_bytes) {
  EncodeFn fn = get_encode_fn();
  if (fn == nullptr) return -1;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {row_stride_bytes};
  const cuuint32_t box[2] = {32, 32};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

// bf16 tensor map of C with 32x32 boxes and 64-byte swizzle.
static int make_tmap_c_bf16(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t row_stride_bytes) {
  EncodeFn fn = get_encode_fn();
  if (fn == nullptr) return -1;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {row_stride_bytes};
  const cuuint32_t box[2] = {32, 32};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

template <int CTAS, bool A_MN, bool B_MN, int EPI>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const Params& p, int num_sms,
                  cudaStream_t stream) {
  auto kern = gemm_kernel<CTAS, A_MN, B_MN, EPI>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return -2;
    configured = true;
  }
  const int tiles = ((p.M + BM * CTAS - 1) / (BM * CTAS)) * ((p.N + p.width - 1) / p.width) * p.splits;
  const int units = num_sms / CTAS;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(CTAS * (tiles < units ? tiles : units)));
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
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

template <int CTAS>
static int launch_layout(const GemmArgs& g, const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc,
                         const Params& p, int num_sms, cudaStream_t stream) {
  const int key = (g.a_mn_major ? 4 : 0) | (g.b_mn_major ? 2 : 0) | (g.epilogue == kEpiAccumF32 ? 1 : 0);
  switch (key) {
    case 0: return launch<CTAS, false, false, kEpiStoreBf16>(ta, tb, tc, p, num_sms, stream);
    case 1: return launch<CTAS, false, false, kEpiAccumF32>(ta, tb, tc, p, num_sms, stream);
    case 2: return launch<CTAS, false, true, kEpiStoreBf16>(ta, tb, tc, p, num_sms, stream);
    case 3: return launch<CTAS, false, true, kEpiAccumF32>(ta, tb, tc, p, num_sms, stream);
    case 4: return launch<CTAS, true, false, kEpiStoreBf16>(ta, tb, tc, p, num_sms, stream);
    case 5: return launch<CTAS, true, false, kEpiAccumF32>(ta, tb, tc, p, num_sms, stream);
    case 6: return launch<CTAS, true, true, kEpiStoreBf16>(ta, tb, tc, p, num_sms, stream);
    default: return launch<CTAS, true, true, kEpiAccumF32>(ta, tb, tc, p, num_sms, stream);
  }
}

// 0: choose by shape, 128 / 256: forced by PIPER_GEMM_TILE
int gemm_forced_tile() {
  static int v = -1;
  if (v < 0) {
    const char* env = getenv("PIPER_GEMM_TILE");
    v = env == nullptr ? 0 : atoi(env);
    if (v != 128 && v != 256) v = 0;
  }
  return v;
}

// One CTA (128 rows) or a pair (256) per tile where gemm_cost does not tell them apart.  Pairs load a third fewer operand
// bytes per flop and draw less power (4096 x 28672 x 4096 in a long loop 733 us with one CTA per tile, 690 us in pairs), but
// a pair starts later and hands every tile over between its SMs (512 x 768 x 256 5.2 us and 6.0 us, 1024 x 4096 x 4096
// 25.8 and 26.4 us).  So near ties go to pairs where there are rounds enough: by the number of rounds if all SMs had a 256 x
// 256 tile each, and in a single such round for long contractions over well-filled SMs; wide fp32 outputs (weight gradients
// that add into a bucket) of fewer than two rounds go to single CTAs.  Of 1,410 random products (M 100-8192, N 256-16384, K
// 64-14400, both directions) 255 are near ties, and on 70 of those where this rule and the lower cost differ it is the faster one 55
// times and 1.0 % behind the better choice on average, the lower cost 4.9 % (7641 x 3376 x 200 26.9 us by one CTA, 23.4 in pairs;
// 536 x 6272 x 3968 into fp32 38.4 and 41.8 us).
int gemm_tile_rows(int M, int N, int K, bool f32_out, int num_sms) {
  const long long n_tiles = (N + 255) / 256;
  const long long tiles256 = (M + 255) / 256 * n_tiles;
  const long long rounds256 = (tiles256 + num_sms - 1) / num_sms;
  const long long rounds128 = ((M + 127) / 128 * n_tiles + num_sms - 1) / num_sms;
  const bool fits = M >= 256 && N >= 256 && rounds256 * 1000 < rounds128 * 599;
  const bool fills = tiles256 >= num_sms || tiles256 * K >= 3072ll * num_sms;
  const bool pays = !f32_out || M >= N || tiles256 >= 2 * num_sms;
  return fits && fills && pays ? 256 : 128;
}

// Cycles of a launch, up to what all shapes have in common: rounds of tiles over the SMs (or pairs), each as long as the
// MMAs of its k-blocks, the fill of their operands from L2 (65 bytes per cycle and SM) or the epilogue of the tile
// before it, and the last epilogue and the start, which is longer for a pair.  The constants are fitted to 89 launches
// in all widths by one CTA and by two (outputs from 100 x 688 to 28672 x 4096, K from 64 to 32000, all layouts, bf16 and
// fp32): the shape it picks is 1.1 % behind the fastest of the sixteen on average, 14 % at most (few tiles over a long
// contraction), where 256 columns throughout are 17 % behind in pairs and 25 % by single CTAs.  Narrower tiles even out the last round: 4096 x 5120 x
// 2048 in 23 x 16 tiles of 224 columns 56.3 us, in 20 x 16 of 256 columns 58.8 us; 1000 x 3072 x 8192 in 64 tiles of 192 columns
// 37.6 us, in 48 of 256 columns 44.6 us; and a small problem covers more SMs: 512 x 768 x 256 5.2 and 7.2 us.
static double gemm_cost(int M, int N, int K, bool b_mn, bool f32_out, int ctas, int width, int num_sms, int splits = 1) {
  const double k_blocks = ((K + BK - 1) / BK + splits - 1) / splits;
  const long long tiles =
      static_cast<long long>((M + BM * ctas - 1) / (BM * ctas)) * ((N + width - 1) / width) * splits;
  const long long units = num_sms / ctas;
  const double rounds = static_cast<double>((tiles + units - 1) / units);
  const int b_rows = b_mn ? (width / ctas + 63) / 64 * 64 : width / ctas;
  const double block = std::max(2.0 * width, (BM + b_rows) * 128 / 65.0);
  const double epilogue = 2000 + (f32_out ? 15 : 10) * width;
  return rounds * std::max(k_blocks * block, epilogue) + epilogue + (ctas == 2 ? 2500 : 2000);
}

GemmShape gemm_shape(int M, int N, int K, bool b_mn, bool f32_out, int num_sms) {
  GemmShape best[2] = {{1, 256, 1}, {2, 256, 1}};
  double cost[2];
  for (int i = 0; i < 2; ++i) {
    for (int width = 256; width >= 32; width -= 32) {
      const double c = num_sms <= i ? 1e300 : gemm_cost(M, N, K, b_mn, f32_out, i + 1, width, num_sms);
      if (width == 256 || c < cost[i]) {
        cost[i] = c;
        best[i].width = width;
      }
    }
  }
  // within 3 % of one another the model does not tell them apart
  const bool close = std::max(cost[0], cost[1]) < 1.03 * std::min(cost[0], cost[1]);
  const bool pair = close ? gemm_tile_rows(M, N, K, f32_out, num_sms) == 256 : cost[1] < cost[0];
  return best[pair ? 1 : 0];
}

constexpr long long kMaxSplitFloats = 16ll << 20;       // 64 MiB of scratch

long long gemm_split_floats(int M, int N, int splits) {
  return splits > 1 ? static_cast<long long>(splits) * ((M + 31) / 32 * 32) * ((N + 7) / 8 * 8) : 0;
}

// Parts of the contraction (and the shape of their tiles) where few output tiles leave most SMs without one: an input
// gradient of few tokens, whose contraction is the layer's output width.  Every part is a tile that leaves fp32 sums in
// scratch, and split_sum_kernel adds them in order.  Against one part by gemm_cost, a split launch takes its tiles as that has
// them, or the time that the operands take out of memory (3,400 bytes per cycle), and 10,000 cycles and 3 per 1,000 sums
// more for the sums' way through scratch; it has to save 8 %.  Fitted to 51 shapes (M 100-1500, N 256-4096, K 2048-128256) in 1 to 32
// parts: the choice is 1 % behind the fastest on average, 15 % at most, and never behind one part.  us in one part and split:
// 128 x 2048 x 128256 410 and 93 (floor 85), 500 x 2048 x 128256 563 and 211, 100 x 4096 x 28672 138 and 57, 512 x 2048 x 16384 75 and
// 45, 128 x 1024 x 8192 30 and 15, 1500 x 256 x 32000 133 and 41; not split 1000 x 4096 x 28672 164 and 179, 512 x 4096 x 6144 25 and 31.
// Products with both operands K-major, the forward pass, are never split, although 100 x 4096 x 14336 would take 37 us instead of
// 64: a token's row has the same bits in a batch of any size.  (That is kept for products; the attention between them adds a
// row's sums in an order that depends on the batch, see attn_tiles_per_cta.)
GemmShape gemm_split_shape(int M, int N, int K, bool b_mn, bool f32_out, int num_sms) {
  const GemmShape whole = gemm_shape(M, N, K, b_mn, f32_out, num_sms);
  const int k_blocks = (K + BK - 1) / BK;
  if (!b_mn || f32_out || k_blocks < 8) return whole;
  const double memory = 2.0 * K * (static_cast<double>(M) + N) / 3400;
  const double unsplit = std::max(gemm_cost(M, N, K, b_mn, f32_out, whole.ctas, whole.width, num_sms), memory);
  // no split is faster than the arithmetic of all SMs, or than memory
  const double least = std::max(static_cast<double>(M) * N * K / (4096.0 * num_sms), memory);
  if (least + 14000 > 0.92 * unsplit) return whole;
  GemmShape best = whole;
  double cost = 0.92 * unsplit;
  for (const int splits : {2, 3, 4, 6, 8, 12, 16, 24, 32}) {
    if (splits > k_blocks / 4 || gemm_split_floats(M, N, splits) > kMaxSplitFloats) break;
    const double sums = 10000 + 0.003 * splits * M * N;
    for (int ctas = 1; ctas <= 2 && ctas <= num_sms; ++ctas)
      for (int width = 256; width >= 32; width -= 32) {
        const double c = std::max(gemm_cost(M, N, K, b_mn, true, ctas, width, num_sms, splits), memory) + sums;
        if (c < cost) {
          cost = c;
          best = {ctas, width, splits};
        }
      }
  }
  // as many parts as have k-blocks
  const int per = (k_blocks + best.splits - 1) / best.splits;
  best.splits = (k_blocks + per - 1) / per;
  return best;
}

static int gemm_launch_shape(const GemmArgs& g, GemmShape shape, int num_sms, cudaStream_t stream) {
  if (shape.ctas < 1 || shape.ctas > 2 || shape.width < 32 || shape.width > 256 || shape.width % 32 != 0) return -1;
  if (num_sms < 2) shape.ctas = 1;
  const int k_blocks = (g.K + BK - 1) / BK;
  const uint32_t b_rows = shape.width / shape.ctas;
  CUtensorMap ta, tb, tc;
  int rc;
  // K-major operand: dims {K, rows}, box {64, rows of a CTA}; MN-major operand: dims {rows, K}, box {64, 64}.
  rc = g.a_mn_major ? make_tmap_2d_bf16(&ta, g.a, g.M, g.K, g.lda * 2, 64, BK)
                    : make_tmap_2d_bf16(&ta, g.a, g.K, g.M, g.lda * 2, BK, BM);
  if (rc != 0) return rc;
  rc = g.b_mn_major ? make_tmap_2d_bf16(&tb, g.b, g.N, g.K, g.ldb * 2, 64, BK)
                    : make_tmap_2d_bf16(&tb, g.b, g.K, g.N, g.ldb * 2, BK, b_rows);
  if (rc != 0) return rc;
  const int rows = (g.M + 31) / 32 * 32, ld = (g.N + 7) / 8 * 8;      // of a part in scratch: the output boxes have 32 rows
  if (shape.splits > 1)
    rc = make_tmap_c_f32(&tc, g.scratch, g.N, static_cast<uint64_t>(shape.splits) * rows, static_cast<uint64_t>(ld) * 4);
  else
    rc = g.epilogue == kEpiAccumF32 ? make_tmap_c_f32(&tc, g.c, g.N, g.M, static_cast<uint64_t>(g.ldc) * 4)
                                    : make_tmap_c_bf16(&tc, g.c, g.N, g.M, static_cast<uint64_t>(g.ldc) * 2);
  if (rc != 0) return rc;
  const int stage = A_STAGE_BYTES + (g.b_mn_major ? (b_rows + 63) / 64 * MN_BOX_BYTES : b_rows * BK * 2);
  Params p;
  // Contractions over a few k-blocks wait for their epilogues, above all for fp32 reduce-adds; two blocks in flight per
  // warp cost a stage or two that they do not fill (3840 x 5760 x 152 into fp32 26.1 and 23.4 us).
  p.c_bufs = g.epilogue == kEpiAccumF32 && g.K <= 8 * BK ? 2 : 1;
  const int fit = (OPERAND_BYTES - (p.c_bufs - 1) * EPI_WARPS * C_STAGE_BYTES) / stage;
  p.M = g.M;
  p.N = g.N;
  p.K = g.K;
  p.width = shape.width;
  p.stages = fit < MAX_STAGES ? fit : MAX_STAGES;
  p.accumulate = shape.splits > 1 ? 0 : g.accumulate;
  p.splits = shape.splits;
  p.k_per = (k_blocks + shape.splits - 1) / shape.splits;
  p.split_rows = rows;
  const int tiles_m = (g.M + BM * shape.ctas - 1) / (BM * shape.ctas), tiles_n = (g.N + shape.width - 1) / shape.width;
  // An operand that stays in L2 (126 MB) is best read whole by every wave (4096 x 28672 x 4096: 701 us, in bands of 8
  // 717 us); one that does not is read from DRAM again by each, and bands of 8 tiles make the wave square (4096 x 4096 x
  // 28672: 799 and 761 us, x 14336: 389 and 381 us).
  const bool n_fast = tiles_n < tiles_m;
  const long long fast_bytes = 2ll * (n_fast ? g.N : g.M) * g.K / shape.splits;
  p.band = fast_bytes > (96ll << 20) ? 8 : (n_fast ? tiles_n : tiles_m);
  p.status = g.status;
  p.sched = gemm_sched_slot();
  GemmArgs l = g;
  if (shape.splits > 1) l.epilogue = kEpiAccumF32;
  rc = shape.ctas == 2 ? launch_layout<2>(l, ta, tb, tc, p, num_sms, stream)
                       : launch_layout<1>(l, ta, tb, tc, p, num_sms, stream);
  if (rc != 0 || shape.splits == 1) return rc;
  const long long threads = static_cast<long long>(g.M) * (ld / 8);
  launch_overlapped(split_sum_kernel, static_cast<unsigned>((threads + 255) / 256), 256, 0, stream,
      g.scratch, static_cast<__nv_bfloat16*>(g.c), g.M, g.N, rows, ld, g.ldc, shape.splits);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int gemm_bf16_launch(const GemmArgs& g, int num_sms, cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return 0;
  GemmShape shape = g.shape;
  if (shape.ctas == 0) {
    const int tile = gemm_forced_tile();
    shape = tile != 0 ? GemmShape{tile / 128, 256, 1}
                      : gemm_shape(g.M, g.N, g.K, g.b_mn_major != 0, g.epilogue != kEpiStoreBf16, num_sms);
  }
  if (shape.splits > 1) {
    const int k_blocks = (g.K + BK - 1) / BK, per = (k_blocks + shape.splits - 1) / shape.splits;
    if (g.scratch == nullptr || g.epilogue != kEpiStoreBf16 || (k_blocks + per - 1) / per != shape.splits) return -1;
  }
  return gemm_launch_shape(g, shape, num_sms, stream);
}

}  // namespace piper
