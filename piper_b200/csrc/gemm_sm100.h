// Host-side interface of the tcgen05 GEMM family (gemm_sm100.cu,
// grouped_gemm_sm100.cu).  Plain C++ / CUDA runtime types only, so the
// kernels build without any framework headers.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace piper {

enum : int {
  kEpiStoreBf16 = 0,   // C (bf16) = acc
  kEpiAccumF32 = 1,    // C (fp32) = acc, or C += acc when accumulate != 0
};

// The shape of a launch: CTAs per tile (1 or 2, 128 rows each), columns (a multiple of 32 up to 256), and parts of the
// contraction.
struct GemmShape {
  int ctas, width, splits;
};

// C[M,N] = A[M,K] * B[N,K]^T.
//   a_mn_major == 0: A is stored row-major [M, K] with row stride lda (elements).
//   a_mn_major == 1: A is stored row-major [K, M] with row stride lda.
//   b_mn_major == 0: B is stored row-major [N, K] with row stride ldb.
//   b_mn_major == 1: B is stored row-major [K, N] with row stride ldb.
// Base pointers must be 16-byte aligned and lda/ldb multiples of 8 elements
// (TMA global-stride rule); ldc is in elements of the output type.
struct GemmArgs {
  const void* a;
  const void* b;
  void* c;
  long long lda, ldb, ldc;
  int M, N, K;
  int a_mn_major, b_mn_major;
  int epilogue;     // kEpi*
  int accumulate;   // only for kEpiAccumF32
  int* status;      // device int, 0 = ok (see ptx.cuh)
  GemmShape shape = {0, 0, 1};   // ctas 0: by PIPER_GEMM_TILE or gemm_shape
  float* scratch = nullptr;      // gemm_split_floats() floats where shape.splits > 1 (kEpiStoreBf16 only)
};

// Returns 0 on success, a negative code for a launch/set-up failure, or the
// CUresult of a failed tensor-map encode.
int gemm_bf16_launch(const GemmArgs& args, int num_sms, cudaStream_t stream);

// The tile height (128: one CTA, 256: a CTA pair) that gemm_shape takes where the model of its costs is undecided.
int gemm_tile_rows(int M, int N, int K, bool f32_out, int num_sms);

// The shape that gemm_bf16_launch chooses: the contraction in one part.
GemmShape gemm_shape(int M, int N, int K, bool b_mn_major, bool f32_out, int num_sms);

// The shape to launch where there may be scratch, and the scratch of one in `splits` parts (each with k-blocks of 64).
GemmShape gemm_split_shape(int M, int N, int K, bool b_mn_major, bool f32_out, int num_sms);
int gemm_forced_tile();   // of PIPER_GEMM_TILE, 0: none
long long gemm_split_floats(int M, int N, int splits);

enum : int {
  kGroupedFwd = 0,     // Y[rows, N]  = X[rows, K] * W[e]^T
  kGroupedDgrad = 1,   // dX[rows, K] = dY[rows, N] * W[e]
  kGroupedWgrad = 2,   // dW[e][N, K] (+)= dY[rows_e]^T * X[rows_e]   (fp32 output)
};

// Grouped GEMMs of the expert MLP.  Rows of x / dy / out are grouped: group g
// owns rows [g_start[g], g_start[g] + g_len[g]), g_len a multiple of 128 with
// zero padding rows, and uses expert g % experts of w [experts, N, K].
// g_start / g_len live on the device.  rows_capacity is the row count of the
// row buffers.  out is bf16 [rows_capacity, N] (fwd), bf16 [rows_capacity, K]
// (dgrad) or [experts, N, K] (wgrad; fp32, where accumulate selects += or =, or bf16).
struct GroupedGemmArgs {
  int mode;
  const void* x;        // [rows_capacity, K]   (fwd, wgrad)
  const void* dy;       // [rows_capacity, N]   (dgrad, wgrad)
  const void* w;        // [experts, N, K]      (fwd, dgrad)
  void* out;
  const int* g_start;
  const int* g_len;
  int num_groups, experts;
  int N, K;
  long long rows_capacity;
  int accumulate;
  int out_bf16;         // weight gradient as bf16 instead of fp32 (never accumulates)
  int* status;
};

int grouped_gemm_launch(const GroupedGemmArgs& args, int num_sms, cudaStream_t stream);

// Two zeroed ints of device memory for the dynamic tile scheduler of one launch (next tile, finished CTAs; rearmed by the
// kernel), or null for static tile striding.
int* gemm_sched_slot();

constexpr int kMaxPeers = 8;

// Y[M, N] = X[M, K] * W[N, K]^T with W sharded by rows: w_shards[p] points at
// rank p's rows [p*rows_per_shard, (p+1)*rows_per_shard) (local or peer-mapped
// memory, rows_per_shard a multiple of 64); shard my_index is this rank's own.
// When w_full is not null every remote row crosses NVLink once, into w_full
// ([N, K], local memory, complete when the kernel ends), and scratch must
// point at scratch_ints >= ceil(N / 256) + 2 ints of device memory that no
// other launch in flight uses.  When w_full is null each CTA loads the weight
// boxes it needs straight from their owners.
struct AgGemmArgs {
  const void* x;
  const void* w_shards[kMaxPeers];
  void* w_full;
  void* y;
  int M, N, K;
  int rows_per_shard, num_peers, my_index;
  int* scratch;
  int scratch_ints;
  int* status;
};

int ag_gemm_launch(const AgGemmArgs& args, int num_sms, cudaStream_t stream);

// fp32 tensor map of an output matrix with 32x32 boxes and 128-byte swizzle (layout of the fp32 epilogue staging).
int make_tmap_c_f32(CUtensorMap* out, const void* base, uint64_t cols, uint64_t rows, uint64_t row_stride_bytes);

// Encodes a 2-D bf16 tensor map with 128-byte swizzle.
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                      uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer);

}  // namespace piper
