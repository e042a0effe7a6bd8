// Memory-bound kernels of the transformer block for sm_100a: RMSNorm
// (optionally fused with the residual add), QK-norm + RoPE on the packed QKV
// projection, SwiGLU, embedding gather / scatter-add, row-wise cross-entropy
// with in-place gradient, and the flat-buffer Adam update.  All of them move
// 16-byte vectors and keep fp32 math in registers; none allocates.
#include "elementwise.h"

#include "ptx.cuh"

#include <cuda_bf16.h>
#include <stdint.h>

#include <type_traits>

namespace piper {
namespace {

struct alignas(16) bf16x8 {
  __nv_bfloat162 v[4];
};

__device__ __forceinline__ void unpack8(const bf16x8& p, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p.v[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ bf16x8 pack8(const float (&f)[8]) {
  bf16x8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.v[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return p;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) scratch[w] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? scratch[threadIdx.x] : 0.f;
  if (w == 0) {
    t = warp_sum(t);
    if (l == 0) scratch[0] = t;
  }
  __syncthreads();
  return scratch[0];
}

template <int THREADS>
__device__ __forceinline__ float block_max(float v, float* scratch) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) scratch[w] = v;
  __syncthreads();
  float t = (threadIdx.x < THREADS / 32) ? scratch[threadIdx.x] : -INFINITY;
  if (w == 0) {
    t = warp_max(t);
    if (l == 0) scratch[0] = t;
  }
  __syncthreads();
  return scratch[0];
}

// ------------------------------------------------------------------ RMSNorm
// One CTA per row.  Optional residual: h = x + res is written to h_out and
// normalised, so the block's "x = x + f(norm(x))" costs one pass.
constexpr int NORM_THREADS = 256;

__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd, int D, float eps) {
  grid_begin(x, res, w);
  __shared__ float scratch[32];
  const long long row = blockIdx.x;
  const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
  const bf16x8* rr = res ? reinterpret_cast<const bf16x8*>(res + row * D) : nullptr;
  bf16x8* hr = h_out ? reinterpret_cast<bf16x8*>(h_out + row * D) : nullptr;
  const int nvec = D / 8;
  float ss = 0.f;
  for (int i = threadIdx.x; i < nvec; i += NORM_THREADS) {
    float f[8];
    unpack8(xr[i], f);
    if (rr) {
      float g[8];
      unpack8(rr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      // Round the residual stream to bf16 before it is normalised, so that
      // forward and backward see the same values.
      const bf16x8 hp = pack8(f);
      hr[i] = hp;
      unpack8(hp, f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = block_sum<NORM_THREADS>(ss, scratch);
  const float r = rsqrtf(ss / D + eps);
  if (threadIdx.x == 0) rstd[row] = r;
  const bf16x8* src = rr ? reinterpret_cast<const bf16x8*>(h_out + row * D) : xr;
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  bf16x8* yr = reinterpret_cast<bf16x8*>(y + row * D);
  for (int i = threadIdx.x; i < nvec; i += NORM_THREADS) {
    float f[8], g[8];
    unpack8(src[i], f);
    unpack8(wr[i], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f[j] * r * g[j];
    yr[i] = pack8(f);
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)), plus an optional pass-through
// gradient dres added to dx (the residual branch).  Column sums of dy*xhat
// go to dw_partial[blockIdx.x][D]; a second kernel reduces them in a fixed
// order, so the weight gradient is reproducible.
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, int T, int D) {
  grid_begin(dy, x, w, rstd, dres);
  extern __shared__ float dw_acc[];   // D floats
  __shared__ float scratch[32];
  for (int i = threadIdx.x; i < D; i += NORM_THREADS) dw_acc[i] = 0.f;
  __syncthreads();
  const int nvec = D / 8;
  const bf16x8* wr = reinterpret_cast<const bf16x8*>(w);
  for (long long row = blockIdx.x; row < T; row += gridDim.x) {
    const bf16x8* dyr = reinterpret_cast<const bf16x8*>(dy + row * D);
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + row * D);
    const float r = rstd[row];
    float dot = 0.f;
    for (int i = threadIdx.x; i < nvec; i += NORM_THREADS) {
      float a[8], b[8], g[8];
      unpack8(dyr[i], a);
      unpack8(xr[i], b);
      unpack8(wr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += a[j] * g[j] * b[j] * r;
    }
    dot = block_sum<NORM_THREADS>(dot, scratch) / D;
    const bf16x8* drr = dres ? reinterpret_cast<const bf16x8*>(dres + row * D) : nullptr;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + row * D);
    for (int i = threadIdx.x; i < nvec; i += NORM_THREADS) {
      float a[8], b[8], g[8], o[8];
      unpack8(dyr[i], a);
      unpack8(xr[i], b);
      unpack8(wr[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = b[j] * r;
        o[j] = r * (a[j] * g[j] - xhat * dot);
        dw_acc[i * 8 + j] += a[j] * xhat;   // column owned by this thread
      }
      if (drr) {
        float e[8];
        unpack8(drr[i], e);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += e[j];
      }
      dxr[i] = pack8(o);
    }
  }
  __syncthreads();
  float* out = dw_partial + static_cast<long long>(blockIdx.x) * D;
  for (int i = threadIdx.x; i < D; i += NORM_THREADS) out[i] = dw_acc[i];
}

// Register-resident variants: THREADS threads (a multiple of 32, at most 256) own a row of 8 * VPT * THREADS elements, VPT
// 8-element vectors each, so the row is read from memory exactly once and its reduction needs a single barrier (the per-warp
// sums alternate between two scratch rows; a thread can only reach the write of row k+2 after every thread has passed the
// barrier of row k+1, i.e. after all reads of row k).  A row of one warp needs none.
// Sum over the THREADS threads of a row; barrier 1 + group is theirs.
template <int THREADS>
__device__ __forceinline__ float row_sum(float v, float* scratch, int warp, int group) {
  v = warp_sum(v);
  if (THREADS == 32) return v;
  if ((threadIdx.x & 31) == 0) scratch[warp] = v;
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(THREADS) : "memory");
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) t += scratch[i];
  return t;
}

// Forward: bound by memory.  As many CTAs as are resident walk the rows (1,024 threads per SM, 512 of the widest rows, which
// take 115 registers a thread) and fetch the next one before the current one is reduced: with a CTA per row every row paid for
// its first loads, for the norm weights behind the barrier and for a last wave.  Residual and norm, 4096 x 4096: 27.7 and 23.5
// us (134 MB, 5.7 TB/s), 8192 x 8192 115 and 87 us, 8192 x 2048 28.2 and 24.0 us; 1000 x 4096 7.7 us both ways.  With more CTAs than
// fit, four per SM of 8192-wide rows, and two: 592 rows 10.6 and 9.5 us, 1777 22.9 and 22.3, 8192 86.7 and 87.6.  8192 rows
// of 256, 1024, 2560 and 3072 by a CTA each that reads them twice and so: 13.4 19.9 39.7 47.5 and 5.7 12.6 27.1 34.1 us.
template <int VPT, int THREADS>
constexpr int NORM_FWD_CTAS = (VPT == 4 ? 512 : 1024) / THREADS;   // per SM, which holds 32

template <int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS, NORM_FWD_CTAS<VPT, THREADS>)
rmsnorm_fwd_reg_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                       const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                       __nv_bfloat16* __restrict__ h_out, float* __restrict__ rstd, long long T, float eps) {
  grid_begin(x, res, w);
  constexpr int D = VPT * 8 * THREADS;
  __shared__ float scratch[2][THREADS / 32];
  bf16x8 wv[VPT], nx[VPT], nr[VPT];
#pragma unroll
  for (int v = 0; v < VPT; ++v) wv[v] = reinterpret_cast<const bf16x8*>(w)[threadIdx.x + v * THREADS];
  auto fetch = [&](long long rw) {
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      nx[v] = reinterpret_cast<const bf16x8*>(x + rw * D)[threadIdx.x + v * THREADS];
      if (res) nr[v] = reinterpret_cast<const bf16x8*>(res + rw * D)[threadIdx.x + v * THREADS];
    }
  };
  long long row = blockIdx.x;
  if (row < T) fetch(row);
  int parity = 0;
  for (; row < T; row += gridDim.x, parity ^= 1) {
    float f[VPT][8];
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      unpack8(nx[v], f[v]);
      if (res) {
        float g[8];
        unpack8(nr[v], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[v][j] += g[j];
        const bf16x8 hp = pack8(f[v]);   // the residual stream is bf16: normalise what is stored
        reinterpret_cast<bf16x8*>(h_out + row * D)[threadIdx.x + v * THREADS] = hp;
        unpack8(hp, f[v]);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) ss += f[v][j] * f[v][j];
    }
    if (row + gridDim.x < T) fetch(row + gridDim.x);
    ss = row_sum<THREADS>(ss, scratch[parity], threadIdx.x >> 5, 0);
    const float r = rsqrtf(ss / D + eps);
    if (threadIdx.x == 0) rstd[row] = r;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      float g[8];
      unpack8(wv[v], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[v][j] = f[v][j] * r * g[j];
      reinterpret_cast<bf16x8*>(y + row * D)[threadIdx.x + v * THREADS] = pack8(f[v]);
    }
  }
}

// Two CTAs per SM (one of the widest rows): the row vectors stay packed (bf16) in registers and are unpacked where they are
// used, which keeps two vectors of 256 threads under 128 registers with the next row's loads in flight; with fewer registers
// they spill (4096 columns under 102: 50 -> 69 us for 8192 rows).  CTAs are as many as there are strips of weight-gradient sums,
// so narrow rows are worked on several at a time, whose sums a CTA adds in their order at the end.  8192 rows of
// 256, 1024, 2560 and 3072 by a CTA of 256 threads a row, sums in shared memory, and so: 46.8 53.8 107.2 111.8 and 5.3 13.8 39.4
// 42.7 us (4.7 TB/s).
template <int VPT, int THREADS>
constexpr int NORM_BWD_ROWS = VPT == 1 && THREADS < 384 ? 384 / THREADS : 1;

template <int VPT, int THREADS>
__global__ void __launch_bounds__(THREADS * NORM_BWD_ROWS<VPT, THREADS>, VPT <= 2 ? 2 : 1)
rmsnorm_bwd_reg_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                       const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                       float* __restrict__ dw_partial, int T) {
  grid_begin(dy, x, w, rstd, dres);
  constexpr int D = VPT * 8 * THREADS, ROWS = NORM_BWD_ROWS<VPT, THREADS>;
  const int rows = ROWS == 1 ? 1 : blockDim.x / THREADS;
  const int group = ROWS == 1 ? 0 : threadIdx.x / THREADS, tid = threadIdx.x - group * THREADS;
  __shared__ float scratch[2][THREADS * ROWS / 32];
  extern __shared__ float strips[];              // [rows][D] where there are several
  const int first_warp = group * (THREADS / 32);
  bf16x8 gw[VPT];
  float dw[VPT][8];
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    gw[v] = reinterpret_cast<const bf16x8*>(w)[tid + v * THREADS];
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[v][j] = 0.f;
  }
  // The next row's vectors are fetched before the current row is reduced, so the loads overlap the barrier.
  bf16x8 na[VPT], nb[VPT], ne[VPT];
  float nr = 0.f;
  const long long step = static_cast<long long>(gridDim.x) * rows;
  long long row = static_cast<long long>(group) * gridDim.x + blockIdx.x;
  auto fetch = [&](long long rw) {
    const bf16x8* dyr = reinterpret_cast<const bf16x8*>(dy + rw * D);
    const bf16x8* xr = reinterpret_cast<const bf16x8*>(x + rw * D);
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      na[v] = dyr[tid + v * THREADS];
      nb[v] = xr[tid + v * THREADS];
    }
    if (dres) {
      const bf16x8* er = reinterpret_cast<const bf16x8*>(dres + rw * D);
#pragma unroll
      for (int v = 0; v < VPT; ++v) ne[v] = er[tid + v * THREADS];
    }
    nr = rstd[rw];
  };
  if (row < T) fetch(row);
  int parity = 0;
  for (; row < T; row += step, parity ^= 1) {
    bf16x8 ca[VPT], cb[VPT], ce[VPT];
    const float r = nr;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      ca[v] = na[v];
      cb[v] = nb[v];
      if (dres) ce[v] = ne[v];
    }
    if (row + step < T) fetch(row + step);
    float dot = 0.f;
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      float a[8], b[8], g[8];
      unpack8(ca[v], a);
      unpack8(cb[v], b);
      unpack8(gw[v], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) dot += a[j] * g[j] * (b[j] * r);
    }
    dot = row_sum<THREADS>(dot, scratch[parity] + first_warp, tid >> 5, group) / D;
    bf16x8* dxr = reinterpret_cast<bf16x8*>(dx + row * D);
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      float a[8], b[8], g[8], o[8];
      unpack8(ca[v], a);
      unpack8(cb[v], b);
      unpack8(gw[v], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xhat = b[j] * r;
        o[j] = r * (a[j] * g[j] - xhat * dot);
        dw[v][j] += a[j] * xhat;
      }
      if (dres) {
        float e[8];
        unpack8(ce[v], e);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += e[j];
      }
      dxr[tid + v * THREADS] = pack8(o);
    }
  }
  float* out = dw_partial + static_cast<long long>(blockIdx.x) * D;
  if (rows > 1) {
#pragma unroll
    for (int v = 0; v < VPT; ++v) {
      float4* o4 = reinterpret_cast<float4*>(strips + group * D + (tid + v * THREADS) * 8);
      o4[0] = make_float4(dw[v][0], dw[v][1], dw[v][2], dw[v][3]);
      o4[1] = make_float4(dw[v][4], dw[v][5], dw[v][6], dw[v][7]);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += blockDim.x) {
      float s = 0.f;
      for (int g = 0; g < rows; ++g) s += strips[g * D + c];
      out[c] = s;
    }
    return;
  }
#pragma unroll
  for (int v = 0; v < VPT; ++v) {
    float4* o4 = reinterpret_cast<float4*>(out + (tid + v * THREADS) * 8);
    o4[0] = make_float4(dw[v][0], dw[v][1], dw[v][2], dw[v][3]);
    o4[1] = make_float4(dw[v][4], dw[v][5], dw[v][6], dw[v][7]);
  }
}

// dw[c] (+)= sum_b partial[b][c]; fp32 output (the flat gradient bucket) or bf16 where that is given.  The columns from
// `split` on go to a second weight.  A block owns 32 columns; its 32 thread rows each sum a contiguous slice of the partials
// and the slices are added in a fixed order, so the result does not depend on timing.
struct WeightGrad {
  float* f32;
  __nv_bfloat16* bf16;
  int accumulate;
};

constexpr int RED_SLICES = 32;
__global__ void __launch_bounds__(32 * RED_SLICES)
reduce_partials_kernel(const float* __restrict__ partial, int nblocks, int D, WeightGrad first, WeightGrad second, int split) {
  grid_begin(partial);
  __shared__ float part[RED_SLICES][32];
  const int c = blockIdx.x * 32 + threadIdx.x;
  const int per = (nblocks + RED_SLICES - 1) / RED_SLICES;
  const int b0 = threadIdx.y * per;
  const int b1 = min(nblocks, b0 + per);
  float s = 0.f;
  if (c < D) {
#pragma unroll 4
    for (int b = b0; b < b1; ++b) s += partial[static_cast<long long>(b) * D + c];
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || c >= D) return;
  s = 0.f;
#pragma unroll
  for (int i = 0; i < RED_SLICES; ++i) s += part[i][threadIdx.x];
  const WeightGrad o = c < split ? first : second;
  const int i = c < split ? c : c - split;
  if (o.f32) o.f32[i] = o.accumulate ? o.f32[i] + s : s;
  if (o.bf16) o.bf16[i] = __float2bfloat16(o.accumulate ? __bfloat162float(o.bf16[i]) + s : s);
}

// --------------------------------------------------------- QK-norm + RoPE
// qkv is the packed projection [T, (Hq + 2*Hkv) * hd], hd = 128 or 64; v heads are copied.
// rope pairs: interleaved (x[2i], x[2i+1]) or half-split (x[i], x[i+hd/2]).
// cos/sin are fp32 [S, hd/2]; position of token t is t % S.
//
// A group of hd/16 lanes handles one (token, head) vector.  Lane l owns the two 16-byte vectors [8l, 8l + 8) and
// [hd/2 + 8l, hd/2 + 8l + 8), so a group reads and writes contiguous memory with every instruction, and both members of
// each of its eight rope pairs are its own: pairs 8l .. 8l + 7 in the half-split form, 4l .. 4l + 3 and hd/4 + 4l ..
// hd/4 + 4l + 3 in the interleaved one.
//
// A warp takes (token, run of heads) tasks: its groups walk neighbouring heads of one token, whose cos/sin entries are
// loaded once, and fetch the next head before they work on the current one.  The tasks are ordered by kind (query, key,
// value heads), and the grid is what is resident at once: a warp has one kind at a time, hence one set of norm weights
// and one set of weight-gradient sums in registers.
// Bound by memory; 32 neighbouring bytes per lane (interleaved) or 640 to 2,368 CTAs of one pass each, without fetching ahead,
// stayed far from it.  In us, forward and backward, so then and now: 4096 x (32 + 2 x 8) x 128 32.8 -> 19.4 (5.2 TB/s) and 30.1 ->
// 19.6; 4096 x (32 + 2 x 4) x 128 with norms 23.7 -> 19.7 and 62.1 -> 32.7 (3.9 TB/s); 16384 x (32 + 2 x 4) x 128 with norms 84.8 ->
// 64.0 and 185.7 -> 103.5; 8192 x (32 + 2 x 8) x 64 32.8 -> 29.2 and 28.1 -> 29.2; 512 x (4 + 2 x 4) x 64 2.6 -> 2.5 and 2.3 -> 2.5.
template <int HD>
struct RopeGroup {
  static constexpr int LANES = HD / 16;
  static constexpr int GROUPS = 32 / LANES;      // of a warp
  int lane, group, off0, off1;
  unsigned mask;
  __device__ __forceinline__ RopeGroup() {
    const int wl = threadIdx.x & 31;
    lane = wl & (LANES - 1);
    group = wl / LANES;
    mask = ((1u << LANES) - 1u) << (wl & ~(LANES - 1));
    off0 = 8 * lane;
    off1 = HD / 2 + 8 * lane;
  }
  __device__ __forceinline__ void sum2(float& u, float& v) const {
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      u += __shfl_xor_sync(mask, u, o);
      v += __shfl_xor_sync(mask, v, o);
    }
  }
  __device__ __forceinline__ float sum(float v) const {
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
  }
  // The cos or sin entries of the lane's pairs, out of the row of one position.
  template <bool INTER>
  __device__ __forceinline__ void load_angles(const float* row, float sign, float (&f)[8]) const {
    const float4 lo = *reinterpret_cast<const float4*>(row + (INTER ? 4 * lane : 8 * lane));
    const float4 hi = *reinterpret_cast<const float4*>(row + (INTER ? HD / 4 + 4 * lane : 8 * lane + 4));
    f[0] = lo.x * sign; f[1] = lo.y * sign; f[2] = lo.z * sign; f[3] = lo.w * sign;
    f[4] = hi.x * sign; f[5] = hi.y * sign; f[6] = hi.z * sign; f[7] = hi.w * sign;
  }
};

// (a, b) -> (a*c - b*s, a*s + b*c) on the lane's eight pairs.
template <bool INTER>
__device__ __forceinline__ void rope_rotate(float (&v0)[8], float (&v1)[8], const float (&c)[8], const float (&s)[8]) {
  if (INTER) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float a0 = v0[2 * p], b0 = v0[2 * p + 1], a1 = v1[2 * p], b1 = v1[2 * p + 1];
      v0[2 * p] = a0 * c[p] - b0 * s[p];
      v0[2 * p + 1] = a0 * s[p] + b0 * c[p];
      v1[2 * p] = a1 * c[4 + p] - b1 * s[4 + p];
      v1[2 * p + 1] = a1 * s[4 + p] + b1 * c[4 + p];
    }
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float a = v0[j], b = v1[j];
      v0[j] = a * c[j] - b * s[j];
      v1[j] = a * s[j] + b * c[j];
    }
  }
}

struct RopeArgs {
  const __nv_bfloat16* x;        // forward: qkv; backward: the gradient of the output
  const __nv_bfloat16* pre;      // backward with norms: qkv before them
  __nv_bfloat16* out;
  const float *cosp, *sinp;
  const __nv_bfloat16 *qw, *kw;  // norm weights of the query and key heads, or null
  float* partial;                // sums of their gradients, [CTA][query, key][hd], or null
  long long T;
  int S, Hq, Hkv;
  float eps;
  int run;                       // heads of a task
};

enum RopeMode { kRopeCopy, kRopePlain, kRopeNorm };

// The tasks of one kind: heads [first_head, first_head + n) of every token.  `task` is the warp's first one and becomes its
// first one of the kind behind.  dw: sums of the weight gradient over the tasks, elements off0 .. and off1 ..
template <int HD, RopeMode MODE, bool BWD, bool INTER>
__device__ __forceinline__ void rope_tasks(const RopeArgs& a, const RopeGroup<HD>& g, int first_head, int n,
                                           const __nv_bfloat16* w, unsigned& task, unsigned warps, float (&dw)[16]) {
  constexpr bool PRE = BWD && MODE == kRopeNorm;
  const int runs = (n + a.run - 1) / a.run;
  const unsigned tasks = static_cast<unsigned>(a.T) * runs;     // the launcher keeps this below 2^31
  const int heads = a.Hq + 2 * a.Hkv;
  bf16x8 pw0, pw1;
  if (MODE == kRopeNorm) {
    pw0 = *reinterpret_cast<const bf16x8*>(w + g.off0);
    pw1 = *reinterpret_cast<const bf16x8*>(w + g.off1);
  }
  for (; task < tasks; task += warps) {
    const unsigned t = task / static_cast<unsigned>(runs);
    const int r = static_cast<int>(task - t * runs);
    int h = r * a.run + g.group;
    const int h1 = min(n, (r + 1) * a.run);
    if (h >= h1) continue;
    long long at = (static_cast<long long>(t) * heads + first_head + h) * HD;
    bf16x8 n0 = *reinterpret_cast<const bf16x8*>(a.x + at + g.off0), n1 = *reinterpret_cast<const bf16x8*>(a.x + at + g.off1);
    bf16x8 m0, m1;
    if (PRE) {
      m0 = *reinterpret_cast<const bf16x8*>(a.pre + at + g.off0);
      m1 = *reinterpret_cast<const bf16x8*>(a.pre + at + g.off1);
    }
    float c[8], s[8];
    if (MODE != kRopeCopy) {
      const int pos = static_cast<int>(t % static_cast<unsigned>(a.S)) * (HD / 2);
      g.template load_angles<INTER>(a.cosp + pos, 1.f, c);
      g.template load_angles<INTER>(a.sinp + pos, BWD ? -1.f : 1.f, s);
    }
#pragma unroll 1
    for (; h < h1; h += g.GROUPS) {
      const bf16x8 p0 = n0, p1 = n1, q0 = m0, q1 = m1;
      __nv_bfloat16* dst = a.out + at;
      at += g.GROUPS * HD;
      if (h + g.GROUPS < h1) {
        n0 = *reinterpret_cast<const bf16x8*>(a.x + at + g.off0);
        n1 = *reinterpret_cast<const bf16x8*>(a.x + at + g.off1);
        if (PRE) {
          m0 = *reinterpret_cast<const bf16x8*>(a.pre + at + g.off0);
          m1 = *reinterpret_cast<const bf16x8*>(a.pre + at + g.off1);
        }
      }
      if (MODE == kRopeCopy) {
        *reinterpret_cast<bf16x8*>(dst + g.off0) = p0;
        *reinterpret_cast<bf16x8*>(dst + g.off1) = p1;
        continue;
      }
      float v0[8], v1[8], w0[8], w1[8];
      unpack8(p0, v0);
      unpack8(p1, v1);
      if (MODE == kRopeNorm) {
        unpack8(pw0, w0);
        unpack8(pw1, w1);
      }
      if (BWD) {
        rope_rotate<INTER>(v0, v1, c, s);
        if (MODE == kRopeNorm) {
          float x0[8], x1[8];
          unpack8(q0, x0);
          unpack8(q1, x1);
          float ss = 0.f, dot = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            ss += x0[j] * x0[j] + x1[j] * x1[j];
            dot += v0[j] * w0[j] * x0[j] + v1[j] * w1[j] * x1[j];
          }
          g.sum2(ss, dot);
          const float rs = rsqrtf(ss / HD + a.eps);
          dot = dot * rs / HD;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xh0 = x0[j] * rs, xh1 = x1[j] * rs;
            dw[j] += v0[j] * xh0;
            dw[8 + j] += v1[j] * xh1;
            v0[j] = rs * (v0[j] * w0[j] - xh0 * dot);
            v1[j] = rs * (v1[j] * w1[j] - xh1 * dot);
          }
        }
      } else {
        if (MODE == kRopeNorm) {
          float ss = 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) ss += v0[j] * v0[j] + v1[j] * v1[j];
          const float rs = rsqrtf(g.sum(ss) / HD + a.eps);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            v0[j] = v0[j] * rs * w0[j];
            v1[j] = v1[j] * rs * w1[j];
          }
        }
        rope_rotate<INTER>(v0, v1, c, s);
      }
      *reinterpret_cast<bf16x8*>(dst + g.off0) = pack8(v0);
      *reinterpret_cast<bf16x8*>(dst + g.off1) = pack8(v1);
    }
  }
  task -= tasks;
}

// NORM: there are norm weights, of the query heads, the key heads or both.  Backward: un-rotate the gradient (RoPE is an
// orthogonal map, so its transpose is the rotation by -theta), then the RMSNorm backward per head; the weight-gradient
// sums of a warp are added over its lane groups, those of a CTA over its warps, and reduce_partials_kernel adds the CTAs', all in
// a fixed order.  (Sixteen shared-memory atomics per lane and head took 147 us for 4096 tokens of 32 + 2 x 4 heads x 128.  One
// atomic per element and CTA into cleared fp32 sums, which are then rounded, takes four launches more for two weights.)
// The backward pass with norms has 128 registers, two CTAs of which fill an SM, and is the one form that spills (40 bytes of stores,
// 96 of loads): 16 sums, two vectors each of gradient and input, the next ones and the weights.  It is at 3.9 TB/s, the others at 5.2.
template <bool NORM, bool BWD>
constexpr int ROPE_CTAS = !NORM ? 4 : BWD ? 2 : 3;     // per SM

// The heads of one kind with the norm they have, and the warp's sums of its weight gradient into sdw.
template <int HD, bool NORM, bool BWD, bool INTER>
__device__ __forceinline__ void rope_kind(const RopeArgs& a, const RopeGroup<HD>& g, int first_head, int n,
                                          const __nv_bfloat16* w, bool want_dw, float* sdw, unsigned& task, unsigned warps) {
  float dw[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) dw[j] = 0.f;
  if (!NORM || w == nullptr) {
    rope_tasks<HD, kRopePlain, BWD, INTER>(a, g, first_head, n, nullptr, task, warps, dw);
    return;
  }
  rope_tasks<HD, kRopeNorm, BWD, INTER>(a, g, first_head, n, w, task, warps, dw);
  if (!want_dw) return;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 16; ++j) {
#pragma unroll
    for (int o = g.LANES; o < 32; o <<= 1) dw[j] += __shfl_xor_sync(0xffffffffu, dw[j], o);
    if (g.group == 0) sdw[(j < 8 ? g.off0 : g.off1) + (j & 7)] = dw[j];
  }
}

template <int HD, bool NORM, bool BWD, bool INTER>
__global__ void __launch_bounds__(256, ROPE_CTAS<NORM, BWD>)
qk_rope_kernel(const __grid_constant__ RopeArgs a) {
  grid_begin();
  __shared__ float sdw[NORM && BWD ? 8 : 1][2 * HD];
  const bool want_dw = NORM && BWD && a.partial != nullptr;
  const RopeGroup<HD> g;
  const int w = NORM && BWD ? threadIdx.x >> 5 : 0;
  unsigned task = blockIdx.x * 8 + (threadIdx.x >> 5);
  const unsigned warps = gridDim.x * 8;
  rope_kind<HD, NORM, BWD, INTER>(a, g, 0, a.Hq, a.qw, want_dw, sdw[w], task, warps);
  rope_kind<HD, NORM, BWD, INTER>(a, g, a.Hq, a.Hkv, a.kw, want_dw, sdw[w] + HD, task, warps);
  float none[16];
  rope_tasks<HD, kRopeCopy, BWD, INTER>(a, g, a.Hq + a.Hkv, a.Hkv, nullptr, task, warps, none);
  if (want_dw) {
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * HD; i += blockDim.x) {
      if ((i < HD ? a.qw : a.kw) == nullptr) continue;
      float v = 0.f;
#pragma unroll
      for (int k = 0; k < (NORM && BWD ? 8 : 1); ++k) v += sdw[k][i];
      a.partial[static_cast<long long>(blockIdx.x) * 2 * HD + i] = v;
    }
  }
}

// ------------------------------------------------------------------- SwiGLU
// h13 = [gate | up] of width 2F per row; act = silu(gate) * up.
// Threads walk the flattened [T][F/8] vector index with a grid stride; row and column advance incrementally
// (stride_rows, stride_cols = stride / (F/8), stride % (F/8) come from the host), so the loop has no division.
struct VecWalk {
  long long row;
  int c;
  __device__ __forceinline__ VecWalk(int vecs) {
    const long long i0 = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    row = i0 / vecs;
    c = static_cast<int>(i0 - row * vecs);
  }
  __device__ __forceinline__ void next(int vecs, int stride_rows, int stride_cols) {
    row += stride_rows;
    c += stride_cols;
    if (c >= vecs) {
      c -= vecs;
      ++row;
    }
  }
};

// 4 n / (1 + exp(-g)): both passes divide by d = (1 + exp(-g)) / 4 with its approximate reciprocal r (1 ulp).  The quarter keeps
// the reciprocal of every finite divisor a normal number; an infinite one is held at a value whose reciprocal is flushed to zero.
// One step of Markstein's, q - r (d q - n) with fused multiply-adds (IBM J. Res. Dev. 34, 1990), brings the quotient to the
// rounding of the exact one; in this form of it a zero keeps its sign.  His theorem wants a correctly rounded r, so it is the gates
// that show it: there are 65,536, and a test divides by all of them.  IEEE divisions have range checks that this needs
// none of.  With them and so, in us: 4096 x 14336 forward 74.0 and 62.8 (352 MB, 5.6 TB/s), backward 107.7 and 106.9; 49,024 x 768
// forward 51.0 and 43.2, backward 73.2 and 68.6.  Without the step a sigmoid that is a unit of fp32 off now and then turns the
// rounding of gradients, and of all that follows from them, and nothing is faster (backward 108.6 and 73.0).
__device__ __forceinline__ float over_sigmoid_divisor(float n, float g) {
  const float d = fminf(fmaf(__expf(-g), 0.25f, 0.25f), 0x1.8p126f);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = n * r;
  return fabsf(n) < 1e37f ? fmaf(-fmaf(d, q, -n), r, q) : q;     // an infinite q has no remainder
}

__device__ __forceinline__ float silu(float g) { return over_sigmoid_divisor(0.25f * g, g); }
__device__ __forceinline__ float sigmoid(float g) { return over_sigmoid_divisor(0.25f, g); }

__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ h13, __nv_bfloat16* __restrict__ act, long long T, int F,
                  int stride_rows, int stride_cols) {
  grid_begin(h13);
  const int vecs = F / 8;
  for (VecWalk w(vecs); w.row < T; w.next(vecs, stride_rows, stride_cols)) {
    const bf16x8* base = reinterpret_cast<const bf16x8*>(h13 + w.row * 2 * F);
    float g[8], u[8], o[8];
    unpack8(base[w.c], g);
    unpack8(base[vecs + w.c], u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = silu(g[j]) * u[j];
    reinterpret_cast<bf16x8*>(act + w.row * F)[w.c] = pack8(o);
  }
}

__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ h13, const __nv_bfloat16* __restrict__ dact,
                  __nv_bfloat16* __restrict__ dh13, long long T, int F, int stride_rows, int stride_cols) {
  grid_begin(h13, dact);
  const int vecs = F / 8;
  for (VecWalk w(vecs); w.row < T; w.next(vecs, stride_rows, stride_cols)) {
    const bf16x8* base = reinterpret_cast<const bf16x8*>(h13 + w.row * 2 * F);
    float g[8], u[8], d[8], dg[8], du[8];
    unpack8(base[w.c], g);
    unpack8(base[vecs + w.c], u);
    unpack8(reinterpret_cast<const bf16x8*>(dact + w.row * F)[w.c], d);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sg = sigmoid(g[j]);
      du[j] = d[j] * (g[j] * sg);
      dg[j] = d[j] * u[j] * sg * (1.f + g[j] * (1.f - sg));
    }
    bf16x8* ob = reinterpret_cast<bf16x8*>(dh13 + w.row * 2 * F);
    ob[w.c] = pack8(dg);
    ob[vecs + w.c] = pack8(du);
  }
}

// ---------------------------------------------------------------- embedding
__global__ void embedding_fwd_kernel(const long long* __restrict__ tokens,
                                     const __nv_bfloat16* __restrict__ table, __nv_bfloat16* __restrict__ out,
                                     long long T, int D, int V, int* status) {
  grid_begin(tokens, table);
  const long long row = blockIdx.x;
  long long tok = tokens[row];
  if (tok < 0 || tok >= V) {   // recorded, not trapped
    if (threadIdx.x == 0) report_bad_argument(status, 41, row, tok);
    tok = 0;
  }
  const bf16x8* src = reinterpret_cast<const bf16x8*>(table + tok * D);
  bf16x8* dst = reinterpret_cast<bf16x8*>(out + row * D);
  for (int i = threadIdx.x; i < D / 8; i += blockDim.x) dst[i] = src[i];
}

// dtable[tok] += dout[row]; fp32 atomics straight into the gradient bucket.
__global__ void embedding_bwd_kernel(const long long* __restrict__ tokens,
                                     const __nv_bfloat16* __restrict__ dout, float* __restrict__ dtable,
                                     long long T, int D, int V) {
  const long long row = blockIdx.x;
  const long long tok = tokens[row];
  if (tok < 0 || tok >= V) return;
  const __nv_bfloat16* src = dout + row * D;
  float* dst = dtable + tok * D;
  for (int i = threadIdx.x; i < D; i += blockDim.x) atomicAdd(dst + i, __bfloat162float(src[i]));
}

// Embedding gradient straight into a bf16 table, cleared first: rows of one token value are summed in fp32 in a compact
// [T, D] buffer at the position of its first occurrence, then rounded once into the table.  The fp32 table it replaces
// cost a clear, a read and a conversion of V rows for the T that are touched.
// owner[v] = T - (lowest position of v), 0 for a value that does not occur: cleared by the same memset as the sums.
__global__ void embedding_owner_kernel(const long long* __restrict__ tokens, int* __restrict__ owner, int T, int V) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  const long long tok = tokens[i];
  if (tok >= 0 && tok < V) atomicMax(owner + tok, T - i);
}

__global__ void __launch_bounds__(128)
embedding_compact_kernel(const long long* __restrict__ tokens, const __nv_bfloat16* __restrict__ dout,
                         const int* __restrict__ owner, float* __restrict__ acc, int T, int D, int V) {
  const long long row = blockIdx.x;
  const long long tok = tokens[row];
  if (tok < 0 || tok >= V) return;
  const bf16x8* src = reinterpret_cast<const bf16x8*>(dout + row * D);
  float4* dst = reinterpret_cast<float4*>(acc + static_cast<long long>(T - owner[tok]) * D);
  for (int i = threadIdx.x; i < D / 8; i += blockDim.x) {
    float f[8];
    unpack8(src[i], f);
    atomicAdd(dst + 2 * i, make_float4(f[0], f[1], f[2], f[3]));
    atomicAdd(dst + 2 * i + 1, make_float4(f[4], f[5], f[6], f[7]));
  }
}

__global__ void __launch_bounds__(128)
embedding_scatter_kernel(const long long* __restrict__ tokens, const int* __restrict__ owner,
                         const float* __restrict__ acc, __nv_bfloat16* __restrict__ dtable, int T, int D, int V) {
  const long long row = blockIdx.x;
  const long long tok = tokens[row];
  if (tok < 0 || tok >= V || T - owner[tok] != row) return;
  const float4* src = reinterpret_cast<const float4*>(acc + row * D);
  bf16x8* dst = reinterpret_cast<bf16x8*>(dtable + tok * D);
  for (int i = threadIdx.x; i < D / 8; i += blockDim.x) {
    const float4 a = src[2 * i], b = src[2 * i + 1];
    const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    dst[i] = pack8(f);
  }
}

// ------------------------------------------------------------ cross-entropy
// One CTA per row of bf16 logits [T, V]: online max / sum-exp, per-token loss
// and log-sum-exp.  ignore_index rows produce loss 0.
constexpr int CE_THREADS = 512;

__global__ void __launch_bounds__(CE_THREADS)
ce_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
              float* __restrict__ loss, float* __restrict__ lse, int V, long long ld,
              long long ignore_index) {
  grid_begin(logits, labels);
  __shared__ float scratch[32];
  const long long row = blockIdx.x;
  const __nv_bfloat16* lr = logits + row * ld;
  const int nvec = V / 8;
  float m = -INFINITY, s = 0.f;
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    float f[8];
    unpack8(reinterpret_cast<const bf16x8*>(lr)[i], f);
    float lm = f[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) lm = fmaxf(lm, f[j]);
    if (lm > m) {
      s *= __expf(m - lm);
      m = lm;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += __expf(f[j] - m);
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += CE_THREADS) {
    const float f = __bfloat162float(lr[i]);
    if (f > m) {
      s *= __expf(m - f);
      m = f;
    }
    s += __expf(f - m);
  }
  const float gm = block_max<CE_THREADS>(m, scratch);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum<CE_THREADS>(s, scratch);
  if (threadIdx.x == 0) {
    const float l = gm + logf(gs);
    lse[row] = l;
    const long long y = labels[row];
    loss[row] = (y == ignore_index || y < 0 || y >= V) ? 0.f : l - __bfloat162float(lr[y]);
  }
}

// mean = sum(loss) / n over the n rows whose label is not ignore_index (1 where there is none), and n.  One CTA: a sum, a
// comparison, a conversion, a count, a clamp and a division as launches of their own: 128 x 1024 logits, forward and backward,
// 175 us a pass and 137 with this kernel; 4096 x 32000 190 and 162.
__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ loss, const long long* __restrict__ labels, float* __restrict__ mean,
               float* __restrict__ count, long long T, long long ignore_index) {
  grid_begin(loss, labels);
  __shared__ double sums[32];
  __shared__ int counts[32];
  double s = 0.0;
  int n = 0;
#pragma unroll 4
  for (long long i = threadIdx.x; i < T; i += 1024) {
    s += loss[i];
    n += labels[i] != ignore_index;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sums[threadIdx.x >> 5] = s;
    counts[threadIdx.x >> 5] = n;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  s = 0.0;
  n = 0;
  for (int w = 0; w < 32; ++w) {
    s += sums[w];
    n += counts[w];
  }
  if (n < 1) n = 1;
  *mean = static_cast<float>(s / n);
  *count = static_cast<float>(n);
}

// dlogits = (softmax - onehot) * gscale[0] * row_scale, written to `out`
// (may alias logits).
__global__ void __launch_bounds__(CE_THREADS)
ce_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const long long* __restrict__ labels,
              const float* __restrict__ lse, const float* __restrict__ gscale, float row_scale,
              __nv_bfloat16* __restrict__ out, int V, long long ld, long long ignore_index) {
  grid_begin(logits, labels, lse, gscale);
  const long long row = blockIdx.x;
  const __nv_bfloat16* lr = logits + row * ld;
  __nv_bfloat16* orow = out + row * ld;
  const long long y = labels[row];
  const bool ignored = (y == ignore_index || y < 0 || y >= V);
  const float sc = ignored ? 0.f : gscale[0] * row_scale;
  const float l = lse[row];
  const int nvec = V / 8;
  for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
    float f[8];
    unpack8(reinterpret_cast<const bf16x8*>(lr)[i], f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float p = __expf(f[j] - l);
      f[j] = (p - ((i * 8 + j) == y ? 1.f : 0.f)) * sc;
    }
    reinterpret_cast<bf16x8*>(orow)[i] = pack8(f);
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += CE_THREADS) {
    const float p = __expf(__bfloat162float(lr[i]) - l);
    orow[i] = __float2bfloat16((p - (i == y ? 1.f : 0.f)) * sc);
  }
}

// --------------------------------------------------------------------- Adam
// Flat-buffer Adam / AdamW: fp32 master / m / v, fp32 gradient (scaled by
// grad_scale), bf16 parameter copy written in the same pass.  decoupled != 0
// is AdamW (the decay shrinks the weight directly); otherwise the decay is
// the L2 term of torch.optim.Adam, added to the gradient before the moments.
__global__ void adam_flat_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v,
                                 const float* __restrict__ grad, __nv_bfloat16* __restrict__ param,
                                 long long n, float lr, float b1, float b2, float eps, float wd,
                                 float bc1, float bc2, float grad_scale, int decoupled) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float p = master[i];
    float g = grad[i] * grad_scale;
    if (!decoupled) g += wd * p;
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float denom = sqrtf(vi / bc2) + eps;
    p = p - lr * (mi / bc1) / denom - (decoupled ? lr * wd * p : 0.f);
    master[i] = p;
    if (param) param[i] = __float2bfloat16(p);
  }
}

__global__ void cast_f32_to_bf16_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out,
                                        long long n, float scale) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    out[i] = __float2bfloat16(in[i] * scale);
}

// acc (fp32) += g (bf16): gradient accumulation into the flat bucket for
// parameters whose gradient comes from autograd as a bf16 tensor.
__global__ void accum_bf16_into_f32_kernel(const __nv_bfloat16* __restrict__ g, float* __restrict__ acc,
                                           long long n) {
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    acc[i] += __bfloat162float(g[i]);
}

// out = a + b over n bf16 elements (n % 8 == 0): the residual add at a stage boundary.
__global__ void add_bf16_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ b,
                                __nv_bfloat16* __restrict__ out, long long nvec) {
  grid_begin(a, b);
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    float x[8], y[8];
    unpack8(reinterpret_cast<const bf16x8*>(a)[i], x);
    unpack8(reinterpret_cast<const bf16x8*>(b)[i], y);
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] += y[j];
    reinterpret_cast<bf16x8*>(out)[i] = pack8(x);
  }
}

// True when every non-null pointer is 16-byte aligned (the kernels use 16-byte vector accesses).
template <typename... P>
inline bool aligned16(P... ptrs) {
  return ((reinterpret_cast<uintptr_t>(static_cast<const void*>(ptrs)) | ...) & 15u) == 0;
}

inline int grid_for(long long work, int threads, int max_blocks = 148 * 16) {
  long long b = (work + threads - 1) / threads;
  if (b > max_blocks) b = max_blocks;
  if (b < 1) b = 1;
  return static_cast<int>(b);
}

}  // namespace

#define PIPER_LAUNCH_OK() (cudaGetLastError() == cudaSuccess ? 0 : -3)

// Vectors per thread of the register-resident kernels: as few as leave a row at most 256 threads.  0: the row does not divide.
static int norm_vectors(int D) {
  if (D % 256 == 0 && D <= 2048) return 1;
  if (D % 512 == 0 && D <= 4096) return 2;
  return D % 1024 == 0 && D <= 8192 ? 4 : 0;
}

// Calls fn with the vectors and threads of a row of D elements as constants; false where there are none.
template <class F>
static bool with_norm_shape(int D, F fn) {
  const int vpt = norm_vectors(D);
  auto at = [&](auto v) {
    constexpr int V = decltype(v)::value;
    switch (D / (256 * V)) {
      case 8: fn(v, std::integral_constant<int, 256>()); return;
      case 7: fn(v, std::integral_constant<int, 224>()); return;
      case 6: fn(v, std::integral_constant<int, 192>()); return;
      case 5: fn(v, std::integral_constant<int, 160>()); return;
      default: break;
    }
    if constexpr (V == 1) {
      switch (D / 256) {
        case 4: fn(v, std::integral_constant<int, 128>()); return;
        case 3: fn(v, std::integral_constant<int, 96>()); return;
        case 2: fn(v, std::integral_constant<int, 64>()); return;
        default: fn(v, std::integral_constant<int, 32>()); return;
      }
    }
  };
  if (vpt == 1) at(std::integral_constant<int, 1>());
  else if (vpt == 2) at(std::integral_constant<int, 2>());
  else if (vpt == 4) at(std::integral_constant<int, 4>());
  return vpt != 0;
}

int rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd,
                long long T, int D, float eps, int num_sms, cudaStream_t st) {
  if (D % 8 != 0) return -1;
  if (T == 0) return 0;
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  const auto* rp = static_cast<const __nv_bfloat16*>(res);
  const auto* wp = static_cast<const __nv_bfloat16*>(w);
  auto* yp = static_cast<__nv_bfloat16*>(y);
  auto* hp = static_cast<__nv_bfloat16*>(h_out);
  const bool done = with_norm_shape(D, [&](auto vpt, auto threads) {
    constexpr int VPT = decltype(vpt)::value, THREADS = decltype(threads)::value;
    const long long ctas = static_cast<long long>(NORM_FWD_CTAS<VPT, THREADS>) * num_sms;
    launch_overlapped(rmsnorm_fwd_reg_kernel<VPT, THREADS>, static_cast<unsigned>(T < ctas ? T : ctas), THREADS, 0, st, xp, rp, wp, yp, hp, rstd, T, eps);
  });
  if (done) return PIPER_LAUNCH_OK();
  launch_overlapped(rmsnorm_fwd_kernel, static_cast<unsigned>(T), NORM_THREADS, 0, st,
      static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(res),
      static_cast<const __nv_bfloat16*>(w), static_cast<__nv_bfloat16*>(y),
      static_cast<__nv_bfloat16*>(h_out), rstd, D, eps);
  return PIPER_LAUNCH_OK();
}

// Two strips per SM of a 148-SM part, whatever the device: the allocation-free entry point sizes its built-in
// scratch array (PIPER_NOALLOC_MAX_STRIPS) from this fixed bound.
int rmsnorm_bwd_num_partials(long long T) {
  const int cap = 148 * 2;
  return static_cast<int>(T < cap ? (T > 0 ? T : 1) : cap);
}

int rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres,
                void* dx, float* dw_partial, float* dw_f32, void* dw_bf16, int accumulate, long long T,
                int D, cudaStream_t st) {
  if (D % 8 != 0 || D * sizeof(float) > 160 * 1024) return -1;
  if (T < 0 || T > 2147483647LL) return -1;      // the kernels index rows with a 32-bit int
  if (T == 0) return 0;
  const int nb = rmsnorm_bwd_num_partials(T);
  const dim3 red_grid((D + 31) / 32), red_block(32, RED_SLICES);
  const WeightGrad out{dw_f32, static_cast<__nv_bfloat16*>(dw_bf16), accumulate};
  const bool done = with_norm_shape(D, [&](auto vpt, auto threads) {
    constexpr int VPT = decltype(vpt)::value, THREADS = decltype(threads)::value;
    // several rows at a time where a CTA has several to do
    const long long each = (T + nb - 1) / nb;
    const int rows = static_cast<int>(each < NORM_BWD_ROWS<VPT, THREADS> ? each : NORM_BWD_ROWS<VPT, THREADS>);
    launch_overlapped(rmsnorm_bwd_reg_kernel<VPT, THREADS>, nb, rows * THREADS, rows > 1 ? rows * D * sizeof(float) : 0, st,
        static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), rstd,
        static_cast<const __nv_bfloat16*>(dres), static_cast<__nv_bfloat16*>(dx), dw_partial, static_cast<int>(T));
  });
  if (done) {
    launch_overlapped(reduce_partials_kernel, red_grid, red_block, 0, st, dw_partial, nb, D, out, out, D);
    return PIPER_LAUNCH_OK();
  }
  static bool configured = false;
  if (!configured) {
    cudaFuncSetAttribute(rmsnorm_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
    configured = true;
  }
  launch_overlapped(rmsnorm_bwd_kernel, nb, NORM_THREADS, D * sizeof(float), st,
      static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x),
      static_cast<const __nv_bfloat16*>(w), rstd, static_cast<const __nv_bfloat16*>(dres),
      static_cast<__nv_bfloat16*>(dx), dw_partial, static_cast<int>(T), D);
  launch_overlapped(reduce_partials_kernel, red_grid, red_block, 0, st, dw_partial, nb, D, out, out, D);
  return PIPER_LAUNCH_OK();
}

// `grid` is the most CTAs that may run, or 0, and becomes those that do.
// Heads of a task: more of them share one load of cos/sin and fetch ahead, fewer make more tasks to run at a time.
// Four per lane group at 128 (two at 64, whose runs would span half a token) where that leaves two tasks per resident warp.
// In us for 1, 2, 4 and 8 heads per lane group: 4096 x (32 + 2 x 4) x 128 with norms forward 21.6 19.6 19.7 21.8, backward 36.5 32.9
// 32.7 32.8; 16384 tokens 75.7 66.5 64.2 63.7, 123.3 108.8 103.8 101.1; 8192 x (32 + 2 x 8) x 128 38.0 35.8 35.4 36.1; 8192 x (32 +
// 2 x 8) x 64 30.2 29.2 30.2 30.2; 128 x (32 + 2 x 8) x 128 2.6 2.7 3.4 4.6.
template <int HD, bool NORM, bool BWD>
static int qk_rope_launch(RopeArgs a, bool interleaved, int num_sms, int& grid, cudaStream_t st) {
  int resident = ROPE_CTAS<NORM, BWD> * num_sms;
  if (grid > 0 && grid < resident) resident = grid;
  auto tasks = [&](int run) { return a.T * ((a.Hq + run - 1) / run + 2ll * ((a.Hkv + run - 1) / run)); };
  constexpr int groups = RopeGroup<HD>::GROUPS;
  a.run = (HD == 128 ? 4 : 2) * groups;
  while (a.run > groups && tasks(a.run) < 2ll * 8 * resident) a.run /= 2;
  if (tasks(a.run) >= (1ll << 31)) return -1;
  const long long blocks = (tasks(a.run) + 7) / 8;
  grid = static_cast<int>(blocks < resident ? blocks : resident);
  auto kern = interleaved ? qk_rope_kernel<HD, NORM, BWD, true> : qk_rope_kernel<HD, NORM, BWD, false>;
  launch_overlapped(kern, grid, 256, 0, st, a);
  return PIPER_LAUNCH_OK();
}

template <bool BWD>
static int qk_rope(const RopeArgs& a, int hd, bool interleaved, int num_sms, int& grid, cudaStream_t st) {
  if (a.T == 0 || a.Hq + 2 * a.Hkv == 0) {
    grid = 0;
    return 0;
  }
  if (hd != 128 && hd != 64) return -1;
  if (static_cast<long long>(a.S) * (hd / 2) >= (1ll << 31)) return -1;
  if (!aligned16(a.x, a.pre, a.out, a.cosp, a.sinp, a.qw, a.kw)) return -4;
  if (a.qw != nullptr || a.kw != nullptr)
    return hd == 128 ? qk_rope_launch<128, true, BWD>(a, interleaved, num_sms, grid, st)
                     : qk_rope_launch<64, true, BWD>(a, interleaved, num_sms, grid, st);
  return hd == 128 ? qk_rope_launch<128, false, BWD>(a, interleaved, num_sms, grid, st)
                   : qk_rope_launch<64, false, BWD>(a, interleaved, num_sms, grid, st);
}

int qk_rope_fwd(const void* in, void* out, const float* cosp, const float* sinp, const void* qw,
                const void* kw, long long T, int S, int Hq, int Hkv, int hd, int interleaved, float eps,
                int num_sms, cudaStream_t st) {
  const RopeArgs a{static_cast<const __nv_bfloat16*>(in), nullptr, static_cast<__nv_bfloat16*>(out), cosp, sinp,
                   static_cast<const __nv_bfloat16*>(qw), static_cast<const __nv_bfloat16*>(kw), nullptr,
                   T, S, Hq, Hkv, eps, 0};
  int grid = 0;
  return qk_rope<false>(a, hd, interleaved != 0, num_sms, grid, st);
}

int qk_rope_bwd(const void* dout, const void* in, void* din, const float* cosp, const float* sinp,
                const void* qw, const void* kw, float* partial, int strips, float* dqw_f32, void* dqw_bf16, float* dkw_f32,
                void* dkw_bf16, long long T, int S, int Hq, int Hkv, int hd, int interleaved, float eps, int num_sms,
                cudaStream_t st) {
  // buckets add up, bf16 gradients are written (zeros where there are no tokens)
  const WeightGrad q{dqw_f32, static_cast<__nv_bfloat16*>(dqw_bf16), dqw_f32 != nullptr};
  const WeightGrad k{dkw_f32, static_cast<__nv_bfloat16*>(dkw_bf16), dkw_f32 != nullptr};
  const bool want_q = q.f32 || q.bf16, want_k = k.f32 || k.bf16;
  const RopeArgs a{static_cast<const __nv_bfloat16*>(dout), static_cast<const __nv_bfloat16*>(in),
                   static_cast<__nv_bfloat16*>(din), cosp, sinp, static_cast<const __nv_bfloat16*>(qw),
                   static_cast<const __nv_bfloat16*>(kw), want_q || want_k ? partial : nullptr, T, S, Hq, Hkv, eps, 0};
  if ((want_q && !qw) || (want_k && !kw) || ((want_q || want_k) && (!partial || strips < 1))) return -1;
  int grid = want_q || want_k ? strips : 0;
  const int rc = qk_rope<true>(a, hd, interleaved != 0, num_sms, grid, st);
  if (rc != 0 || !(want_q || want_k)) return rc;
  const WeightGrad none{nullptr, nullptr, 0};
  const bool same = want_q && want_k && (q.f32 ? q.f32 == k.f32 : q.bf16 == k.bf16);   // one weight for both: in turn
  launch_overlapped(reduce_partials_kernel, 2 * hd / 32, dim3(32, RED_SLICES), 0, st, partial, grid, 2 * hd, q, same ? none : k, hd);
  if (same) launch_overlapped(reduce_partials_kernel, 2 * hd / 32, dim3(32, RED_SLICES), 0, st, partial, grid, 2 * hd, none, k, hd);
  return PIPER_LAUNCH_OK();
}

int swiglu_fwd(const void* h13, void* act, long long T, int F, cudaStream_t st) {
  if (F % 8 != 0) return -1;
  if (T == 0) return 0;
  const int vecs = F / 8;
  const int blocks = grid_for(T * vecs, 256);
  const long long stride = static_cast<long long>(blocks) * 256;
  launch_overlapped(swiglu_fwd_kernel, blocks, 256, 0, st, static_cast<const __nv_bfloat16*>(h13), static_cast<__nv_bfloat16*>(act), T,
                                            F, static_cast<int>(stride / vecs), static_cast<int>(stride % vecs));
  return PIPER_LAUNCH_OK();
}

int swiglu_bwd(const void* h13, const void* dact, void* dh13, long long T, int F, cudaStream_t st) {
  if (F % 8 != 0) return -1;
  if (T == 0) return 0;
  const int vecs = F / 8;
  const int blocks = grid_for(T * vecs, 256);
  const long long stride = static_cast<long long>(blocks) * 256;
  launch_overlapped(swiglu_bwd_kernel, blocks, 256, 0, st, static_cast<const __nv_bfloat16*>(h13),
                                            static_cast<const __nv_bfloat16*>(dact), static_cast<__nv_bfloat16*>(dh13),
                                            T, F, static_cast<int>(stride / vecs), static_cast<int>(stride % vecs));
  return PIPER_LAUNCH_OK();
}

int embedding_fwd(const long long* tokens, const void* table, void* out, long long T, int D, int V,
                  int* status, cudaStream_t st) {
  if (D % 8 != 0) return -1;
  if (T == 0) return 0;
  launch_overlapped(embedding_fwd_kernel, static_cast<unsigned>(T), 128, 0, st,
      tokens, static_cast<const __nv_bfloat16*>(table), static_cast<__nv_bfloat16*>(out), T, D, V, status);
  return PIPER_LAUNCH_OK();
}

int embedding_bwd(const long long* tokens, const void* dout, float* dtable, long long T, int D, int V,
                  cudaStream_t st) {
  if (T == 0) return 0;
  embedding_bwd_kernel<<<static_cast<unsigned>(T), 256, 0, st>>>(
      tokens, static_cast<const __nv_bfloat16*>(dout), dtable, T, D, V);
  return PIPER_LAUNCH_OK();
}

long long embedding_bwd_scratch(long long T, int D, int V) { return (V + 3ll) / 4 * 4 + T * D; }

int embedding_bwd_bf16(const long long* tokens, const void* dout, int* scratch, void* dtable, long long T, int D, int V,
                       cudaStream_t st) {
  if (D % 8 != 0 || T >= (1ll << 31)) return -1;
  if (cudaMemsetAsync(dtable, 0, static_cast<size_t>(V) * D * 2, st) != cudaSuccess) return -3;
  if (T == 0) return 0;
  const long long words = embedding_bwd_scratch(T, D, V);
  if (cudaMemsetAsync(scratch, 0, static_cast<size_t>(words) * 4, st) != cudaSuccess) return -3;
  float* acc = reinterpret_cast<float*>(scratch + (words - T * D));
  const unsigned n = static_cast<unsigned>(T);
  const int t = static_cast<int>(T);
  embedding_owner_kernel<<<(n + 255) / 256, 256, 0, st>>>(tokens, scratch, t, V);
  embedding_compact_kernel<<<n, 128, 0, st>>>(tokens, static_cast<const __nv_bfloat16*>(dout), scratch, acc, t, D, V);
  embedding_scatter_kernel<<<n, 128, 0, st>>>(tokens, scratch, acc, static_cast<__nv_bfloat16*>(dtable), t, D, V);
  return PIPER_LAUNCH_OK();
}

int ce_fwd(const void* logits, const long long* labels, float* loss, float* lse, long long T, int V,
           long long ld, long long ignore_index, cudaStream_t st) {
  if (ld % 8 != 0) return -1;
  if (T == 0) return 0;
  launch_overlapped(ce_fwd_kernel, static_cast<unsigned>(T), CE_THREADS, 0, st,
      static_cast<const __nv_bfloat16*>(logits), labels, loss, lse, V, ld, ignore_index);
  return PIPER_LAUNCH_OK();
}

int ce_mean(const float* loss, const long long* labels, float* mean, float* count, long long T, long long ignore_index,
            cudaStream_t st) {
  if (T < 0 || T >= (1ll << 24)) return -1;      // the count is exact in fp32
  launch_overlapped(ce_mean_kernel, 1, 1024, 0, st, loss, labels, mean, count, T, ignore_index);
  return PIPER_LAUNCH_OK();
}

int ce_bwd(const void* logits, const long long* labels, const float* lse, const float* gscale,
           float row_scale, void* out, long long T, int V, long long ld, long long ignore_index,
           cudaStream_t st) {
  if (ld % 8 != 0) return -1;
  if (T == 0) return 0;
  launch_overlapped(ce_bwd_kernel, static_cast<unsigned>(T), CE_THREADS, 0, st,
      static_cast<const __nv_bfloat16*>(logits), labels, lse, gscale, row_scale,
      static_cast<__nv_bfloat16*>(out), V, ld, ignore_index);
  return PIPER_LAUNCH_OK();
}

int adam_flat(float* master, float* m, float* v, const float* grad, void* param_bf16, long long n,
              float lr, float b1, float b2, float eps, float wd, int step, float grad_scale, int decoupled,
              cudaStream_t st) {
  if (n == 0) return 0;
  const float bc1 = 1.f - powf(b1, static_cast<float>(step));
  const float bc2 = 1.f - powf(b2, static_cast<float>(step));
  adam_flat_kernel<<<grid_for(n, 256), 256, 0, st>>>(master, m, v, grad,
                                                    static_cast<__nv_bfloat16*>(param_bf16), n, lr, b1, b2,
                                                    eps, wd, bc1, bc2, grad_scale, decoupled);
  return PIPER_LAUNCH_OK();
}

int cast_f32_to_bf16(const float* in, void* out, long long n, float scale, cudaStream_t st) {
  if (n == 0) return 0;
  cast_f32_to_bf16_kernel<<<grid_for(n, 256), 256, 0, st>>>(in, static_cast<__nv_bfloat16*>(out), n, scale);
  return PIPER_LAUNCH_OK();
}

int add_bf16(const void* a, const void* b, void* out, long long n, cudaStream_t st) {
  if (n % 8 != 0) return -1;
  if (n == 0) return 0;
  launch_overlapped(add_bf16_kernel, grid_for(n / 8, 256), 256, 0, st, static_cast<const __nv_bfloat16*>(a),
                                                       static_cast<const __nv_bfloat16*>(b),
                                                       static_cast<__nv_bfloat16*>(out), n / 8);
  return PIPER_LAUNCH_OK();
}

int accum_bf16_into_f32(const void* g, float* acc, long long n, cudaStream_t st) {
  if (n == 0) return 0;
  accum_bf16_into_f32_kernel<<<grid_for(n, 256), 256, 0, st>>>(static_cast<const __nv_bfloat16*>(g), acc, n);
  return PIPER_LAUNCH_OK();
}

}  // namespace piper
