// Mixture-of-experts routing kernels for sm_100a: softmax + top-k router,
// scatter of token rows into zero-padded per-expert segments, weighted
// combine, and the backward passes.  One warp handles one token.
#include "moe.h"

#include "ptx.cuh"

#include <cuda_bf16.h>
#include <stdint.h>

namespace piper {
namespace {

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

constexpr int MAX_PER_LANE = 8;   // E <= 256
constexpr int MAX_K = 8;

// Softmax probabilities of one token, E/32 values per lane (expert e lives in
// lane e % 32, slot e / 32).
template <int SLOTS>
__device__ __forceinline__ void token_softmax(const __nv_bfloat16* row, int E, int lane, float (&p)[SLOTS]) {
  float mx = -INFINITY;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    const int e = s * 32 + lane;
    p[s] = (e < E) ? __bfloat162float(row[e]) : -INFINITY;
    mx = fmaxf(mx, p[s]);
  }
  mx = warp_max(mx);
  float sum = 0.f;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) {
    p[s] = (s * 32 + lane < E) ? __expf(p[s] - mx) : 0.f;
    sum += p[s];
  }
  sum = warp_sum(sum);
  const float inv = 1.f / sum;
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) p[s] *= inv;
}

// Bound by the serial chain of k arg-max rounds: probabilities are compared as integers (same order for values >= 0,
// and a NaN stays selectable instead of selecting nothing), so a round is two warp reductions in hardware; lane j
// keeps the j-th choice and the k results are written, and counted, at once.  4096 tokens, 128 experts, top 8:
// 17 us with ten shuffles a round and one lane writing, 10 us so.
template <int SLOTS>
__global__ void route_kernel(const __nv_bfloat16* __restrict__ logits, float* __restrict__ weights,
                             int* __restrict__ idx, int* __restrict__ counts, long long T, int E, int k,
                             int renorm) {
  grid_begin(logits);
  const long long t = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  float p[SLOTS];
  token_softmax<SLOTS>(logits + t * E, E, lane, p);
  int key[SLOTS];
#pragma unroll
  for (int s = 0; s < SLOTS; ++s) key[s] = s * 32 + lane < E ? (__float_as_int(p[s]) & 0x7fffffff) : -1;
  float my_w = 0.f, total = 0.f;
  int my_e = 0;
  for (int j = 0; j < k; ++j) {
    // arg-max over the remaining probabilities; ties go to the lower expert index
    int best = key[0], slot = 0;
#pragma unroll
    for (int s = 1; s < SLOTS; ++s)
      if (key[s] > best) { best = key[s]; slot = s; }
    const int top = __reduce_max_sync(0xffffffffu, best);
    const int e = __reduce_min_sync(0xffffffffu, best == top ? slot * 32 + lane : 0x7fffffff);
    const float w = __int_as_float(top);
    total += w;
    if (lane == j) { my_w = w; my_e = e; }
#pragma unroll
    for (int s = 0; s < SLOTS; ++s)
      if (s * 32 + lane == e) key[s] = -1;     // remove from further rounds
  }
  if (lane < k) {
    weights[t * k + lane] = my_w * (renorm ? 1.f / total : 1.f);
    idx[t * k + lane] = my_e;
    atomicAdd(counts + my_e, 1);
  }
}

// w_j = p_j / S (renorm) or p_j; dp_i for selected i, then dlogits = p * (dp - <dp, p>).
__global__ void route_bwd_kernel(const __nv_bfloat16* __restrict__ logits, const int* __restrict__ idx,
                                 const float* __restrict__ weights, const float* __restrict__ dweights,
                                 __nv_bfloat16* __restrict__ dlogits, long long T, int E, int k, int renorm) {
  grid_begin(logits, idx, weights, dweights);
  const long long t = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  float p[MAX_PER_LANE], dp[MAX_PER_LANE];
  token_softmax<MAX_PER_LANE>(logits + t * E, E, lane, p);
#pragma unroll
  for (int s = 0; s < MAX_PER_LANE; ++s) dp[s] = 0.f;
  float S = 1.f, dot_w = 0.f;
  if (renorm) {
    S = 0.f;
    for (int j = 0; j < k; ++j) {
      const int e = idx[t * k + j];
      const float pe = __shfl_sync(0xffffffffu, p[e >> 5], e & 31);
      S += pe;
      dot_w += dweights[t * k + j] * weights[t * k + j];
    }
  }
  for (int j = 0; j < k; ++j) {
    const int e = idx[t * k + j];
    const float g = renorm ? (dweights[t * k + j] - dot_w) / S : dweights[t * k + j];
    if ((e & 31) == lane) dp[e >> 5] = g;
  }
  float inner = 0.f;
#pragma unroll
  for (int s = 0; s < MAX_PER_LANE; ++s) inner += dp[s] * p[s];
  inner = warp_sum(inner);
#pragma unroll
  for (int s = 0; s < MAX_PER_LANE; ++s) {
    const int e = s * 32 + lane;
    if (e < E) dlogits[t * E + e] = __float2bfloat16(p[s] * (dp[s] - inner));
  }
}

// One warp: a scan over each source's segments (one thread walking 128 groups took 5 us of dependent loads).  It also clears
// the permutation's cursors and copies the counts where a dispatch wants them: launches of their own took longer than this.
__global__ void group_table_kernel(const int* __restrict__ counts, int num_groups, int experts,
                                   const int* __restrict__ row_base, int* __restrict__ g_start,
                                   int* __restrict__ g_len, int* __restrict__ total, int* __restrict__ cursor,
                                   int* __restrict__ copy) {
  grid_begin(counts, row_base);
  const int lane = threadIdx.x;
  int run = 0, last = 0;
  for (int s0 = 0; s0 < num_groups; s0 += experts) {
    if (row_base != nullptr) run = row_base[s0 / experts];
    const int n = min(experts, num_groups - s0);
#pragma unroll 4
    for (int e0 = 0; e0 < n; e0 += 32) {
      const int g = s0 + e0 + lane;
      const bool in = e0 + lane < n;
      const int n_g = in ? counts[g] : 0;
      const int len = (n_g + 127) / 128 * 128;
      int inc = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (in) {
        g_start[g] = run + inc - len;
        g_len[g] = len;
        if (cursor != nullptr) cursor[g] = 0;
        if (copy != nullptr) copy[g] = n_g;
      }
      run += __shfl_sync(0xffffffffu, inc, 31);
      if (run > last) last = run;
    }
  }
  if (lane == 0 && total != nullptr) total[0] = last;
}

constexpr int ROW_THREADS = 128;      // four tokens per CTA: enough CTAs for the small token counts
constexpr int PAD_CTAS = 4;           // CTAs that clear the padding of one group

// Zeroes part `part` of rows [g_start + counts, g_start + g_len) of group g.
__device__ __forceinline__ void zero_padding(__nv_bfloat16* __restrict__ rows, const int* __restrict__ g_start,
                                             const int* __restrict__ g_len, const int* __restrict__ counts, int g,
                                             int part, int D, long long rows_cap, int* status) {
  const int first = g_start[g] + counts[g];
  const int last = g_start[g] + g_len[g];
  if (counts[g] < 0 || g_start[g] < 0 || last < first || last > rows_cap) {
    if (threadIdx.x == 0 && part == 0) report_bad_argument(status, 35, g, last);
    return;                                   // a segment outside the buffer is left alone
  }
  const uint4 z = make_uint4(0, 0, 0, 0);
  const long long nvec = static_cast<long long>(last - first) * (D / 8);
  uint4* base = reinterpret_cast<uint4*>(rows + static_cast<long long>(first) * D);
  for (long long i = part * ROW_THREADS + threadIdx.x; i < nvec; i += PAD_CTAS * ROW_THREADS) base[i] = z;
}

// One warp per token: the first k lanes claim the rows of its entries together, then the token row is read once and
// written k times; the first CTAs clear the padding rows of the segments (behind the tokens' they would be a tail of long
// CTAs: 8192 x 2048 over 64 experts, top 8, 91.3 us behind and 88.6 us in front).  4096 tokens x 2048, top 8 of 128: 47 us with
// the clearing in a launch of its own, 46 us together; 4096 x 4096, top 2 of 8: 41 and 21 us.
__global__ void __launch_bounds__(ROW_THREADS)
permute_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ idx, const int* __restrict__ g_start,
               const int* __restrict__ g_len, const int* __restrict__ counts, int* __restrict__ cursor,
               int* __restrict__ pos, __nv_bfloat16* __restrict__ rows, long long T, int D, int k, int E,
               long long rows_cap, unsigned token_ctas, int* status) {
  grid_begin(x, idx, g_start, g_len, counts);
  const unsigned pad_ctas = E * PAD_CTAS;
  if (blockIdx.x < pad_ctas) {
    const int b = static_cast<int>(blockIdx.x);
    zero_padding(rows, g_start, g_len, counts, b / PAD_CTAS, b % PAD_CTAS, D, rows_cap, status);
    return;
  }
  const long long t = (static_cast<long long>(blockIdx.x - pad_ctas) * ROW_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  const uint4* src = reinterpret_cast<const uint4*>(x + t * D);
  const int nvec = D / 8;
  for (int j0 = 0; j0 < k; j0 += 32) {
    const int kk = min(32, k - j0);
    int mine = -1;
    if (lane < kk) {
      const long long slot = t * k + j0 + lane;
      const int e = idx[slot];
      if (e >= 0 && e < E) mine = g_start[e] + atomicAdd(cursor + e, 1);
      if (mine < 0 || mine >= rows_cap) {       // rejected: recorded, the copy is skipped
        report_bad_argument(status, 31, e, mine);
        mine = -1;
      }
      pos[slot] = mine < 0 ? 0 : mine;
    }
    for (int i0 = 0; i0 < nvec; i0 += 128) {
      uint4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u * 32 + lane < nvec) v[u] = src[i0 + u * 32 + lane];
      for (int j = 0; j < kk; ++j) {
        const int r = __shfl_sync(0xffffffffu, mine, j);
        if (r < 0) continue;
        uint4* dst = reinterpret_cast<uint4*>(rows + static_cast<long long>(r) * D);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (i0 + u * 32 + lane < nvec) dst[i0 + u * 32 + lane] = v[u];
      }
    }
  }
}

// The rows of a token's entries [j0, j0 + K), one per lane, then broadcast: the gather loops below keep K loads in
// flight per lane instead of one that waits for its own index.  A row outside the buffer is reported and becomes -1.
template <int K>
__device__ __forceinline__ void token_rows(const int* __restrict__ pos, long long t, int k, int j0, int lane,
                                           long long rows_cap, int tag, int* status, int (&r)[K]) {
  int mine = -1;
  if (lane < K && j0 + lane < k) {
    mine = pos[t * k + j0 + lane];
    if (mine < 0 || mine >= rows_cap) {
      report_bad_argument(status, tag, t, mine);
      mine = -1;
    }
  }
#pragma unroll
  for (int j = 0; j < K; ++j) r[j] = __shfl_sync(0xffffffffu, mine, j);
}

// out[t] = sum_j weights[t, j] * rows[pos[t, j]] (weights == nullptr: plain sum); K entries at a time, any k.
// 4096 tokens x 2048, top 8: 50 us with one row in flight per lane, 32 us (4.7 TB/s) with eight.
template <int K>
__global__ void __launch_bounds__(ROW_THREADS)
gather_sum_kernel(const __nv_bfloat16* __restrict__ rows, const int* __restrict__ pos,
                  const float* __restrict__ weights, __nv_bfloat16* __restrict__ out, long long T, int D, int k,
                  long long rows_cap, int tag, int* status) {
  grid_begin(rows, pos, weights);
  const long long t = (static_cast<long long>(blockIdx.x) * ROW_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  int r[K];
  float w[K];
  auto load_entries = [&](int j0) {
    token_rows<K>(pos, t, k, j0, lane, rows_cap, tag, status, r);
#pragma unroll
    for (int j = 0; j < K; ++j) w[j] = weights == nullptr ? 1.f : j0 + j < k ? weights[t * k + j0 + j] : 0.f;
  };
  load_entries(0);
  // one or two entries: the launcher passes k == K, and the loads of four or two vectors go out together
#pragma unroll (K >= 4 ? 1 : 4 / K)
  for (int i0 = 0; i0 < D / 8; i0 += 32) {
    const int i = i0 + lane;
    const bool in = i < D / 8;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j0 = 0; j0 < (K >= 4 ? k : K); j0 += K) {
      if (K >= 4 && k > K) load_entries(j0);
      uint4 q[K];
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (in && r[j] >= 0) q[j] = reinterpret_cast<const uint4*>(rows + static_cast<long long>(r[j]) * D)[i];
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (!in || r[j] < 0) continue;
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q[j]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 f = __bfloat1622float2(h[c]);
          acc[2 * c] += w[j] * f.x;
          acc[2 * c + 1] += w[j] * f.y;
        }
      }
    }
    if (in) {
      uint4 o;
      __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int c = 0; c < 4; ++c) oh[c] = __floats2bfloat162_rn(acc[2 * c], acc[2 * c + 1]);
      reinterpret_cast<uint4*>(out + t * D)[i] = o;
    }
  }
}

// drows[pos[t, j]] = weights[t, j] * dout[t], dweights[t, j] = <rows[pos[t, j]], dout[t]>; K entries share one read
// of dout.  The CTAs behind the tokens' clear the padding rows of drows.  4096 tokens x 2048, top 8: 59 us + 10 us of
// clearing with one row at a time, 49 us together.
template <int K>
__global__ void __launch_bounds__(ROW_THREADS)
combine_bwd_kernel(const __nv_bfloat16* __restrict__ rows, const __nv_bfloat16* __restrict__ dout,
                   const int* __restrict__ pos, const float* __restrict__ weights,
                   __nv_bfloat16* __restrict__ drows, float* __restrict__ dweights,
                   const int* __restrict__ g_start, const int* __restrict__ g_len, const int* __restrict__ counts,
                   long long T, int D, int k, long long rows_cap, unsigned token_ctas, int* status) {
  grid_begin(rows, dout, pos, weights, g_start, g_len, counts);
  if (blockIdx.x >= token_ctas) {
    const int b = static_cast<int>(blockIdx.x - token_ctas);
    zero_padding(drows, g_start, g_len, counts, b / PAD_CTAS, b % PAD_CTAS, D, rows_cap, status);
    return;
  }
  const long long t = (static_cast<long long>(blockIdx.x) * ROW_THREADS + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  for (int j0 = 0; j0 < k; j0 += K) {
    int r[K];
    float w[K], dot[K];
    token_rows<K>(pos, t, k, j0, lane, rows_cap, 34, status, r);
#pragma unroll
    for (int j = 0; j < K; ++j) {
      w[j] = j0 + j < k ? weights[t * k + j0 + j] : 0.f;
      dot[j] = 0.f;
    }
#pragma unroll 1
    for (int i = lane; i < D / 8; i += 32) {
      const uint4 g = reinterpret_cast<const uint4*>(dout + t * D)[i];
      uint4 q[K];
#pragma unroll
      for (int j = 0; j < K; ++j)
        if (r[j] >= 0) q[j] = reinterpret_cast<const uint4*>(rows + static_cast<long long>(r[j]) * D)[i];
      const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&g);
#pragma unroll
      for (int j = 0; j < K; ++j) {
        if (r[j] < 0) continue;
        const __nv_bfloat162* qh = reinterpret_cast<const __nv_bfloat162*>(&q[j]);
        uint4 o;
        __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 gf = __bfloat1622float2(gh[c]);
          const float2 qf = __bfloat1622float2(qh[c]);
          dot[j] += gf.x * qf.x + gf.y * qf.y;
          oh[c] = __floats2bfloat162_rn(w[j] * gf.x, w[j] * gf.y);
        }
        reinterpret_cast<uint4*>(drows + static_cast<long long>(r[j]) * D)[i] = o;
      }
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const float d = warp_sum(dot[j]);
      if (lane == 0 && j0 + j < k) dweights[t * k + j0 + j] = d;
    }
  }
}

inline unsigned warps_grid(long long warps, int threads) {
  return static_cast<unsigned>((warps * 32 + threads - 1) / threads);
}

}  // namespace

#define PIPER_LAUNCH_OK() (cudaGetLastError() == cudaSuccess ? 0 : -3)

int moe_route(const void* logits, float* weights, int* idx, int* counts, long long T, int E, int k, int renorm,
              cudaStream_t st) {
  if (E > 32 * MAX_PER_LANE || k > MAX_K || k > E || k < 1) return -1;
  if (T == 0) return 0;
  auto kern = E <= 32 ? route_kernel<1> : E <= 64 ? route_kernel<2> : E <= 128 ? route_kernel<4> : route_kernel<8>;
  launch_overlapped(kern, warps_grid(T, ROW_THREADS), ROW_THREADS, 0, st, static_cast<const __nv_bfloat16*>(logits), weights, idx,
                                                           counts, T, E, k, renorm);
  return PIPER_LAUNCH_OK();
}

int moe_route_bwd(const void* logits, const int* idx, const float* weights, const float* dweights, void* dlogits,
                  long long T, int E, int k, int renorm, cudaStream_t st) {
  if (E > 32 * MAX_PER_LANE || k > MAX_K) return -1;
  if (T == 0) return 0;
  launch_overlapped(route_bwd_kernel, warps_grid(T, 256), 256, 0, st, static_cast<const __nv_bfloat16*>(logits), idx, weights,
                                                       dweights, static_cast<__nv_bfloat16*>(dlogits), T, E, k,
                                                       renorm);
  return PIPER_LAUNCH_OK();
}

int moe_group_table(const int* counts, int num_groups, int experts, const int* row_base, int* g_start, int* g_len,
                    int* total, int* cursor, int* copy, cudaStream_t st) {
  if (num_groups <= 0 || experts <= 0) return -1;
  launch_overlapped(group_table_kernel, 1, 32, 0, st, counts, num_groups, experts, row_base, g_start, g_len, total, cursor, copy);
  return PIPER_LAUNCH_OK();
}

int moe_permute(const void* x, const int* idx, const int* g_start, const int* g_len, const int* counts, int* cursor,
                int* pos, void* rows, long long T, int D, int E, int k, long long rows_cap, int* status,
                cudaStream_t st) {
  if (D % 8 != 0) return -1;
  const unsigned token_ctas = warps_grid(T, ROW_THREADS);
  launch_overlapped(permute_kernel, token_ctas + E * PAD_CTAS, ROW_THREADS, 0, st,
      static_cast<const __nv_bfloat16*>(x), idx, g_start, g_len, counts, cursor, pos, static_cast<__nv_bfloat16*>(rows),
      T, D, k, E, rows_cap, token_ctas, status);
  return PIPER_LAUNCH_OK();
}

// Entries per pass: all of them where k is 1, 2, 4 or 8, else passes of eight.
static int gather_sum(const void* rows, const int* pos, const float* weights, void* out, long long T, int D, int k,
                      long long rows_cap, int tag, int* status, cudaStream_t st) {
  if (D % 8 != 0) return -1;
  if (T == 0) return 0;
  auto kern = k == 1 ? gather_sum_kernel<1> : k == 2 ? gather_sum_kernel<2> : k <= 4 ? gather_sum_kernel<4>
                                                                                      : gather_sum_kernel<8>;
  launch_overlapped(kern, warps_grid(T, ROW_THREADS), ROW_THREADS, 0, st, static_cast<const __nv_bfloat16*>(rows), pos, weights,
                                                           static_cast<__nv_bfloat16*>(out), T, D, k, rows_cap, tag,
                                                           status);
  return PIPER_LAUNCH_OK();
}

int moe_permute_bwd(const void* drows, const int* pos, void* dx, long long T, int D, int k, long long rows_cap,
                    int* status, cudaStream_t st) {
  return gather_sum(drows, pos, nullptr, dx, T, D, k, rows_cap, 32, status, st);
}

int moe_combine(const void* rows, const int* pos, const float* weights, void* out, long long T, int D, int k,
                long long rows_cap, int* status, cudaStream_t st) {
  return gather_sum(rows, pos, weights, out, T, D, k, rows_cap, 33, status, st);
}

int moe_combine_bwd(const void* rows, const void* dout, const int* pos, const float* weights, void* drows,
                    float* dweights, const int* g_start, const int* g_len, const int* counts, int num_groups,
                    long long T, int D, int k, long long rows_cap, int* status, cudaStream_t st) {
  if (D % 8 != 0) return -1;
  const unsigned token_ctas = warps_grid(T, ROW_THREADS);
  if (token_ctas + num_groups == 0) return 0;
  auto kern = k == 1 ? combine_bwd_kernel<1> : k == 2 ? combine_bwd_kernel<2> : k <= 4 ? combine_bwd_kernel<4>
                                                                                        : combine_bwd_kernel<8>;
  launch_overlapped(kern, token_ctas + num_groups * PAD_CTAS, ROW_THREADS, 0, st,
      static_cast<const __nv_bfloat16*>(rows), static_cast<const __nv_bfloat16*>(dout), pos, weights,
      static_cast<__nv_bfloat16*>(drows), dweights, g_start, g_len, counts, T, D, k, rows_cap, token_ctas, status);
  return PIPER_LAUNCH_OK();
}

}  // namespace piper
