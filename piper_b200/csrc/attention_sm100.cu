// Causal grouped-query flash attention for sm_100a, forward and backward,
// on the packed projection qkv[T, (Hq + 2*Hkv) * hd] (T = B*S tokens, each
// sequence a multiple of 128 long).  All matrix products run on tcgen05 with
// accumulators in tensor memory; operands arrive by TMA (no multicast) in
// 128-byte-swizzled tiles, and the probability / score-gradient tiles the
// threads produce go back to tensor memory, from where they feed the next
// tcgen05.mma.
//
// Forward (attn_fwd_kernel): one CTA per two query tiles of 128 rows; online softmax, P and O in tensor memory.
//
// Backward (attn_bwd_kernel): S and dP are recomputed; threads form P = exp(S - lse) and dS = P (dP - delta) as bf16
// in tensor memory.  Two kinds of CTA in one launch:
//   dK/dV: stationary tile = 128 key rows of one kv head (K, V); streams 64-row Q/dO tiles of every query head in
//          the group, or of some where the group is split over several CTAs; accumulates dK = dS^T Q and dV = P^T dO.
//   dQ:    stationary tile = 128 query rows of one head (Q, dO); streams 128-row K and V blocks; dQ = dS K.
// No gradient is reduced with atomics, so they are reproducible.
//
// Every mbarrier wait is bounded (see ptx.cuh); on expiry a status code is
// recorded and the CTA unwinds and frees its TMEM.
#include "attention_sm100.h"

#include "ptx.cuh"

namespace piper {
namespace {

// Bounded wait on an mbarrier phase (see mbar_wait in ptx.cuh).
__device__ __forceinline__ bool await(uint64_t* bar, uint32_t parity, int* status) {
  return mbar_wait(bar, parity, status);
}

// The same for a whole warp, with one outcome for all its lanes: a lane that gave up while its neighbours saw
// the phase complete must not leave them alone at the next warp-wide synchronisation.
__device__ __forceinline__ bool await_all(uint64_t* bar, uint32_t parity, int* status) {
  return __all_sync(0xffffffffu, await(bar, parity, status));
}

// One arrival per warp: the lanes converge first, so whatever each of them wrote (and fenced) before the call
// is ordered before the arrival that lane 0 performs for all of them.  256 threads arriving one by one on the
// same barrier word would serialise in the shared-memory atomic unit several times per tile.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Writes 32 consecutive bf16 values (given as 16 packed words) of row `row`,
// starting at 16-byte chunk index `chunk0` (multiple of 4) of a 128-byte
// swizzled row.  `tile` is the 1024-byte-aligned base of a [rows][128 B] tile.
__device__ __forceinline__ void store_row_chunk_sw128(uint8_t* tile, int row, int chunk0,
                                                      const uint32_t (&w)[16]) {
  uint8_t* rbase = tile + row * 128;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int phys = (chunk0 + q) ^ (row & 7);
    *reinterpret_cast<uint4*>(rbase + phys * 16) =
        make_uint4(w[4 * q + 0], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  }
}

// ================================================================= forward
// Bound by the tensor cores and the exponential unit alike: a 128x128 score tile of head dimension 128 costs 1,024
// cycles of MMA and 1,024 cycles of ex2 (16 per cycle and SM).  A CTA therefore works on two query tiles (A, B) that
// share one K/V stream: while four softmax warps turn the scores of one tile into probabilities, the MMAs of the
// other tile run.  The probabilities go back to the tensor memory columns of their scores and feed P V from there, so
// no thread writes shared memory in the loop; the output accumulates in tensor memory and is rescaled in every block in
// which a row maximum of the warp has grown.  (Letting the maximum go stale until it has grown by 2^8 saves 8-15 % of
// the time, but the largest probability of a row is then rounded to bf16 where it is exactly 1 otherwise: error against
// 64 bits 2.05e-3 -> 2.09e-3 at S = 4096.)
// Where there are too few tiles for pairs, a CTA works on one, and its even and odd key blocks take the places of two tiles,
// each with its own maxima, sums and output in tensor memory, merged at the end: a block alone is a serial chain of scores,
// softmax and P V, 1.3 us long at head dimension 64.  us with one chain and with two: 1 x 2048, 4 heads x 64 24.0 and 16.7, 1 x 4096, 8
// heads x 64 45.8 and 31.7, 1 x 8192, 4 heads x 128 107.5 and 63.4, 1 x 512, 32 heads x 128 10.4 and 8.9.
// Tiles of one kv head are numbered query block major, so a pair is two heads of the group on the same rows where
// the group is even, and neighbouring query blocks otherwise.
// S = 4096, 32 q / 8 kv heads x 128: 237 us with one CTA per 128 query rows and probabilities through shared memory,
// 127 us so; S = 8192, 32 / 8 x 64: 745 and 421 us.
//
// Warps 0-3: softmax of tile A, 4-7: of tile B (one query row per thread, row == TMEM lane); 8: TMA; 9: MMA.
constexpr int FWD_THREADS = 320;

template <int HD>
struct FwdSmem {
  static constexpr int HALVES = HD / 64;
  static constexpr int TILE = 128 * HD * 2;     // Q, K or V tile
  static constexpr int STAGES = 5;              // K0, V0, K1, V1, ... through one ring
  static constexpr int Q_OFF = 0;               // 2 tiles; each takes its output tile at the end
  static constexpr int KV_OFF = 2 * TILE;
  static constexpr int BAR_OFF = KV_OFF + STAGES * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

struct FwdBars {
  uint64_t q_full;
  uint64_t kv_full[5], kv_empty[5];
  uint64_t s_full[2];          // scores of tile t are in tensor memory
  uint64_t p_full[2][2];       // first / second 64 key columns of its probabilities are
  uint64_t o_done[2];          // P V of the tile's last block has been accumulated
  uint32_t tmem_base;
};

// ONE: one tile per CTA, else tiles_per_cta, two.  A constant for the one case only: the loops of two tiles lose 0.6 % both to
// the other case's decisions and with their own number as a constant (1 x 8192, 32 / 4 heads x 128, 523.5 and 526.6 us).
template <int HD, bool ONE>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap tmap_out,
                float* __restrict__ lse, int S, int Hq, int Hkv, int B, int tiles_per_cta, float scale_log2,
                int* status) {
  using L = FwdSmem<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  FwdBars* bars = reinterpret_cast<FwdBars*>(smem + L::BAR_OFF);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  // longest rows first over all heads: the kv head and the sequence vary fastest, the query blocks fall
  const int group = Hq / Hkv;
  const int tiles = group * (S / 128);
  const int pairs = (tiles + tiles_per_cta - 1) / tiles_per_cta;
  const int gb = static_cast<int>(blockIdx.x) % (Hkv * B);
  const int pair = pairs - 1 - static_cast<int>(blockIdx.x) / (Hkv * B);
  const int g = gb % Hkv;
  const int b = gb / Hkv;
  const int t0 = pair * tiles_per_cta;
  const bool two = !ONE && tiles_per_cta == 2 && t0 + 1 < tiles;
  const int qblk0 = t0 / group, head0 = g * group + t0 % group;
  const int qblk1 = (t0 + 1) / group, head1 = g * group + (t0 + 1) % group;
  // one tile: its even key blocks take the place of tile A, the odd ones that of tile B, and the two are merged at the end
  const bool halves = ONE && qblk0 > 0;
  const int n0 = halves ? (qblk0 + 2) / 2 : qblk0 + 1;
  const int n1 = two ? qblk1 + 1 : halves ? (qblk0 + 1) / 2 : 0;     // n1 >= n0 where there are two tiles
  const int n_blocks = two ? n1 : qblk0 + 1;
  const long long tok0 = static_cast<long long>(b) * S;

  if (threadIdx.x == 0) {
    mbar_init(&bars->q_full, 1);
    for (int i = 0; i < L::STAGES; ++i) {
      mbar_init(&bars->kv_full[i], 1);
      mbar_init(&bars->kv_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_full[i][0], 4);        // one arrival per softmax warp
      mbar_init(&bars->p_full[i][1], 4);
      mbar_init(&bars->o_done[i], 1);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmap);
    tma_prefetch_desc(&tmap_out);
  }
  if (warp == 9) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  grid_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  // columns: [0,128) S/P of tile A  [128,256) of tile B  [256,256+HD) O of tile A  [384,384+HD) of tile B

  if (warp == 8) {
    // ------------------------------------------------------------- TMA
    if (lane == 0) {
      mbar_arrive_expect_tx(&bars->q_full, (two ? 2 : 1) * L::TILE);
      for (int t = 0; t < (two ? 2 : 1); ++t)
        for (int h = 0; h < L::HALVES; ++h)
          tma_load_2d(smem + L::Q_OFF + t * L::TILE + h * 16384, &tmap, &bars->q_full,
                      (t ? head1 : head0) * HD + 64 * h, static_cast<int>(tok0) + (t ? qblk1 : qblk0) * 128);
      int it = 0, s = 0;
      uint32_t ph = 1;
      for (; it < 2 * n_blocks; ++it) {         // even: K of block it / 2, odd: V
        if (!await(&bars->kv_empty[s], ph, status)) break;
        mbar_arrive_expect_tx(&bars->kv_full[s], L::TILE);
        const int col = (Hq + ((it & 1) ? Hkv : 0) + g) * HD;
        for (int h = 0; h < L::HALVES; ++h)
          tma_load_2d(smem + L::KV_OFF + s * L::TILE + h * 16384, &tmap, &bars->kv_full[s], col + 64 * h,
                      static_cast<int>(tok0) + (it >> 1) * 128);
        if (++s == L::STAGES) { s = 0; ph ^= 1; }
      }
      grid_launch();
      if (it < 2 * n_blocks) {
        // Unwinding after a failed wait: let the copies already issued land
        // before the CTA and its shared memory go away.
        await(&bars->q_full, 0, nullptr);
        for (int jj = it - 1; jj >= 0 && jj >= it - L::STAGES; --jj)
          await(&bars->kv_full[jj % L::STAGES], (jj / L::STAGES) & 1, nullptr);
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------- MMA
    // The whole warp walks the loop with uniform values and one elected lane issues: in a divergent single-lane
    // branch every descriptor has to be moved into uniform registers for each MMA.
    constexpr uint32_t idesc_qk = umma_idesc_bf16(128, 128, false, false);
    constexpr uint32_t idesc_pv = umma_idesc_bf16(128, HD, false, true);
    const uint64_t dq0 = umma_desc_sw128(smem_u32(smem + L::Q_OFF), 16, 1024);
    const uint64_t dk_base = umma_desc_sw128(smem_u32(smem + L::KV_OFF), 16, 1024);
    const uint64_t dv_base = umma_desc_sw128(smem_u32(smem + L::KV_OFF), 16384, 1024);

    auto issue_s = [&](int t, int st) {
      const uint64_t dq = dq0 + (halves ? 0 : t * L::TILE >> 4);
      const uint64_t dk = dk_base + (st * L::TILE >> 4);
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks) {
        const uint32_t off = ((ks / 4) * 16384 + (ks % 4) * 32) >> 4;
        umma_bf16_ss(tmem_base + t * 128, dq + off, dk + off, idesc_qk, ks > 0 ? 1u : 0u);
      }
      umma_commit(&bars->s_full[t]);
    };
    auto issue_pv = [&](int t, int st, int half, bool first) {
      const uint64_t dv = dv_base + (st * L::TILE >> 4);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int ks = half * 4 + k;
        umma_bf16_ts(tmem_base + 256 + t * 128, tmem_base + t * 128 + ks * 8, dv + (ks * 2048 >> 4), idesc_pv,
                     (first && ks == 0) ? 0u : 1u);
      }
    };
    bool ok = await_all(&bars->q_full, 0, status);
    ok = ok && await_all(&bars->kv_full[0], 0, status);
    if (ok) {
      tc_fence_after();
      if (elect_one()) {
        issue_s(0, 0);
        if (two) issue_s(1, 0);
        umma_commit(&bars->kv_empty[0]);
      }
      __syncwarp();
    }
    if (halves) {
      // block b belongs to half b % 2; its K is entry 2b of the ring, its V entry 2b + 1
      auto entry = [&](int e) { return await_all(&bars->kv_full[e % L::STAGES], (e / L::STAGES) & 1, status); };
      auto scores = [&](int b) -> bool {
        if (!entry(2 * b)) return false;
        tc_fence_after();
        if (elect_one()) {
          issue_s(b & 1, 2 * b % L::STAGES);
          umma_commit(&bars->kv_empty[2 * b % L::STAGES]);
        }
        __syncwarp();
        return true;
      };
      ok = ok && scores(1);
      for (int b = 0; b < n_blocks && ok; ++b) {
        const int t = b & 1, v_st = (2 * b + 1) % L::STAGES;
        const uint32_t p_ph = (b >> 1) & 1;
        ok = entry(2 * b + 1) && await_all(&bars->p_full[t][0], p_ph, status);
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) issue_pv(t, v_st, 0, b < 2);
        __syncwarp();
        if (!(ok = await_all(&bars->p_full[t][1], p_ph, status))) break;
        tc_fence_after();
        if (elect_one()) {
          issue_pv(t, v_st, 1, false);
          if (b + 2 >= n_blocks) umma_commit(&bars->o_done[t]);
          umma_commit(&bars->kv_empty[v_st]);
        }
        __syncwarp();
        if (b + 2 < n_blocks) ok = scores(b + 2);
      }
    }
    int st = 1;                    // ring slot of V of block j; K of block j + 1 follows it
    uint32_t ph = 0;
    for (int j = 0; j < n_blocks && ok && (!ONE || !halves); ++j) {
      const int v_st = st;
      const uint32_t v_ph = ph;
      if (++st == L::STAGES) { st = 0; ph ^= 1; }
      const int k_st = st;
      const uint32_t k_ph = ph;
      if (++st == L::STAGES) { st = 0; ph ^= 1; }
      const bool more = j + 1 < n_blocks;
      ok = await_all(&bars->kv_full[v_st], v_ph, status);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int nt = t ? n1 : n0;
        if (!ok || j >= nt) continue;
        const bool last_user = t == 1 || !two;
        ok = await_all(&bars->p_full[t][0], j & 1, status);
        if (!ok) continue;
        tc_fence_after();
        if (elect_one()) issue_pv(t, v_st, 0, j == 0);
        __syncwarp();
        ok = await_all(&bars->p_full[t][1], j & 1, status);
        if (!ok) continue;
        tc_fence_after();
        if (elect_one()) {
          issue_pv(t, v_st, 1, false);
          if (j == nt - 1) umma_commit(&bars->o_done[t]);
          if (last_user) umma_commit(&bars->kv_empty[v_st]);
        }
        __syncwarp();
        if (j + 1 < nt) {
          // the scores of the next block replace the probabilities just consumed: MMAs execute in issue order
          ok = await_all(&bars->kv_full[k_st], k_ph, status);
          if (!ok) continue;
          tc_fence_after();
          if (elect_one()) {
            issue_s(t, k_st);
            if (last_user) umma_commit(&bars->kv_empty[k_st]);
          }
          __syncwarp();
        }
      }
      if (!more) break;
    }
  } else if (warp < 4 || two || halves) {
    // --------------------------------------------------- softmax + output
    const int t = warp >> 2;
    const int n_t = t ? n1 : n0;
    const int qblk = t && !halves ? qblk1 : qblk0;
    const int head = t && !halves ? head1 : head0;
    const int row = (warp & 3) * 32 + lane;      // query row == TMEM lane
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t ts = tmem_base + lane_sel + t * 128;
    const uint32_t to = tmem_base + lane_sel + 256 + t * 128;
    float m_run = -INFINITY;
    float l_run = 0.f;
    bool ok = true;
    for (int j = 0; j < n_t; ++j) {
      if (!await_all(&bars->s_full[t], j & 1, status)) { ok = false; break; }
      tc_fence_after();
      uint32_t sv[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32(ts + c * 32, sv[c]);
      tmem_ld_wait();
      if ((halves ? 2 * j + t : j) == qblk) {
        // causal mask, applied once to the registers of the only tile that needs it: a score of -inf then
        // drops out of the maximum and turns into a probability of exactly zero below
#pragma unroll
        for (int i = 0; i < 128; ++i)
          if (i > row) sv[i / 32][i % 32] = 0xff800000u;
      }
      float mx[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx[c] = __uint_as_float(sv[c][0]);
#pragma unroll
        for (int i = 1; i < 31; i += 2)
          mx[c] = fmaxf(mx[c], fmaxf(__uint_as_float(sv[c][i]), __uint_as_float(sv[c][i + 1])));
        mx[c] = fmaxf(mx[c], __uint_as_float(sv[c][31]));
      }
      const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
      float alpha = 1.f;
      bool grown = false;
      if (j == 0) {
        m_run = m_blk;
      } else if ((grown = __any_sync(0xffffffffu, m_blk > m_run))) {
        const float m_new = fmaxf(m_run, m_blk);
        alpha = fast_exp2((m_run - m_new) * scale_log2);
        l_run *= alpha;
        m_run = m_new;
      }
      const float2 sl2 = make_float2(scale_log2, scale_log2);
      const float msc = m_run * scale_log2;
      const float2 nm2 = make_float2(-msc, -msc);
      float2 rs[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 p = fma2(make_float2(__uint_as_float(sv[c][2 * i]), __uint_as_float(sv[c][2 * i + 1])), sl2, nm2);
          p.x = fast_exp2(p.x);
          p.y = fast_exp2(p.y);
          rs[i & 1] = add2(rs[i & 1], p);
          w[i] = pack_bf16x2(p.x, p.y);
        }
        tmem_st_32x16(ts + c * 16, w);
        if (c == 1 && grown) {
          // Here rather than before the exponentials: half of the scores' registers are free for the loads, and the
          // first half of the probabilities waits for it in any case.  P V of block j - 1 is complete: the commit
          // behind s_full of block j came after it.
#pragma unroll 1
          for (int h = 0; h < HD / 64; ++h) {
            uint32_t r[2][32];
            tmem_ld_32x32(to + h * 64, r[0]);
            tmem_ld_32x32(to + h * 64 + 32, r[1]);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 64; ++i) r[i / 32][i % 32] = __float_as_uint(__uint_as_float(r[i / 32][i % 32]) * alpha);
            tmem_st_32x32(to + h * 64, r[0]);
            tmem_st_32x32(to + h * 64 + 32, r[1]);
          }
        }
        if (c & 1) {
          tmem_st_wait();
          tc_fence_before();
          warp_arrive(&bars->p_full[t][c >> 1], lane);
        }
      }
      l_run += (rs[0].x + rs[0].y) + (rs[1].x + rs[1].y);
    }
    float wa = 1.f, wb = 0.f;                    // weights of the two halves' sums; the first half's warps write the tile
    if (halves) {
      // maxima and sums of the second half, through the buffer of the second query tile
      float2* other = reinterpret_cast<float2*>(smem + L::Q_OFF + L::TILE);
      if (t == 1) other[row] = make_float2(m_run, l_run);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (t == 0) {
        const float2 o = other[row];
        const float m = fmaxf(m_run, o.x);
        wa = fast_exp2((m_run - m) * scale_log2);
        wb = fast_exp2((o.x - m) * scale_log2);
        l_run = l_run * wa + o.y * wb;
        m_run = m;
        ok = ok && await_all(&bars->o_done[1], 0, status);
      }
    }
    if ((!ONE || !(halves && t == 1)) && ok && await_all(&bars->o_done[t], 0, status)) {
      // the tile's Q operand has been read for the last time; its buffer takes the output, 32 rows per warp
      tc_fence_after();
      const float inv = 1.f / l_run;
      const float2 fa = make_float2(wa * inv, wa * inv), fb = make_float2(wb * inv, wb * inv);
      uint8_t* obuf = smem + L::Q_OFF + t * L::TILE;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t r[32], r2[32], w[16];
        tmem_ld_32x32(to + c * 32, r);
        if (halves) tmem_ld_32x32(to + 128 + c * 32, r2);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (!ONE) {
            w[i] = pack_bf16x2(__uint_as_float(r[2 * i]) * inv, __uint_as_float(r[2 * i + 1]) * inv);
            continue;
          }
          float2 v = mul2(make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), fa);
          if (halves) v = fma2(make_float2(__uint_as_float(r2[2 * i]), __uint_as_float(r2[2 * i + 1])), fb, v);
          w[i] = pack_bf16x2(v.x, v.y);
        }
        store_row_chunk_sw128(obuf + (c >> 1) * 16384, row, (c & 1) * 4, w);
      }
      lse[(static_cast<long long>(b) * Hq + head) * S + qblk * 128 + row] =
          m_run * (scale_log2 * 0.6931471805599453f) + logf(l_run);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        for (int h = 0; h < L::HALVES; ++h)
          tma_store_2d_bulk(&tmap_out, obuf + h * 16384 + (warp & 3) * 32 * 128, head * HD + 64 * h,
                            static_cast<int>(tok0) + qblk * 128 + (warp & 3) * 32);
        bulk_commit_group();
        bulk_wait_group<0>();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ================================================================ backward
// delta[b, h, s] = sum_d dO[t, h, d] * O[t, h, d]; HD/8 lanes per (t, h), one 16-byte vector of each per lane.
template <int HD>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                  float* __restrict__ delta, int* __restrict__ arrived, int n_arrived, long long T, int S, int Hq) {
  grid_begin(o, d_o);
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n_arrived; i += gridDim.x * 256) arrived[i] = 0;
  constexpr int LANES = HD / 8;
  const int wl = threadIdx.x & 31;
  const int lane = wl & (LANES - 1);
  const unsigned mask = ((1u << LANES) - 1u) << (wl & ~(LANES - 1));
  const unsigned total = static_cast<unsigned>(T * Hq);   // the launcher keeps T * Hq below 2^31
  const unsigned stride = gridDim.x * (256 / LANES);
  for (unsigned gi = blockIdx.x * (256 / LANES) + threadIdx.x / LANES; gi < total; gi += stride) {
    const uint4 a = *reinterpret_cast<const uint4*>(o + static_cast<long long>(gi) * HD + 8 * lane);
    const uint4 b = *reinterpret_cast<const uint4*>(d_o + static_cast<long long>(gi) * HD + 8 * lane);
    const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&a);
    const __nv_bfloat162* bp = reinterpret_cast<const __nv_bfloat162*>(&b);
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = __bfloat1622float2(ap[i]), y = __bfloat1622float2(bp[i]);
      s += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) s += __shfl_xor_sync(mask, s, off);
    const unsigned t = gi / static_cast<unsigned>(Hq), h = gi - t * Hq;
    const unsigned bi = t / static_cast<unsigned>(S), si = t - bi * S;
    if (lane == 0) delta[(static_cast<long long>(bi) * Hq + h) * S + si] = s;
  }
}

// The dK/dV pass streams 64-row tiles through two tensor memory stages (dK, dV and two 64-wide pairs of S' and dP' fill
// it).  Warps 0-7 turn the even tiles' scores into probabilities and score gradients, warps 8-15 the odd tiles' (four warps
// per 32 columns), so each group has the MMAs of two tiles' time for its work; warp 16: TMA, warp 17: MMA.  P' and dS' (bf16) replace their
// own fp32 scores in tensor memory and are the A operand of the accumulating MMAs from there: no thread writes shared
// memory in the loop.  Bound by the MMAs: a 128x64x16 one with both operands in shared memory reads 6 KiB (48 cycles)
// for 32 cycles of arithmetic.  Both passes and the delta kernel at S = 4096, 32 q / 8 kv heads x 128: 653 us with
// probabilities through shared memory in two launches, 391 us so (this kernel alone 379 us, and 427 us with dQ on
// 64-row tiles as well).  With eight softmax warps instead of sixteen: 376 and 374 us, 3 x 1408, 32 / 8 x 64 142 and 138 us.
// The scores come out of tensor memory as fragments, not as rows: lse and delta belong to the columns here, and with a row
// per lane every lane reads all 32 pairs of its columns, 1,784 shared-memory wavefronts per 128 x 128 scores beside the 1,024
// (head dimension 64) that the MMAs read their operands in.  A fragment has 4 rows x 8 columns per thread: a quarter of them.
// This kernel at 3 x 1408, 32 / 8 x 64: 139 us by rows, 128 us so; 1 x 4096, 32 / 8 x 128, which is short of power: 382 and 375 us.
constexpr int BWD_THREADS = 576;
constexpr int BWD_TMA_WARP = 16, BWD_MMA_WARP = 17;

template <int HD>
struct BwdSmem {
  static constexpr int HALVES = HD / 64;
  static constexpr int X_TILE = 128 * HD * 2;      // stationary tile; takes a gradient tile at the end
  static constexpr int Y_TILE = 64 * HD * 2;       // streamed tile
  static constexpr int Y_HALF = 64 * 128;          // one 64x64 box
  static constexpr int X1_OFF = 0;
  static constexpr int X2_OFF = X_TILE;
  static constexpr int Y_STAGES = 4;
  static constexpr int Y_OFF = 2 * X_TILE;         // Y_STAGES x (Y1, Y2)
  static constexpr int VEC_OFF = Y_OFF + Y_STAGES * 2 * Y_TILE;   // Y_STAGES x (lse[64], delta[64]) floats
  static constexpr int VEC_BYTES = 64 * 4;
  static constexpr int BAR_OFF = VEC_OFF + Y_STAGES * 2 * VEC_BYTES;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

struct BwdBars {
  uint64_t x_full;
  uint64_t y_full[4], y_empty[4];     // streamed tiles (BwdSmem::Y_STAGES)
  uint64_t s_full[2], dp_full[2];     // S' and dP' of a stage are in tensor memory
  uint64_t p_full[2];                 // P' stands in the place of S'
  uint64_t ds_full[2];                // dS' stands in the place of dP'
  uint64_t acc_full;
  uint32_t tmem_base;
  int last;                           // this CTA has to add the parts
};

// dK and dV of key block xb of kv head g.  The query heads of the group may be split over `parts` CTAs; each accumulates over
// its own and leaves its sums in `partial` ([part][slice of 64 columns][column][row]), and the one that finishes last
// (by `arrived`, no CTA waits) adds them in the order of the parts, so the gradients are reproducible.
template <int HD>
__device__ __forceinline__ void attn_dkv_cta(const CUtensorMap* tmap_qkv_x, const CUtensorMap* tmap_qkv_y,
                                             const CUtensorMap* tmap_do_y, const CUtensorMap* tmap_dqkv,
                                             const float* __restrict__ lse, const float* __restrict__ delta, int xb,
                                             int g, int b, int part, int parts, float* __restrict__ partial,
                                             int* __restrict__ arrived, int S, int Hq, int Hkv, float scale,
                                             float scale_log2, int* status) {
  using L = BwdSmem<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  BwdBars* bars = reinterpret_cast<BwdBars*>(smem + L::BAR_OFF);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int heads = Hq / Hkv / parts;          // query heads of this CTA
  const int head0 = g * (Hq / Hkv) + part * heads;
  const int tok0 = b * S;

  // for each of its query heads streams q tiles i in [2*xb, S/64 - 1]
  const int tiles_per_head = S / 64 - 2 * xb;
  const int n_iter = tiles_per_head * heads;

  if (threadIdx.x == 0) {
    mbar_init(&bars->x_full, 1);
    for (int i = 0; i < L::Y_STAGES; ++i) {
      mbar_init(&bars->y_full[i], 1);
      mbar_init(&bars->y_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->dp_full[i], 1);
      mbar_init(&bars->p_full[i], 8);         // one arrival per softmax warp of the stage
      mbar_init(&bars->ds_full[i], 8);
    }
    mbar_init(&bars->acc_full, 1);
    fence_mbar_init();
    tma_prefetch_desc(tmap_qkv_x);
    tma_prefetch_desc(tmap_qkv_y);
    tma_prefetch_desc(tmap_do_y);
    tma_prefetch_desc(tmap_dqkv);
  }
  if (warp == BWD_MMA_WARP) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  grid_wait(lse, delta);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  // columns: [0,64) S'0  [64,128) S'1  [128,192) dP'0  [192,256) dP'1
  //          [256,256+HD) acc1   [384,384+HD) acc2
  const uint32_t tmem_acc1 = tmem_base + 256;
  const uint32_t tmem_acc2 = tmem_base + 384;
  bool done = false;                           // (softmax warps) the gradients are complete

  if (warp == BWD_TMA_WARP) {
    // ------------------------------------------------------------- TMA
    if (lane == 0) {
      const int xrow = tok0 + xb * 128;
      mbar_arrive_expect_tx(&bars->x_full, 2 * L::X_TILE);
      for (int h = 0; h < L::HALVES; ++h) {
        tma_load_2d(smem + L::X1_OFF + h * 16384, tmap_qkv_x, &bars->x_full, (Hq + g) * HD + 64 * h, xrow);
        tma_load_2d(smem + L::X2_OFF + h * 16384, tmap_qkv_x, &bars->x_full, (Hq + Hkv + g) * HD + 64 * h, xrow);
      }
      int it = 0;
      int hh = head0, ti = 2 * xb;           // query head and tile of iteration it
      for (; it < n_iter; ++it) {
        const int st = it % L::Y_STAGES;
        if (!await(&bars->y_empty[st], ((it / L::Y_STAGES) & 1) ^ 1, status)) break;
        const int yrow = tok0 + ti * 64;
        uint8_t* yb = smem + L::Y_OFF + st * 2 * L::Y_TILE;
        mbar_arrive_expect_tx(&bars->y_full[st], 2 * L::Y_TILE + 2 * L::VEC_BYTES);
        for (int h = 0; h < L::HALVES; ++h) {
          uint8_t* y1 = yb + h * L::Y_HALF;
          uint8_t* y2 = y1 + L::Y_TILE;
          tma_load_2d(y1, tmap_qkv_y, &bars->y_full[st], hh * HD + 64 * h, yrow);
          tma_load_2d(y2, tmap_do_y, &bars->y_full[st], hh * HD + 64 * h, yrow);
        }
        const long long idx = (static_cast<long long>(b) * Hq + hh) * S + ti * 64;
        uint8_t* v = smem + L::VEC_OFF + st * 2 * L::VEC_BYTES;
        bulk_load(v, lse + idx, L::VEC_BYTES, &bars->y_full[st]);
        bulk_load(v + L::VEC_BYTES, delta + idx, L::VEC_BYTES, &bars->y_full[st]);
        if (++ti == S / 64) { ti = 2 * xb; ++hh; }
      }
      grid_launch();
      if (it < n_iter) {
        // Unwinding: wait (bounded) for the copies in flight.
        await(&bars->x_full, 0, nullptr);
        for (int jj = it - 1; jj >= 0 && jj > it - 1 - L::Y_STAGES; --jj)
          await(&bars->y_full[jj % L::Y_STAGES], (jj / L::Y_STAGES) & 1, nullptr);
      }
    }
  } else if (warp == BWD_MMA_WARP) {
    // ------------------------------------------------------------- MMA
    // Uniform control flow with one elected issuing lane (see the forward kernel).  Order per tile i: P' Y2 of i,
    // S' of i + 2 into the columns just consumed, dS' Y1 of i, dP' of i + 2.  MMAs execute in issue order.
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64, false, false);
    constexpr uint32_t idesc_acc = umma_idesc_bf16(128, HD, false, true);
    const uint64_t dx1 = umma_desc_sw128(smem_u32(smem + L::X1_OFF), 16, 1024);
    const uint64_t dx2 = umma_desc_sw128(smem_u32(smem + L::X2_OFF), 16, 1024);
    const uint64_t dyk = umma_desc_sw128(smem_u32(smem + L::Y_OFF), 16, 1024);            // K-major view of a stage
    const uint64_t dyn = umma_desc_sw128(smem_u32(smem + L::Y_OFF), L::Y_HALF, 1024);     // MN-major view
    auto issue_scores = [&](uint32_t tmem_d, uint64_t dx, uint64_t dy) {
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks)
        umma_bf16_ss(tmem_d, dx + (((ks / 4) * 16384 + (ks % 4) * 32) >> 4),
                     dy + (((ks / 4) * L::Y_HALF + (ks % 4) * 32) >> 4), idesc_s, ks > 0 ? 1u : 0u);
    };
    auto issue_acc = [&](uint32_t tmem_d, uint32_t tmem_a, uint64_t dy, bool first) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks)       // contraction over the 64 streamed rows
        umma_bf16_ts(tmem_d, tmem_a + (ks / 2) * 32 + (ks % 2) * 8, dy + (ks * 2048 >> 4), idesc_acc,
                     (first && ks == 0) ? 0u : 1u);
    };
    bool ok = await_all(&bars->x_full, 0, status);
    for (int i = 0; i < 2 && i < n_iter && ok; ++i) {
      ok = await_all(&bars->y_full[i], 0, status);
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t y = dyk + (i * 2 * L::Y_TILE >> 4);
        issue_scores(tmem_base + i * 64, dx1, y);
        umma_commit(&bars->s_full[i]);
        issue_scores(tmem_base + 128 + i * 64, dx2, y + (L::Y_TILE >> 4));
        umma_commit(&bars->dp_full[i]);
      }
      __syncwarp();
    }
    for (int i = 0; i < n_iter && ok; ++i) {
      const int ss = i & 1;
      const uint32_t ph = (i >> 1) & 1;
      const int st = i % L::Y_STAGES;
      const int st2 = (i + 2) % L::Y_STAGES;
      const bool more = i + 2 < n_iter;
      const uint64_t yn = dyn + (st * 2 * L::Y_TILE >> 4);
      const uint64_t yk2 = dyk + (st2 * 2 * L::Y_TILE >> 4);
      if (!(ok = await_all(&bars->p_full[ss], ph, status))) break;
      tc_fence_after();
      if (elect_one()) issue_acc(tmem_acc2, tmem_base + ss * 64, yn + (L::Y_TILE >> 4), i == 0);
      __syncwarp();
      if (more) {
        if (!(ok = await_all(&bars->y_full[st2], ((i + 2) / L::Y_STAGES) & 1, status))) break;
        tc_fence_after();
        if (elect_one()) {
          issue_scores(tmem_base + ss * 64, dx1, yk2);
          umma_commit(&bars->s_full[ss]);
        }
        __syncwarp();
      }
      if (!(ok = await_all(&bars->ds_full[ss], ph, status))) break;
      tc_fence_after();
      if (elect_one()) {
        issue_acc(tmem_acc1, tmem_base + 128 + ss * 64, yn, i == 0);
        umma_commit(&bars->y_empty[st]);
        if (more) {
          issue_scores(tmem_base + 128 + ss * 64, dx2, yk2 + (L::Y_TILE >> 4));
          umma_commit(&bars->dp_full[ss]);
        }
        if (i == n_iter - 1) umma_commit(&bars->acc_full);
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------- P' / dS' tiles + epilogue
    const int wg = warp >> 3;                  // tiles wg, wg + 2, ...; tensor memory stage wg
    const int ch = (warp >> 2) & 1;            // columns [32 ch, 32 ch + 32) of every tile
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t ts = tmem_base + lane_sel + wg * 64 + ch * 32;
    const uint32_t td = ts + 128;
    // Fragment layout (tmem_ld_16x256b_x4): this thread has columns 8c + c0 + {0, 1} of rows 16 h + 8 j + lane / 4 of its
    // warp's 32 x 32 block, c < 4, h, j < 2.
    constexpr uint32_t kUpper = 16u << 16;     // upper 16 lanes of the warp's window
    const int c0 = 2 * (lane & 3);
    const int xpos = xb * 128 + (warp & 3) * 32 + (lane >> 2);   // position of the thread's first row in the sequence
    const float2 sl2 = make_float2(scale_log2, scale_log2);
    constexpr float kNegLog2e = -1.4426950408889634f;
    const float2 neg_one = make_float2(-1.f, -1.f);
    int ti = 2 * xb + wg;   // tiles_per_head is even: the parity of ti is wg throughout
    bool ok = true;
    for (int it = wg; it < n_iter; it += 2) {
      const uint32_t ph = (it >> 1) & 1;
      const int st = it % L::Y_STAGES;
      const float* vl = reinterpret_cast<const float*>(smem + L::VEC_OFF + st * 2 * L::VEC_BYTES) + ch * 32 + c0;
      const float* vd = vl + L::VEC_BYTES / 4;
      if (!await_all(&bars->y_full[st], (it / L::Y_STAGES) & 1, status)) { ok = false; break; }
      float2 nl[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 l2 = *reinterpret_cast<const float2*>(vl + 8 * c);
        nl[c] = make_float2(l2.x * kNegLog2e, l2.y * kNegLog2e);
      }
      if (!await_all(&bars->s_full[wg], ph, status)) { ok = false; break; }
      tc_fence_after();
      uint32_t sv[2][16], w[8];
      tmem_ld_16x256b_x4(ts, sv[0]);
      tmem_ld_16x256b_x4(ts + kUpper, sv[1]);
      tmem_ld_wait();
      // Causal mask, applied once to the registers of the tiles that cross the diagonal (element (x row, y col) is
      // kept iff key <= query): a score of -inf turns into a probability and a score gradient of exactly zero.
      const int ypos0 = ti * 64 + ch * 32;
      if (ypos0 < xb * 128 + 127) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (xpos + 16 * h + 8 * ((i >> 1) & 1) > ypos0 + 8 * (i >> 2) + c0 + (i & 1)) sv[h][i] = 0xff800000u;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {          // word i: columns of c = i / 2, row half i % 2
          uint32_t* v = &sv[h][2 * i];
          float2 p = fma2(make_float2(__uint_as_float(v[0]), __uint_as_float(v[1])), sl2, nl[i >> 1]);
          p.x = fast_exp2(p.x);
          p.y = fast_exp2(p.y);
          v[0] = __float_as_uint(p.x);
          v[1] = __float_as_uint(p.y);
          w[i] = pack_bf16x2(p.x, p.y);
        }
        tmem_st_16x128b_x4(ts + h * kUpper, w);   // over columns this warp has already read
      }
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&bars->p_full[wg], lane);
      float2 dl[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) dl[c] = *reinterpret_cast<const float2*>(vd + 8 * c);
      if (!await_all(&bars->dp_full[wg], ph, status)) { ok = false; break; }
      tc_fence_after();
      uint32_t dv[2][16];
      tmem_ld_16x256b_x4(td, dv[0]);
      tmem_ld_16x256b_x4(td + kUpper, dv[1]);
      tmem_ld_wait();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint32_t* v = &dv[h][2 * i];
          const uint32_t* p = &sv[h][2 * i];
          float2 d = fma2(dl[i >> 1], neg_one, make_float2(__uint_as_float(v[0]), __uint_as_float(v[1])));
          d = mul2(d, make_float2(__uint_as_float(p[0]), __uint_as_float(p[1])));
          w[i] = pack_bf16x2(d.x, d.y);
        }
        tmem_st_16x128b_x4(td + h * kUpper, w);
      }
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&bars->ds_full[wg], lane);
      ti += 2;
      if (ti >= S / 64) ti = 2 * xb + wg;
    }
    done = ok && await_all(&bars->acc_full, 0, status);
  }

  // The gradients leave in slices of 64 columns, of dK first, of dV behind them, four warps per slice.
  constexpr int SLICES = 2 * L::HALVES;
  const int slice = warp >> 2, row = (warp & 3) * 32 + lane;
  const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t ta = (slice < L::HALVES ? tmem_acc1 : tmem_acc2 - L::HALVES * 64) + slice * 64 + lane_sel;
  bool works = warp < 4 * SLICES && done;
  if (parts > 1) {
    if (works) {
      tc_fence_after();
      float* mine = partial + (part * SLICES + slice) * 8192 + row;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(ta + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) __stcg(mine + (c * 32 + i) * 128, __uint_as_float(r[i]));
      }
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) bars->last = atomicAdd(arrived, 1) == parts - 1;
    __syncthreads();
    works = works && bars->last;
    __threadfence();
  }
  if (works) {
    // The stationary operands have been read for the last time; their buffers take the gradient tiles.
    tc_fence_after();
    const bool is_k = slice < L::HALVES;
    const int h = is_k ? slice : slice - L::HALVES;
    uint8_t* obuf = smem + (is_k ? L::X1_OFF : L::X2_OFF) + h * 16384;
    const float sc = is_k ? scale : 1.f;
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
      uint32_t r[32], w[16];
      if (parts == 1) {
        tmem_ld_32x32(ta + c * 32, r);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0;
        for (int p = 0; p < parts; ++p) {
          const float* share = partial + (p * SLICES + slice) * 8192 + c * 32 * 128 + row;
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __ldcg(share + i * 128));
        }
      }
#pragma unroll
      for (int i = 0; i < 16; ++i)
        w[i] = pack_bf16x2(__uint_as_float(r[2 * i]) * sc, __uint_as_float(r[2 * i + 1]) * sc);
      store_row_chunk_sw128(obuf, row, c * 4, w);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      tma_store_2d_bulk(tmap_dqkv, obuf + (warp & 3) * 32 * 128, (Hq + (is_k ? 0 : Hkv) + g) * HD + 64 * h,
                        tok0 + xb * 128 + (warp & 3) * 32);
      bulk_commit_group();
      bulk_wait_group<0>();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == BWD_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// The dQ pass: one query tile of one head against 128-key blocks.  With no dV product the scores need not stay in
// tensor memory, so there is room for 128-wide tiles: S double-buffered, dP whose columns take dS, dQ.  A 128x128x16
// MMA with both operands in shared memory runs at the arithmetic rate (64 cycles) where two 128x64x16 ones take 96.
// The MMAs of a block are dQ of i, dP of i + 1, S of i + 2; four groups of warps share the columns of every block, and
// the exponentials of block i + 1 run under dQ of i and dP of i + 1.
template <int HD>
struct DqSmem {
  static constexpr int HALVES = HD / 64;
  static constexpr int TILE = 128 * HD * 2;
  static constexpr int K_STAGES = 3;               // K is read by S and, two blocks of MMAs later, by dQ
  static constexpr int X1_OFF = 0;                 // Q; takes the dQ tile at the end
  static constexpr int X2_OFF = TILE;              // dO
  static constexpr int K_OFF = 2 * TILE;
  static constexpr int V_OFF = K_OFF + K_STAGES * TILE;    // 2 stages
  static constexpr int BAR_OFF = V_OFF + 2 * TILE;
  static constexpr int TOTAL = BAR_OFF + 256 + 1024;
};

struct DqBars {
  uint64_t x_full;
  uint64_t k_full[3], k_empty[3], v_full[2], v_empty[2];
  uint64_t s_full[2], dp_full, ds_full;
  uint64_t acc_full;
  uint32_t tmem_base;
};

template <int HD>
__device__ __forceinline__ void attn_dq_cta(const CUtensorMap* tmap_qkv_x, const CUtensorMap* tmap_do_x,
                                            const CUtensorMap* tmap_dqkv, const float* __restrict__ lse,
                                            const float* __restrict__ delta, int xb, int hy, int b, int S, int Hq,
                                            int Hkv, float scale, float scale_log2, int* status) {
  using L = DqSmem<HD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  DqBars* bars = reinterpret_cast<DqBars*>(smem + L::BAR_OFF);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int g = hy / (Hq / Hkv);
  const int tok0 = b * S;
  const int n_blocks = xb + 1;

  if (threadIdx.x == 0) {
    mbar_init(&bars->x_full, 1);
    for (int i = 0; i < L::K_STAGES; ++i) {
      mbar_init(&bars->k_full[i], 1);
      mbar_init(&bars->k_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->v_full[i], 1);
      mbar_init(&bars->v_empty[i], 1);
      mbar_init(&bars->s_full[i], 1);
    }
    mbar_init(&bars->dp_full, 1);
    mbar_init(&bars->ds_full, 16);             // one arrival per softmax warp
    mbar_init(&bars->acc_full, 1);
    fence_mbar_init();
    tma_prefetch_desc(tmap_qkv_x);
    tma_prefetch_desc(tmap_do_x);
    tma_prefetch_desc(tmap_dqkv);
  }
  if (warp == BWD_MMA_WARP) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  grid_wait(lse, delta);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
  // columns: [0,128) S even  [128,256) S odd  [256,384) dP, dS  [384,384+HD) dQ

  if (warp == BWD_TMA_WARP) {
    // ------------------------------------------------------------- TMA
    if (lane == 0) {
      mbar_arrive_expect_tx(&bars->x_full, 2 * L::TILE);
      for (int h = 0; h < L::HALVES; ++h) {
        tma_load_2d(smem + L::X1_OFF + h * 16384, tmap_qkv_x, &bars->x_full, hy * HD + 64 * h, tok0 + xb * 128);
        tma_load_2d(smem + L::X2_OFF + h * 16384, tmap_do_x, &bars->x_full, hy * HD + 64 * h, tok0 + xb * 128);
      }
      int kj = 0, vj = 0;
      for (; vj < n_blocks; ++vj) {
        if (!await(&bars->k_empty[kj % L::K_STAGES], ((kj / L::K_STAGES) & 1) ^ 1, status)) break;
        const int ks = kj % L::K_STAGES;
        mbar_arrive_expect_tx(&bars->k_full[ks], L::TILE);
        for (int h = 0; h < L::HALVES; ++h)
          tma_load_2d(smem + L::K_OFF + ks * L::TILE + h * 16384, tmap_qkv_x, &bars->k_full[ks],
                      (Hq + g) * HD + 64 * h, tok0 + kj * 128);
        ++kj;
        if (!await(&bars->v_empty[vj & 1], ((vj >> 1) & 1) ^ 1, status)) break;
        mbar_arrive_expect_tx(&bars->v_full[vj & 1], L::TILE);
        for (int h = 0; h < L::HALVES; ++h)
          tma_load_2d(smem + L::V_OFF + (vj & 1) * L::TILE + h * 16384, tmap_qkv_x, &bars->v_full[vj & 1],
                      (Hq + Hkv + g) * HD + 64 * h, tok0 + vj * 128);
      }
      grid_launch();
      if (vj < n_blocks) {
        // Unwinding: wait (bounded) for the copies in flight.
        await(&bars->x_full, 0, nullptr);
        for (int j = kj - 1; j >= 0 && j >= kj - L::K_STAGES; --j)
          await(&bars->k_full[j % L::K_STAGES], (j / L::K_STAGES) & 1, nullptr);
        for (int j = vj - 1; j >= 0 && j >= vj - 2; --j) await(&bars->v_full[j & 1], (j >> 1) & 1, nullptr);
      }
    }
  } else if (warp == BWD_MMA_WARP) {
    // ------------------------------------------------------------- MMA
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, false, false);
    constexpr uint32_t idesc_acc = umma_idesc_bf16(128, HD, false, true);
    const uint64_t dq = umma_desc_sw128(smem_u32(smem + L::X1_OFF), 16, 1024);
    const uint64_t ddo = umma_desc_sw128(smem_u32(smem + L::X2_OFF), 16, 1024);
    const uint64_t dk = umma_desc_sw128(smem_u32(smem + L::K_OFF), 16, 1024);
    const uint64_t dkn = umma_desc_sw128(smem_u32(smem + L::K_OFF), 16384, 1024);     // MN-major view
    const uint64_t dv = umma_desc_sw128(smem_u32(smem + L::V_OFF), 16, 1024);
    auto issue_scores = [&](uint32_t tmem_d, uint64_t dx, uint64_t dy) {
#pragma unroll
      for (int ks = 0; ks < HD / 16; ++ks) {
        const uint32_t off = ((ks / 4) * 16384 + (ks % 4) * 32) >> 4;
        umma_bf16_ss(tmem_d, dx + off, dy + off, idesc_s, ks > 0 ? 1u : 0u);
      }
    };
    auto s_block = [&](int j) -> bool {
      const int st = j % L::K_STAGES;
      if (!await_all(&bars->k_full[st], (j / L::K_STAGES) & 1, status)) return false;
      tc_fence_after();
      if (elect_one()) {
        issue_scores(tmem_base + (j & 1) * 128, dq, dk + (st * L::TILE >> 4));
        umma_commit(&bars->s_full[j & 1]);
      }
      __syncwarp();
      return true;
    };
    auto dp_block = [&](int j) -> bool {
      if (!await_all(&bars->v_full[j & 1], (j >> 1) & 1, status)) return false;
      tc_fence_after();
      if (elect_one()) {
        issue_scores(tmem_base + 256, ddo, dv + ((j & 1) * L::TILE >> 4));
        umma_commit(&bars->dp_full);
        umma_commit(&bars->v_empty[j & 1]);
      }
      __syncwarp();
      return true;
    };
    bool ok = await_all(&bars->x_full, 0, status) && s_block(0) && dp_block(0) && (n_blocks == 1 || s_block(1));
    for (int i = 0; i < n_blocks && ok; ++i) {
      ok = await_all(&bars->ds_full, i & 1, status);     // and the scores of block i have been read
      if (!ok) break;
      tc_fence_after();
      if (elect_one()) {
        const uint64_t kn = dkn + ((i % L::K_STAGES) * L::TILE >> 4);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)     // dS of 32 keys each at columns 256, 288, 320, 352
          umma_bf16_ts(tmem_base + 384, tmem_base + 256 + (ks / 2) * 32 + (ks % 2) * 8, kn + (ks * 2048 >> 4), idesc_acc,
                       (i == 0 && ks == 0) ? 0u : 1u);
        umma_commit(&bars->k_empty[i % L::K_STAGES]);
        if (i == n_blocks - 1) umma_commit(&bars->acc_full);
      }
      __syncwarp();
      if (i + 1 < n_blocks) ok = dp_block(i + 1);
      if (i + 2 < n_blocks) ok = ok && s_block(i + 2);
    }
  } else {
    // --------------------------------------------------- dS blocks + epilogue
    const int wg = warp >> 2;                  // key columns [32 wg, 32 wg + 32) of every block
    const int row = (warp & 3) * 32 + lane;    // query row == TMEM lane
    const uint32_t lane_sel = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t td = tmem_base + lane_sel + 256 + wg * 32;
    const float2 sl2 = make_float2(scale_log2, scale_log2);
    const long long idx = (static_cast<long long>(b) * Hq + hy) * S + xb * 128 + row;
    const float nl = lse[idx] * -1.4426950408889634f, ndl = -delta[idx];
    const float2 nl2 = make_float2(nl, nl), ndl2 = make_float2(ndl, ndl);
    bool ok = true;
    for (int j = 0; j < n_blocks; ++j) {
      if (!await_all(&bars->s_full[j & 1], (j >> 1) & 1, status)) { ok = false; break; }
      tc_fence_after();
      uint32_t sv[32];
      tmem_ld_32x32(tmem_base + lane_sel + (j & 1) * 128 + wg * 32, sv);
      tmem_ld_wait();
      if (j == xb) {
        // causal mask: a score of -inf turns into a probability and a score gradient of exactly zero
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (wg * 32 + i > row) sv[i] = 0xff800000u;
      }
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float2 p = fma2(make_float2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), sl2, nl2);
        sv[i] = __float_as_uint(fast_exp2(p.x));
        sv[i + 1] = __float_as_uint(fast_exp2(p.y));
      }
      if (!await_all(&bars->dp_full, j & 1, status)) { ok = false; break; }
      tc_fence_after();
      uint32_t dv[32], dw[16];
      tmem_ld_32x32(td, dv);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float2 d = add2(make_float2(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), ndl2);
        d = mul2(d, make_float2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])));
        dw[i] = pack_bf16x2(d.x, d.y);
      }
      tmem_st_32x16(td, dw);                   // over columns this thread has already read
      tmem_st_wait();
      tc_fence_before();
      warp_arrive(&bars->ds_full, lane);
    }
    if (ok && wg < L::HALVES && await_all(&bars->acc_full, 0, status)) {
      // Q has been read for the last time; its buffer takes the dQ tile, one 64-column half per warp group
      tc_fence_after();
      const uint32_t ta = tmem_base + lane_sel + 384 + wg * 64;
      uint8_t* obuf = smem + L::X1_OFF + wg * 16384;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32], w[16];
        tmem_ld_32x32(ta + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i)
          w[i] = pack_bf16x2(__uint_as_float(r[2 * i]) * scale, __uint_as_float(r[2 * i + 1]) * scale);
        store_row_chunk_sw128(obuf, row, c * 4, w);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d_bulk(tmap_dqkv, obuf + (warp & 3) * 32 * 128, hy * HD + 64 * wg,
                          tok0 + xb * 128 + (warp & 3) * 32);
        bulk_commit_group();
        bulk_wait_group<0>();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == BWD_MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// One launch for both passes.  They are independent (dK/dV and dQ go to different columns of d_qkv) and hold a whole
// SM per CTA; the dK/dV CTAs are few and of very different lengths (with grouped heads up to group x S/64 tiles),
// so they start first, longest first, and the many shorter dQ CTAs fill the SMs they leave.
template <int HD>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_qkv_x,   // box {64, 128} over packed qkv
                const __grid_constant__ CUtensorMap tmap_qkv_y,   // box {64, 64}  over packed qkv
                const __grid_constant__ CUtensorMap tmap_do_x,    // box {64, 128} over dO [T, Hq*hd]
                const __grid_constant__ CUtensorMap tmap_do_y,    // box {64, 64}  over dO
                const __grid_constant__ CUtensorMap tmap_dqkv,    // box {64, 32}  over d_qkv
                const float* __restrict__ lse, const float* __restrict__ delta, int B, int S, int Hq, int Hkv,
                int parts, float* __restrict__ partial, int* __restrict__ arrived, float scale, float scale_log2,
                int* status) {
  const int blocks = S / 128;
  const int n_kv = blocks * Hkv * B * parts;
  int idx = blockIdx.x;
  if (idx < n_kv) {
    const int part = idx % parts;
    idx /= parts;
    const int hb = idx % (Hkv * B);
    attn_dkv_cta<HD>(&tmap_qkv_x, &tmap_qkv_y, &tmap_do_y, &tmap_dqkv, lse, delta, idx / (Hkv * B), hb % Hkv, hb / Hkv,
                     part, parts, partial + static_cast<long long>(idx) * parts * HD * 256, arrived + idx, S, Hq, Hkv,
                     scale, scale_log2, status);
  } else {
    idx -= n_kv;
    const int hb = idx % (Hq * B);
    attn_dq_cta<HD>(&tmap_qkv_x, &tmap_do_x, &tmap_dqkv, lse, delta, blocks - 1 - idx / (Hq * B), hb % Hq, hb / Hq, S,
                    Hq, Hkv, scale, scale_log2, status);
  }
}

template <typename K>
int set_smem(K kern, int bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess
             ? 0
             : -2;
}

}  // namespace

int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                      uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer);

// Two query tiles per CTA read every K and V block once for both; one tile in two halves is done in little more than half the
// time of a tile in one chain.  As long as every tile has an SM of its own, or the SMs get through all key blocks of all
// tiles (longest first) before a longest tile and a block have passed, one tile per CTA finishes earlier.  One against
// two on 148 SMs, head dimension 64 / 128, in us: 2 key blocks, 148 tiles 5.4 against 7.1 / 6.6 against 8.4, 180 tiles 9.2 against 7.3 /
// 10.8 against 8.8; 4 blocks, 256 tiles 11.8 against 11.0 / 13.9 against 13.0; 16 blocks, 256 tiles 20.9 against 31.7 / 24.0 against 34.1,
// 448 tiles 35.7 against 32.3 / 41.4 against 34.7; with one block two tiles are never slower.
// That line is right for a tile in one chain; the halves move it, to some 270 tiles at 8 blocks, 350 at 16 and 450 at 32, and in
// between it takes two where one is faster: 8 blocks, 256 tiles 14.7 against 17.7 / 17.3 against 19.7; 16 blocks, 304 tiles 26.0 against
// 31.9 / 30.3 against 34.5; 32 blocks, 288 tiles, the worst, 35.4 against 59.8 / 40.5 against 62.7.
// The number also decides the order in which a row's sums are added (by halves or in one chain, with probabilities rounded
// against other maxima), so that outputs depend in their rounding on batch, heads and SMs: the same sequence alone and in a batch
// that takes two tiles differs by what two roundings to bf16 of every probability and of the output allow.
int attn_tiles_per_cta(int B, int S, int Hq, int num_sms) {
  const long long blocks = S / 128, tiles = static_cast<long long>(B) * Hq * blocks;
  return tiles <= num_sms || tiles * (blocks + 1) / 2 <= (blocks - 1) * num_sms ? 1 : 2;
}

template <int HD>
static int attn_fwd_impl(const CUtensorMap& tm, const CUtensorMap& to, float* lse, int B, int S, int Hq, int Hkv,
                         float softmax_scale, int num_sms, int* status, cudaStream_t st) {
  static bool cfg = false;
  if (!cfg) {
    if (set_smem(attn_fwd_kernel<HD, true>, FwdSmem<HD>::TOTAL) || set_smem(attn_fwd_kernel<HD, false>, FwdSmem<HD>::TOTAL))
      return -2;
    cfg = true;
  }
  const float scale_log2 = softmax_scale * 1.4426950408889634f;
  const long long per_head = static_cast<long long>(Hq / Hkv) * (S / 128);
  const int tiles_per_cta = attn_tiles_per_cta(B, S, Hq, num_sms);
  const long long ctas = (per_head + tiles_per_cta - 1) / tiles_per_cta * Hkv * B;
  if (ctas > 0x7fffffffll) return -1;
  launch_overlapped(tiles_per_cta == 1 ? attn_fwd_kernel<HD, true> : attn_fwd_kernel<HD, false>, static_cast<unsigned>(ctas),
                    FWD_THREADS, FwdSmem<HD>::TOTAL, st, tm, to, lse, S, Hq, Hkv, B, tiles_per_cta, scale_log2,
                    status);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

int attn_fwd(const void* qkv, void* out, float* lse, int B, int S, int Hq, int Hkv, int hd,
             float softmax_scale, int num_sms, int* status, cudaStream_t st) {
  if (S % 128 != 0 || Hq % Hkv != 0 || (hd != 64 && hd != 128)) return -1;
  if (B == 0) return 0;
  const long long T = static_cast<long long>(B) * S;
  const uint64_t W = static_cast<uint64_t>(Hq + 2 * Hkv) * hd;
  const uint64_t Wo = static_cast<uint64_t>(Hq) * hd;
  CUtensorMap tm, to;
  int rc = make_tmap_2d_bf16(&tm, qkv, W, T, W * 2, 64, 128);
  if (rc != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&to, out, Wo, T, Wo * 2, 64, 32)) != 0) return rc;
  return hd == 128 ? attn_fwd_impl<128>(tm, to, lse, B, S, Hq, Hkv, softmax_scale, num_sms, status, st)
                   : attn_fwd_impl<64>(tm, to, lse, B, S, Hq, Hkv, softmax_scale, num_sms, status, st);
}

// CTAs that share the query heads of a key block in the dK/dV pass.  The launch takes the work over the SMs (about 5,800
// cycles per 128 x 128 tile of both passes and 6,000 per CTA) or its longest CTA (1,600 cycles per 64 query rows of each of
// its heads in the first key block, and the exchange of the parts' sums), whichever is longer; splitting has to shorten
// that by 3 %.  One CTA per key block against the split, on 148 SMs: 1 x 5120, 16 q / 2 kv heads x 128 540 and 289 us in two; 1 x
// 4096, 32 / 4 x 128 442 and 374 us in two; 2 x 2048, 32 / 4 x 128 231 and 219 us in two; 1 x 512, 32 / 4 x 128 70 and 37 us in four;
// not split: 1 x 4096, 32 / 8 x 128 368 and 393 us, 8 x 1024, 16 / 2 x 64 124 and 132 us, 8 x 128, 16 / 4 x 128 13.3 and 15.8 us.
int attn_bwd_parts(int B, int S, int Hq, int Hkv, int num_sms) {
  const long long blocks = S / 128, group = Hkv > 0 ? Hq / Hkv : 1;
  auto cost = [&](long long parts) {
    const long long tiles = B * Hq * blocks * (blocks + 1) / 2, ctas = B * blocks * (Hkv * parts + Hq);
    const long long work = (tiles * 5800 + ctas * 6000) / num_sms;
    const long long longest = group / parts * 2 * blocks * 1600 + 6000 + (parts > 1 ? 3000 + 3000 * parts : 0);
    return work > longest ? work : longest;
  };
  int best = 1;
  for (int parts = 2; parts <= 8 && group % parts == 0; parts *= 2)
    if (cost(parts) * 100 < cost(best) * 97) best = parts;
  return best;
}

template <int HD>
static int attn_bwd_impl(const void* qkv, const void* out, const void* d_out, const float* lse,
                         float* delta, float* scratch, void* d_qkv, int B, int S, int Hq, int Hkv,
                         float softmax_scale, int num_sms, int* status, cudaStream_t st) {
  const long long T = static_cast<long long>(B) * S;
  const uint64_t W = static_cast<uint64_t>(Hq + 2 * Hkv) * HD;
  const uint64_t Wo = static_cast<uint64_t>(Hq) * HD;
  if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(d_out) | reinterpret_cast<uintptr_t>(lse) |
        reinterpret_cast<uintptr_t>(delta)) & 15u) != 0)
    return -1;
  if (T * Hq >= (1ll << 31)) return -1;
  CUtensorMap tqx, tqy, tdx, tdy, tdq;
  int rc;
  if ((rc = make_tmap_2d_bf16(&tqx, qkv, W, T, W * 2, 64, 128)) != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&tqy, qkv, W, T, W * 2, 64, 64)) != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&tdx, d_out, Wo, T, Wo * 2, 64, 128)) != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&tdy, d_out, Wo, T, Wo * 2, 64, 64)) != 0) return rc;
  if ((rc = make_tmap_2d_bf16(&tdq, d_qkv, W, T, W * 2, 64, 32)) != 0) return rc;
  constexpr int smem = DqSmem<HD>::TOTAL > BwdSmem<HD>::TOTAL ? DqSmem<HD>::TOTAL : BwdSmem<HD>::TOTAL;
  static bool cfg = false;
  if (!cfg) {
    if (set_smem(attn_bwd_kernel<HD>, smem)) return -2;
    cfg = true;
  }
  // scratch: a counter per key block, padded to 16 bytes, and the parts' sums
  const int parts = scratch == nullptr ? 1 : attn_bwd_parts(B, S, Hq, Hkv, num_sms);
  const int n_kv = S / 128 * Hkv * B;
  int* arrived = reinterpret_cast<int*>(scratch);
  float* partial = scratch == nullptr ? nullptr : scratch + (n_kv + 3) / 4 * 4;
  const long long delta_blocks = (T * Hq * (HD / 8) + 255) / 256;
  launch_overlapped(attn_delta_kernel<HD>, static_cast<unsigned>(delta_blocks < 148 * 16 ? delta_blocks : 148 * 16), 256, 0, st,
      static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(d_out), delta, arrived,
      parts > 1 ? n_kv : 0, T, S, Hq);
  if (cudaGetLastError() != cudaSuccess) return -3;
  launch_overlapped(attn_bwd_kernel<HD>, static_cast<unsigned>(n_kv * parts + S / 128 * Hq * B), BWD_THREADS, smem, st,
      tqx, tqy, tdx, tdy, tdq, lse, delta, B, S, Hq, Hkv, parts, partial, arrived, softmax_scale,
      softmax_scale * 1.4426950408889634f, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

long long attn_bwd_scratch(int B, int S, int Hq, int Hkv, int hd, int num_sms) {
  const int parts = attn_bwd_parts(B, S, Hq, Hkv, num_sms);
  const long long n_kv = static_cast<long long>(S / 128) * Hkv * B;
  return parts == 1 ? 0 : (n_kv + 3) / 4 * 4 + n_kv * parts * hd * 256;
}

int attn_bwd(const void* qkv, const void* out, const void* d_out, const float* lse, float* delta, float* scratch,
             void* d_qkv, int B, int S, int Hq, int Hkv, int hd, float softmax_scale, int num_sms, int* status,
             cudaStream_t st) {
  if (S % 128 != 0 || Hq % Hkv != 0 || (hd != 64 && hd != 128)) return -1;
  if (B == 0) return 0;
  if (hd == 128)
    return attn_bwd_impl<128>(qkv, out, d_out, lse, delta, scratch, d_qkv, B, S, Hq, Hkv, softmax_scale, num_sms, status, st);
  return attn_bwd_impl<64>(qkv, out, d_out, lse, delta, scratch, d_qkv, B, S, Hq, Hkv, softmax_scale, num_sms, status, st);
}

}  // namespace piper
