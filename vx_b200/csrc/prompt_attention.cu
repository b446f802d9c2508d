/* prompt_attention.cu -- attention over the positions of a prompt, f32 queries and an
 * f32 cache, on the tensor cores (nn_attention, nn.vx:349-866, for every position).
 *
 * A block per (128 positions, query head), head_dim 128; 64 keys at a time.  An f32
 * value from 2^-109 on is the exact sum of three bf16 terms (below, the third is cut to
 * the subnormals: 2^-134 of one is lost, as in the output's own terms), and a product
 * keeps the six largest of the nine term products (what is dropped is below 2^-24 of it),
 * as in gemm_f32_tile.cu:
 *
 *   scores   q1 [k1 | k2 | k3], q2 [k1 | k2], q3 k1: the terms of a tile of keys lie
 *            one after another along N, so three instructions a K step do all six
 *            products, those of equal weight in one accumulator each (3 x 64 columns);
 *   weights  expf of the f32 scores against a running maximum, split into three terms
 *            in tensor memory, where the second product takes them from;
 *   values   the six products of one tile, the small ones first, into an accumulator
 *            that starts from zero for each tile of keys; the sum over the tiles is
 *            kept in registers in f32, so that no long sum is left to the tensor core.
 *
 * Thirteen warps: 0-7 hold the 128 rows (two threads a row: half of the keys and half
 * of the output each), 8-11 read keys and values from the cache, split them and write
 * the terms into two 48 KiB buffers of 128-byte-swizzled rows, warp 12 issues
 * the products: those of the next tile's scores before the values of this one,
 * so that they run under the softmax.  The same layout serves the scores (K-major) and
 * the values (N-major), so where the keys are the values a tile is read once.
 *
 * What bounds it: the round between the row threads and the tensor core, about 10 000
 * cycles a tile, of which the products need 3 200 (24 instructions of N = 192 / 128 / 64
 * for the scores and 24 of N = 128 for the values of 128 x 64).  500 positions of 32 heads:
 * 57 us, 207 on the FMA pipe; 1500 positions of 32 heads over one ring with a window of
 * 1024: 182 us, about 600 on the FMA pipe.  With the 32 scores of a thread in registers and
 * the code unrolled over them it was 67 and 203.
 *
 * Magnitudes from 2^56 on, infinities and NaN, whose terms or products could overflow
 * where the scores do not, are noticed while they are read; a block that met one
 * computes its rows with plain multiply-adds as well, a key after another: 1.2 ms for
 * one head of 32 over 500 positions.
 */
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "ptx.cuh"
#include "terms.cuh"

#include <climits>

namespace vxb {
namespace {

constexpr int HD = 128, BQ = 128, BKV = 64;
constexpr int ROW_WARPS = 8, LOAD_WARPS = 4, MMA_WARP = ROW_WARPS + LOAD_WARPS;
constexpr int THREADS = (MMA_WARP + 1) * 32;
constexpr int Q_TERM = BQ * HD * 2, Q_HALF = Q_TERM / 2;
constexpr int KV_TERM = BKV * 128, KV_HALF = 3 * KV_TERM, KV_BYTES = 2 * KV_HALF;
constexpr int S_COL = 0, T_COL = 192, O_COL = 256, P_COL = 384; /* of tensor memory */
constexpr float LOWEST = -3.0e38f;
constexpr uint32_t kLargest = 0x5b800000u; /* 2^56 */

enum { A_Q = 0x91, A_EMPTY, A_KEYS, A_VALUES, A_S_FREE, A_S_FULL, A_P_FULL, A_O_FULL };
__device__ int g_prompt_status; /* first wait that ran out since the last read */

struct Bars {
  uint64_t q_full, full[2], empty[2], s_full, s_free, p_full, o_full;
  uint32_t tmem_base;
  int stop;
  int plain;
  float most[2][2][BQ]; /* [tile parity][half][row] */
};
constexpr int SMEM_BYTES = 3 * Q_TERM + 2 * KV_BYTES + 1024 + (int)sizeof(Bars) + 64;

/* Eight values as three words of four bf16 pairs, a term every `pitch` bytes. */
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ void split2(float x, float y, uint32_t &a, uint32_t &b,
                                       uint32_t &c) {
  a = pack(x, y);
  const float rx = x - __uint_as_float(a << 16);
  const float ry = y - __uint_as_float(a & 0xffff0000u);
  b = pack(rx, ry);
  c = pack(rx - __uint_as_float(b << 16), ry - __uint_as_float(b & 0xffff0000u));
}
__device__ __forceinline__ uint32_t magnitude(float x) {
  return __float_as_uint(x) & 0x7fffffffu;
}
__device__ __forceinline__ void split8(const float4 &u, const float4 &v, uint8_t *at,
                                       int pitch, uint32_t &most) {
  const float x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
  uint32_t w[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    most = max(most, max(magnitude(x[2 * j]), magnitude(x[2 * j + 1])));
    split2(x[2 * j], x[2 * j + 1], w[0][j], w[1][j], w[2][j]);
  }
#pragma unroll
  for (int t = 0; t < 3; ++t)
    *reinterpret_cast<uint4 *>(at + t * pitch) =
        make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
}

/* A wait that ran out: noted, and nobody waits for long from then on. The roles with
   warp-wide steps carry on to their end (over values that mean nothing). */
#define WAIT(bar, parity, code)                                                          \
  do {                                                                                   \
    if (!ptx::mbar_wait((bar), (parity), stop)) {                                        \
      atomicCAS(&g_prompt_status, 0, (code));                                            \
      *stop = 1;                                                                         \
    }                                                                                    \
  } while (0)

template <bool kShared>
__global__ void __launch_bounds__(THREADS, 1)
prompt_attention_kernel(const PromptAttnArgs a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *const kv_smem = smem + 3 * Q_TERM;
  Bars *bars = reinterpret_cast<Bars *>(kv_smem + 2 * KV_BYTES);
  const int tid = threadIdx.x, warp = ptx::warp_index(), lane = tid % 32;

  if (tid == 0) {
    ptx::mbar_init(&bars->q_full, ROW_WARPS);
    for (int s = 0; s < 2; ++s) {
      ptx::mbar_init(&bars->full[s], LOAD_WARPS);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    ptx::mbar_init(&bars->s_full, 1);
    ptx::mbar_init(&bars->s_free, ROW_WARPS);
    ptx::mbar_init(&bars->p_full, ROW_WARPS);
    ptx::mbar_init(&bars->o_full, 1);
    bars->stop = 0;
    bars->plain = 0;
    ptx::fence_barrier_init();
  }
  if (warp == MMA_WARP)
    ptx::tmem_alloc(&bars->tmem_base, 512);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  volatile int *stop = &bars->stop;
  chain_release();
  chain_wait();

  const int head = blockIdx.x, g = head / (a.q_heads / a.kv_heads);
  const int t0 = (int)(gridDim.y - 1 - blockIdx.y) * BQ; /* most keys first */
  const int base = a.positions[0];
  const int first_key = max(0, base + t0 - a.window + 1);
  const int last_key = base + min(t0 + BQ, a.t) - 1;
  const int tiles = (last_key - first_key) / BKV + 1;
  const int row_first = first_key % a.cache_rows;
  const int64_t row_floats = (int64_t)a.kv_heads * HD;
  float o[64]; /* of row `row`: values half * 64 .. */
  float m = LOWEST, l = 0.0f;
  const int quarter = warp & 3, half = (warp >> 2) & 1, row = quarter * 32 + lane;

  if (warp < ROW_WARPS) {
    uint32_t most = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = tid / 16 + 16 * i, c = tid % 16;
      float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v = u;
      if (t0 + r < a.t) {
        const float4 *from = reinterpret_cast<const float4 *>(
            a.q + (t0 + r) * a.q_stride + (int64_t)head * HD + c * 8);
        u = from[0];
        v = from[1];
      }
      split8(u, v, smem + (c >> 3) * Q_HALF + r * 128 + (((c & 7) ^ (r & 7)) << 4),
             Q_TERM, most);
    }
    if (most >= kLargest)
      bars->plain = 1;
    ptx::fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0)
      ptx::mbar_arrive(&bars->q_full);

    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    const int at = base + t0 + row; /* this row's position */
#pragma unroll
    for (int i = 0; i < 64; ++i)
      o[i] = 0.0f;
    /* what the values of the tile before came to */
    auto take_values = [&](float fix) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t v[16];
        ptx::tmem_ld_32x32b_x16(lanes + O_COL + half * 64 + q * 16, v);
        ptx::tmem_ld_wait_for(v);
#pragma unroll
        for (int e = 0; e < 16; ++e)
          o[q * 16 + e] = (o[q * 16 + e] + __uint_as_float(v[e])) * fix;
      }
    };
    for (int j = 0; j < tiles; ++j) {
      WAIT(&bars->s_full, j & 1, A_S_FULL);
      ptx::tc_fence_after_sync();
      /* The keys this row sees are from..to of these 32. Eight at a time, in loops: the
         scores go back to tensor memory until the maximum is known, and the code of a
         tile is short (unrolled it ran at the pace of instruction fetches). */
      const int k0 = first_key + j * BKV + half * 32;
      const int from = at - a.window + 1 - k0, to = at - k0;
      float big = LOWEST;
#pragma unroll 1
      for (int q = 0; q < 32; q += 8) {
        uint32_t x[8], y[8], z[8];
        const uint32_t col = lanes + S_COL + half * 32 + q;
        ptx::tmem_ld_32x32b_x8(col, x);
        ptx::tmem_ld_32x32b_x8(col + BKV, y);
        ptx::tmem_ld_32x32b_x8(col + 2 * BKV, z);
        ptx::tmem_ld_wait_for(x);
        ptx::tmem_ld_wait_for(y);
        ptx::tmem_ld_wait_for(z);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float s = __uint_as_float(x[e]) +
                          (__uint_as_float(y[e]) + __uint_as_float(z[e]));
          const float seen = q + e >= from && q + e <= to ? s * a.scale : LOWEST;
          big = fmaxf(big, seen);
          x[e] = __float_as_uint(seen);
        }
        ptx::tmem_st_32x32b_x8(lanes + T_COL + half * 32 + q, x);
      }
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->s_free);
      bars->most[j & 1][half][row] = big;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
      const float mn = fmaxf(m, fmaxf(big, bars->most[j & 1][half ^ 1][row]));
      const float fix = expf(m - mn);
      m = mn;
      /* the weights of the tile before are read until its values are there */
      if (j > 0) {
        WAIT(&bars->o_full, (j - 1) & 1, A_O_FULL);
        ptx::tc_fence_after_sync();
      }
      float sum = 0.0f;
#pragma unroll 1
      for (int q = 0; q < 32; q += 8) {
        uint32_t x[8], p1[4], p2[4], p3[4];
        ptx::tmem_ld_32x32b_x8(lanes + T_COL + half * 32 + q, x);
        ptx::tmem_ld_wait_for(x);
        float w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          w[e] = q + e >= from && q + e <= to ? expf(__uint_as_float(x[e]) - mn) : 0.0f;
          sum += w[e];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          split2(w[2 * e], w[2 * e + 1], p1[e], p2[e], p3[e]);
        const uint32_t col = lanes + P_COL + half * 16 + q / 2;
        ptx::tmem_st_32x32b_x4(col, p1);
        ptx::tmem_st_32x32b_x4(col + 32, p2);
        ptx::tmem_st_32x32b_x4(col + 64, p3);
      }
      l = l * fix + sum;
      if (j > 0)
        take_values(fix);
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->p_full);
    }
    WAIT(&bars->o_full, (tiles - 1) & 1, A_O_FULL);
    ptx::tc_fence_after_sync();
    take_values(1.0f);
    bars->most[tiles & 1][half][row] = l;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
    l = bars->most[tiles & 1][0][row] + bars->most[tiles & 1][1][row];
  } else if (warp < MMA_WARP) {
    /* an item is a tile of keys or of values: 64 rows of sixteen runs of eight */
    const int items = kShared ? tiles : 2 * tiles;
    const int r0 = (tid - ROW_WARPS * 32) / 16, c = tid % 16; /* rows r0 + 8 i */
    uint8_t *const to =
        kv_smem + (c >> 3) * KV_HALF + r0 * 128 + (((c & 7) ^ r0) << 4);
    float4 v[8][2];
    auto read = [&](int item) {
      const int j = kShared ? item : item >> 1;
      const float *from = (kShared || !(item & 1) ? a.k : a.v) + (int64_t)g * HD + c * 8;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int n = j * BKV + r0 + 8 * i;
        v[i][0] = v[i][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (first_key + n <= last_key) {
          int at = row_first + n;
          if (at >= a.cache_rows)
            at -= a.cache_rows;
          const float4 *p = reinterpret_cast<const float4 *>(from + at * row_floats);
          v[i][0] = p[0];
          v[i][1] = p[1];
        }
      }
    };
    uint32_t most = 0;
    read(0);
    for (int item = 0; item < items; ++item) {
      const int b = item & 1;
      WAIT(&bars->empty[b], ((item >> 1) & 1) ^ 1, A_EMPTY);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        split8(v[i][0], v[i][1], to + b * KV_BYTES + i * 8 * 128, KV_TERM, most);
      if (item + 1 < items)
        read(item + 1);
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->full[b]);
    }
    if (most >= kLargest)
      bars->plain = 1;
  } else {
    const uint32_t of_three = ptx::idesc_f16(true, false, false, BQ, 3 * BKV);
    const uint32_t of_two = ptx::idesc_f16(true, false, false, BQ, 2 * BKV);
    const uint32_t of_one = ptx::idesc_f16(true, false, false, BQ, BKV);
    const uint32_t of_values = ptx::idesc_f16(true, false, true, BQ, HD);
    const uint64_t q_desc = ptx::smem_desc_sw128(ptx::smem_addr(smem), 16, 1024);
    const uint64_t k_desc = ptx::smem_desc_sw128(ptx::smem_addr(kv_smem), 16, 1024);
    const uint64_t v_desc = ptx::smem_desc_sw128(ptx::smem_addr(kv_smem), KV_HALF, 1024);
    auto scores = [&](int j) {
      const int b = kShared ? j & 1 : 0;
      WAIT(&bars->full[b], kShared ? (j >> 1) & 1 : j & 1, A_KEYS);
      __syncwarp();
      ptx::tc_fence_after_sync();
      if (ptx::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t q = q_desc + (((kk / 4) * Q_HALF + (kk % 4) * 32) >> 4);
          const uint64_t k =
              k_desc + ((b * KV_BYTES + (kk / 4) * KV_HALF + (kk % 4) * 32) >> 4);
          ptx::umma_f16_ss(tmem + S_COL, q, k, of_three, kk != 0);
          ptx::umma_f16_ss(tmem + S_COL + BKV, q + (Q_TERM >> 4), k, of_two, 1);
          ptx::umma_f16_ss(tmem + S_COL + 2 * BKV, q + (2 * Q_TERM >> 4), k, of_one, 1);
        }
        ptx::umma_commit(&bars->s_full);
        if (!kShared)
          ptx::umma_commit(&bars->empty[0]);
      }
      __syncwarp();
    };
    WAIT(&bars->q_full, 0, A_Q);
    scores(0);
    for (int j = 0; j < tiles; ++j) {
      if (j + 1 < tiles) {
        WAIT(&bars->s_free, j & 1, A_S_FREE);
        scores(j + 1);
      }
      const int b = kShared ? j & 1 : 1;
      if (!kShared)
        WAIT(&bars->full[1], j & 1, A_VALUES);
      WAIT(&bars->p_full, j & 1, A_P_FULL);
      __syncwarp();
      ptx::tc_fence_after_sync();
      if (ptx::elect_one()) {
#pragma unroll
        for (int n = 0; n < 6; ++n) {
          /* (weight term, value term): 3 1, 2 2, 1 3, 2 1, 1 2, 1 1 */
          const int pt = n == 0 ? 2 : n == 1 || n == 3 ? 1 : 0;
          const int vt = n == 2 ? 2 : n == 1 || n == 4 ? 1 : 0;
#pragma unroll
          for (int kk = 0; kk < BKV / 16; ++kk)
            ptx::umma_f16_ts(tmem + O_COL, tmem + P_COL + pt * 32 + kk * 8,
                             v_desc + ((b * KV_BYTES + vt * KV_TERM + kk * 2048) >> 4),
                             of_values, (n | kk) != 0);
        }
        ptx::umma_commit(&bars->o_full);
        ptx::umma_commit(&bars->empty[b]);
      }
      __syncwarp();
    }
  }
  __syncwarp();
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == MMA_WARP) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, 512);
    return;
  }

  __nv_bfloat16 *terms = (__nv_bfloat16 *)a.terms;
  if (bars->plain) {
    /* a row per warp, a key after another: rare, so short rather than fast */
    for (int r = warp; r < BQ && t0 + r < a.t; r += MMA_WARP) {
      const int64_t t = t0 + r;
      const int pos = base + (int)t, d = head * HD + lane * 4;
      const float4 q = *reinterpret_cast<const float4 *>(a.q + t * a.q_stride + d);
      float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      float pm = LOWEST, pl = 0.0f;
      for (int key = max(0, pos - a.window + 1); key <= pos; ++key) {
        const int64_t from = key % a.cache_rows * row_floats + (int64_t)g * HD + lane * 4;
        const float4 k = *reinterpret_cast<const float4 *>(a.k + from);
        const float4 v = *reinterpret_cast<const float4 *>(a.v + from);
        float s = fmaf(q.w, k.w, fmaf(q.z, k.z, fmaf(q.y, k.y, q.x * k.x)));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
          s += __shfl_xor_sync(0xffffffffu, s, off);
        s *= a.scale;
        const float mn = fmaxf(pm, s), fix = expf(pm - mn), w = expf(s - mn);
        pm = mn;
        pl = fmaf(pl, fix, w);
        acc.x = fmaf(acc.x, fix, w * v.x);
        acc.y = fmaf(acc.y, fix, w * v.y);
        acc.z = fmaf(acc.z, fix, w * v.z);
        acc.w = fmaf(acc.w, fix, w * v.w);
      }
      float out[4] = {acc.x / pl, acc.y / pl, acc.z / pl, acc.w / pl};
      if (a.gate)
        for (int e = 0; e < 4; ++e)
          out[e] *= a.gate[t * a.gate_stride + d + e];
      store_terms4(terms, a.cols, t, d, out);
    }
  } else if (warp < ROW_WARPS && t0 + row < a.t) {
    const int64_t t = t0 + row;
    const int d = head * HD + half * 64;
#pragma unroll
    for (int i = 0; i < 64; i += 8) {
      float out[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        out[e] = o[i + e] / l;
      if (a.gate) {
        const float4 *gate =
            reinterpret_cast<const float4 *>(a.gate + t * a.gate_stride + d + i);
        const float4 u = gate[0], v = gate[1];
        out[0] *= u.x; out[1] *= u.y; out[2] *= u.z; out[3] *= u.w;
        out[4] *= v.x; out[5] *= v.y; out[6] *= v.z; out[7] *= v.w;
      }
      store_terms8(terms, a.cols, t, d + i, out);
    }
  }
}

} // namespace

const char *prompt_attention(const PromptAttnArgs &a, cudaStream_t stream) {
  if (((uintptr_t)a.terms | (uintptr_t)a.q | (uintptr_t)a.k | (uintptr_t)a.v |
       (uintptr_t)a.gate) & 15 ||
      (a.q_stride | a.gate_stride) % 4 != 0 || a.cols % 8 != 0)
    return "the multi-position attention needs 16-byte aligned rows";
  const bool shared = a.k == a.v;
  auto kernel = shared ? prompt_attention_kernel<true> : prompt_attention_kernel<false>;
  if (allow_dynamic_smem((const void *)kernel, SMEM_BYTES) != cudaSuccess)
    return "the multi-position attention could not get its shared memory";
  launch_chained(kernel, dim3(a.q_heads, (a.t + BQ - 1) / BQ), dim3(THREADS), SMEM_BYTES,
                 stream, a);
  return check_launch("the multi-position attention");
}

int prompt_attention_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_prompt_status, sizeof v) != cudaSuccess)
    return -1;
  if (v)
    cudaMemcpyToSymbol(g_prompt_status, &zero, sizeof zero);
  return v;
}

} // namespace vxb
