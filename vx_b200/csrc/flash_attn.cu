/* flash_attn.cu -- attention forward over whole sequences, bf16 in and out,
 * on the sm_100a tensor cores: out = softmax(q k^T * scale [causal]) v with
 * an f32 online softmax, never materialising the S x S scores.
 *
 * The arithmetic is the reference's attention (scores * scale, subtract the
 * running maximum, exponentiate, weighted sum of V over the sum of weights:
 * tests/optimizations/pass/std_nn_kernels_match_loops_on_the_cpu.vx:347-390)
 * applied to every query row, with the probabilities rounded to bf16 before
 * they multiply V, as every tensor-core flash attention does.  O is rescaled
 * only when a row's maximum has grown by more than 2^8 since the value in use;
 * the final division by the row sum makes the result independent of it, but for
 * where the probabilities round.
 *
 * Sequences of whole pairs of Q tiles start from a maximum of zero.  Those of an
 * odd number of tiles (kBy64) round as 64-key tiles do: their maximum starts as
 * that of a row's first 64 keys, and the row sums are kept in the same order.  The
 * two choices are 3e-3 from each other; the second is nearer to 64 bits under a
 * causal mask (2.1e-3 and 2.3e-3 at 2176 positions; a row's first key has weight 1
 * there) and as near without one, and a sequence keeps the one its results have
 * always had.
 * [2, 32, 1152, 128] without a mask takes 66.6 us that way (69.6 before the kernel was
 * set up under the tail of the one before it, where a maximum of zero took 67.6 and
 * kernels of 64-key tiles 88.2).
 *
 * A CTA owns two tiles of 128 query rows of one (batch, head), or a single one, and
 * walks KV tiles of 128 rows:
 *   warp 0      TMA: the Q tiles once, then K and V tiles into rings;
 *   warp 1      issues tcgen05.mma, S = Q K^T and O += P V;
 *   warps 2..   one warpgroup per Q tile, one thread per query row.
 * The probabilities never go through shared memory -- they are written back into
 * tensor memory over the scores they came from, packed two bf16 per column,
 * and the P V product takes its A operand from there, so it only fetches V.
 *
 * TMEM per Q tile: 128 columns of scores (their first 64 then hold P) and 128
 * columns of O; two Q tiles fill the 512 columns.  Shared memory: Q 64 KiB, a
 * K ring and a V ring of two 32 KiB tiles each.  The MMA warp alternates
 * between the two Q tiles -- P V of tile j, then at once the scores of tile
 * j+1 of the same Q tile -- so that one warpgroup's softmax runs under the
 * other's products.
 */
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "ptx.cuh"

#include <cuda_bf16.h>

#include <mutex>

namespace vxb {

bool make_map_16(CUtensorMap *map, const void *base, int64_t inner, int64_t rows,
                 int64_t ld, int box_inner, int box_rows, bool is_bf16);

namespace {

constexpr int HD = 128;  /* head_dim */
constexpr int BQ = 128;  /* query rows per tile */
constexpr int BKV = 128; /* KV rows per tile */
constexpr int NQ = 2;    /* Q tiles per CTA */
constexpr int RING = 2;  /* tiles in the K ring and in the V ring (a power of 2) */
constexpr int TILE_BYTES = 128 * HD * 2; /* 32 KiB: a Q, K or V tile */
constexpr int THREADS = 64 + NQ * 128;

enum { F2_Q = 0x61, F2_K_FREE, F2_V_FREE, F2_K_FULL, F2_V_FULL, F2_P_FULL,
       F2_S_FULL, F2_PV_DONE };

__device__ int g_flash_status;

struct Bars {
  uint64_t q_full;
  uint64_t k_full[RING], k_free[RING], v_full[RING], v_free[RING];
  uint64_t s_full[NQ], p_full[NQ], pv_done[NQ];
  uint32_t tmem_base;
  int stop;
};
constexpr int SMEM_BYTES =
    NQ * TILE_BYTES + 2 * RING * TILE_BYTES + 1024 + (int)sizeof(Bars) + 256;

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

/* Two f32 in one 64-bit register, for the packed FMA and add of sm_100. */
__device__ __forceinline__ uint64_t pair_of(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void halves_of(uint64_t v, float &a, float &b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

/* One pass over the 128 scores of a row, in eight loads of 16 columns with the
   next load in flight under the arithmetic of the one before:
   p = 2^(s * scale_log2 + neg_m), rounded to bf16 pairs into `packed`; `sum`
   gets the f32 row sum and `rel_max` the largest exponent met. The body is
   long (everything is unrolled so that P stays in registers) and the kernel
   holds one copy of it: the instruction cache is a resource here. */
__device__ __forceinline__ void
probabilities(uint32_t s_tmem, float scale_log2, float neg_m,
              uint32_t (&packed)[BKV / 2], float &rel_max, float &sum) {
  uint32_t raw[2][32];
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  uint64_t part2[4] = {0, 0, 0, 0}; /* pairs of partial sums */
  const uint64_t scale2 = pair_of(scale_log2, scale_log2);
  const uint64_t negm2 = pair_of(neg_m, neg_m);
  ptx::tmem_ld_32x32b_x32(s_tmem, raw[0]);
#pragma unroll
  for (int c = 0; c < BKV / 32; ++c) {
    ptx::tmem_ld_wait_for(raw[c & 1]);
    if (c + 1 < BKV / 32)
      ptx::tmem_ld_32x32b_x32(s_tmem + (c + 1) * 32, raw[(c + 1) & 1]);
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
      /* the packed forms halve the instruction count of the scale and the sum
         (the rounding of each lane is that of the scalar instruction) */
      float r0, r1;
      halves_of(fma2(pair_of(__uint_as_float(raw[c & 1][e]),
                             __uint_as_float(raw[c & 1][e + 1])),
                     scale2, negm2),
                r0, r1);
      mx4[(e >> 1) & 3] = max3(mx4[(e >> 1) & 3], r0, r1);
      const float p0 = ex2(r0), p1 = ex2(r1);
      part2[(e >> 1) & 3] = add2(part2[(e >> 1) & 3], pair_of(p0, p1));
      const __nv_bfloat162 pr = __floats2bfloat162_rn(p0, p1);
      packed[c * 16 + (e >> 1)] = *reinterpret_cast<const uint32_t *>(&pr);
    }
  }
  float part4[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float lo, hi;
    halves_of(part2[q], lo, hi);
    part4[q] = lo + hi;
  }
  rel_max = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
  sum = (part4[0] + part4[1]) + (part4[2] + part4[3]);
}

/* The same arithmetic when the maximum is known to hold (the pass after
   row_max): P can go to tensor memory chunk by chunk, over score columns
   that have been read already, so this form is a short loop instead of a
   second copy of the long body above. Returns the row sum. */
__device__ __forceinline__ float
probabilities_stored(uint32_t s_tmem, float scale_log2, float neg_m) {
  float part4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
  for (int c = 0; c < BKV / 32; ++c) {
    uint32_t raw[32], packed[16];
    ptx::tmem_ld_32x32b_x32(s_tmem + c * 32, raw);
    ptx::tmem_ld_wait_for(raw);
#pragma unroll
    for (int e = 0; e < 32; e += 2) {
      const float p0 = ex2(fmaf(__uint_as_float(raw[e]), scale_log2, neg_m));
      const float p1 = ex2(fmaf(__uint_as_float(raw[e + 1]), scale_log2, neg_m));
      part4[(e >> 1) & 3] += p0 + p1;
      const __nv_bfloat162 pr = __floats2bfloat162_rn(p0, p1);
      packed[e >> 1] = *reinterpret_cast<const uint32_t *>(&pr);
    }
    ptx::tmem_st_32x32b_x16(s_tmem + c * 16, packed);
  }
  return (part4[0] + part4[1]) + (part4[2] + part4[3]);
}

/* The row sums of 32 columns' probabilities in the order of 64-key tiles: each half of
   such a tile has a sum of its own. `a`, `b`: exponentials of columns e .. e + 3. */
struct HalfSums {
  float l[2] = {0.0f, 0.0f};
  uint64_t part[2]; /* four chains, two to a word */
  __device__ __forceinline__ void begin() { part[0] = part[1] = 0; }
  __device__ __forceinline__ void add(int e, float a0, float a1, float b0, float b1) {
    part[(e >> 2) & 1] = add2(part[(e >> 2) & 1], add2(pair_of(a0, b0), pair_of(a1, b1)));
  }
  /* 32 columns are done, of half c & 1; fix: what the sum so far is scaled by */
  __device__ __forceinline__ void end(int c, float fix) {
    float p0, p1, p2, p3;
    halves_of(part[0], p0, p1);
    halves_of(part[1], p2, p3);
    l[c & 1] = fmaf(l[c & 1], fix, (p0 + p1) + (p2 + p3));
  }
};

/* probabilities() with those sums. */
__device__ __forceinline__ void
probabilities_by64(uint32_t s_tmem, float scale_log2, float neg_m,
                   uint32_t (&packed)[BKV / 2], float &rel_max, HalfSums &sums) {
  uint32_t raw[2][32];
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  const uint64_t scale2 = pair_of(scale_log2, scale_log2);
  const uint64_t negm2 = pair_of(neg_m, neg_m);
  ptx::tmem_ld_32x32b_x32(s_tmem, raw[0]);
#pragma unroll
  for (int c = 0; c < BKV / 32; ++c) {
    ptx::tmem_ld_wait_for(raw[c & 1]);
    if (c + 1 < BKV / 32)
      ptx::tmem_ld_32x32b_x32(s_tmem + (c + 1) * 32, raw[(c + 1) & 1]);
    sums.begin();
#pragma unroll
    for (int e = 0; e < 32; e += 4) {
      float p[4];
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        float r0, r1;
        halves_of(fma2(pair_of(__uint_as_float(raw[c & 1][e + i]),
                               __uint_as_float(raw[c & 1][e + i + 1])),
                       scale2, negm2),
                  r0, r1);
        mx4[((e + i) >> 1) & 3] = max3(mx4[((e + i) >> 1) & 3], r0, r1);
        p[i] = ex2(r0);
        p[i + 1] = ex2(r1);
        const __nv_bfloat162 pr = __floats2bfloat162_rn(p[i], p[i + 1]);
        packed[c * 16 + ((e + i) >> 1)] = *reinterpret_cast<const uint32_t *>(&pr);
      }
      sums.add(e, p[0], p[1], p[2], p[3]);
    }
    sums.end(c, 1.0f);
  }
  rel_max = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
}

/* probabilities_stored() with those sums. */
__device__ __forceinline__ void
probabilities_by64_stored(uint32_t s_tmem, float scale_log2, float neg_m, float fix,
                          HalfSums &sums) {
#pragma unroll 1
  for (int c = 0; c < BKV / 32; c += 2) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t raw[32], packed[16];
      ptx::tmem_ld_32x32b_x32(s_tmem + (c + h) * 32, raw);
      ptx::tmem_ld_wait_for(raw);
      sums.begin();
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        float p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          p[i] = ex2(fmaf(__uint_as_float(raw[e + i]), scale_log2, neg_m));
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const __nv_bfloat162 pr = __floats2bfloat162_rn(p[i], p[i + 1]);
          packed[(e + i) >> 1] = *reinterpret_cast<const uint32_t *>(&pr);
        }
        sums.add(e, p[0], p[1], p[2], p[3]);
      }
      sums.end(h, c == 0 ? fix : 1.0f);
      ptx::tmem_st_32x32b_x16(s_tmem + (c + h) * 16, packed);
    }
  }
}

/* The largest of `COLUMNS` scores of a row (as stored, before scaling). */
template <int COLUMNS> __device__ __forceinline__ float row_max(uint32_t s_tmem) {
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
  for (int c = 0; c < COLUMNS / 32; ++c) {
    uint32_t raw[32];
    ptx::tmem_ld_32x32b_x32(s_tmem + c * 32, raw);
    ptx::tmem_ld_wait_for(raw);
#pragma unroll
    for (int e = 0; e < 32; ++e)
      mx4[e & 3] = fmaxf(mx4[e & 3], __uint_as_float(raw[e]));
  }
  return fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
}

/* A tile on the diagonal of a causal block: the scores of the columns above
   `limit` become -inf where they lie, in tensor memory, so that the passes
   above need no second form. */
__device__ __forceinline__ void mask_scores(uint32_t s_tmem, int limit) {
#pragma unroll 1
  for (int c = 0; c < BKV / 32; ++c) {
    uint32_t raw[32];
    ptx::tmem_ld_32x32b_x32(s_tmem + c * 32, raw);
    ptx::tmem_ld_wait_for(raw);
    const int first_out = limit + 1 - c * 32;
#pragma unroll
    for (int e = 0; e < 32; ++e)
      if (e >= first_out)
        raw[e] = 0xff800000u;
    ptx::tmem_st_32x32b_x32(s_tmem + c * 32, raw);
  }
  ptx::tmem_st_wait();
}

#define GIVE_UP(code)                                                          \
  do {                                                                         \
    atomicCAS(&g_flash_status, 0, (code));                                    \
    *stop = 1;                                                                 \
  } while (0)

template <bool kBy64>
__global__ void __launch_bounds__(THREADS, 1)
flash_kernel(const __grid_constant__ CUtensorMap map_q,
              const __grid_constant__ CUtensorMap map_k,
              const __grid_constant__ CUtensorMap map_v,
              __nv_bfloat16 *__restrict__ out, int S, int pairs, float scale_log2,
              int causal) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sm_q = smem;
  uint8_t *sm_k = sm_q + NQ * TILE_BYTES;
  uint8_t *sm_v = sm_k + RING * TILE_BYTES;
  Bars *bars = reinterpret_cast<Bars *>(sm_v + RING * TILE_BYTES);

  const int warp = ptx::warp_index(), lane = threadIdx.x % 32;
  /* A head is `pairs` pairs of Q tiles and then single ones. Those come first where a
     later tile meets more keys, and last where they are what is left over. Of a head's
     pairs, and of the single tiles, the heavy ones come first. */
  const int lone = S / BQ - pairs * NQ, heads = gridDim.x / (pairs + lone);
  const int singles = heads * lone;
  int at = blockIdx.x, single = -1;
  if (causal && at < singles)
    single = at;
  else if (causal)
    at -= singles;
  else if (at >= heads * pairs)
    single = at - heads * pairs;
  const bool two = single < 0;
  const int head = two ? at / pairs : single % heads;
  const int q_base = two ? (pairs - 1 - at % pairs) * BQ * NQ
                         : (S / BQ - 1 - single / heads) * BQ;
  const int64_t head_row = (int64_t)head * S;
  /* KV tiles that Q tile 0 and Q tile 1 meet: n0 <= n1 <= n0 + 1, or n1 = 0. */
  const int n0 = causal ? q_base / BKV + 1 : S / BKV;
  const int n1 = !two ? 0 : causal ? (q_base + BQ) / BKV + 1 : S / BKV;
  const int n_max = max(n0, n1);

  if (threadIdx.x == 0) {
    ptx::mbar_init(&bars->q_full, 1);
    for (int s = 0; s < RING; ++s) {
      ptx::mbar_init(&bars->k_full[s], 1);
      ptx::mbar_init(&bars->k_free[s], 1);
      ptx::mbar_init(&bars->v_full[s], 1);
      ptx::mbar_init(&bars->v_free[s], 1);
    }
    for (int w = 0; w < NQ; ++w) {
      ptx::mbar_init(&bars->s_full[w], 1);
      ptx::mbar_init(&bars->p_full[w], 4);
      ptx::mbar_init(&bars->pv_done[w], 1);
    }
    bars->stop = 0;
    ptx::fence_proxy_async_smem();
    ptx::fence_barrier_init();
  }
  if (warp == 1)
    ptx::tmem_alloc(&bars->tmem_base, 512);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  volatile int *stop = &bars->stop;
  chain_release();
  /* Set up under the tail of the kernel before. Every warp waits for its end: the limits of
     the waits below are for this kernel's own work. */
  chain_wait();

  if (warp == 0) {
    /* ------------------------------------------------------------ loader */
    if (lane == 0) {
      ptx::tma_prefetch_desc(&map_q);
      ptx::tma_prefetch_desc(&map_k);
      ptx::tma_prefetch_desc(&map_v);
      const int q_tiles = two ? NQ : 1;
      ptx::mbar_expect_tx(&bars->q_full, q_tiles * TILE_BYTES);
      for (int w = 0; w < q_tiles; ++w)
        for (int h = 0; h < 2; ++h)
          ptx::tma_load_2d(sm_q + w * TILE_BYTES + h * (TILE_BYTES / 2), &map_q,
                           h * 64, (int)(head_row + q_base + w * BQ),
                           &bars->q_full);
      int k_issued = 0, v_issued = 0;
      for (int j = 0; j < n_max; ++j) {
        const int s = j % RING;
        const uint32_t ph = ((j / RING) & 1) ^ 1;
        const int row = (int)(head_row + j * BKV);
        if (!ptx::mbar_wait(&bars->k_free[s], ph, stop)) {
          GIVE_UP(F2_K_FREE);
          break;
        }
        ptx::mbar_expect_tx(&bars->k_full[s], TILE_BYTES);
        for (int h = 0; h < 2; ++h)
          ptx::tma_load_2d(sm_k + s * TILE_BYTES + h * (TILE_BYTES / 2), &map_k,
                           h * 64, row, &bars->k_full[s]);
        ++k_issued;
        if (!ptx::mbar_wait(&bars->v_free[s], ph, stop)) {
          GIVE_UP(F2_V_FREE);
          break;
        }
        ptx::mbar_expect_tx(&bars->v_full[s], TILE_BYTES);
        for (int h = 0; h < 2; ++h)
          ptx::tma_load_2d(sm_v + s * TILE_BYTES + h * (TILE_BYTES / 2), &map_v,
                           h * 64, row, &bars->v_full[s]);
        ++v_issued;
      }
      /* Stay until every copy this thread started has landed. */
      ptx::mbar_wait_alone(&bars->q_full, 0);
      for (int back = 0; back < RING && back < k_issued; ++back) {
        const int j = k_issued - 1 - back;
        ptx::mbar_wait_alone(&bars->k_full[j % RING], (j / RING) & 1);
      }
      for (int back = 0; back < RING && back < v_issued; ++back) {
        const int j = v_issued - 1 - back;
        ptx::mbar_wait_alone(&bars->v_full[j % RING], (j / RING) & 1);
      }
    }
  } else if (warp == 1) {
    /* -------------------------------------------------------- MMA issuer */
    {
      const uint32_t idesc_s = ptx::idesc_f16(true, false, false, BQ, BKV);
      const uint32_t idesc_o = ptx::idesc_f16(true, false, true, BQ, HD);
      bool ok = ptx::mbar_wait_warp(&bars->q_full, 0, stop);
      if (!ok)
        GIVE_UP(F2_Q);
      ptx::tc_fence_after_sync();
      /* Descriptors of the tiles' first K step; a step adds to the address
         field (16-byte units), which cannot carry out of its 14 bits. */
      const uint64_t q_desc[NQ] = {
          ptx::smem_desc_sw128(ptx::smem_addr(sm_q), 16, 1024),
          ptx::smem_desc_sw128(ptx::smem_addr(sm_q + TILE_BYTES), 16, 1024)};
      const uint64_t k_desc[RING] = {
          ptx::smem_desc_sw128(ptx::smem_addr(sm_k), 16, 1024),
          ptx::smem_desc_sw128(ptx::smem_addr(sm_k + TILE_BYTES), 16, 1024)};
      const uint64_t v_desc[RING] = {
          ptx::smem_desc_sw128(ptx::smem_addr(sm_v), TILE_BYTES / 2, 1024),
          ptx::smem_desc_sw128(ptx::smem_addr(sm_v + TILE_BYTES), TILE_BYTES / 2,
                               1024)};
      /* S_w(j) = Q_w K_j^T into the score columns of Q tile w. `wait`: this is
         the first use of K_j; `release`: the last. */
      auto scores = [&](int w, int j, bool wait, bool release) -> bool {
        const int s = j & (RING - 1);
        if (wait && !ptx::mbar_wait_warp(&bars->k_full[s], (j / RING) & 1, stop)) {
          GIVE_UP(F2_K_FULL);
          return false;
        }
        if (wait)
          ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
          const uint64_t qd = w ? q_desc[1] : q_desc[0];
          const uint64_t kd = s ? k_desc[1] : k_desc[0];
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) {
            const uint32_t off = ((kk / 4) * (TILE_BYTES / 2) + (kk % 4) * 32) >> 4;
            ptx::umma_f16_ss(tmem + w * 256, qd + off, kd + off, idesc_s, kk != 0);
          }
          ptx::umma_commit(&bars->s_full[w]);
          if (release)
            ptx::umma_commit(&bars->k_free[s]);
        }
        __syncwarp();
        return true;
      };
      /* O_w += P_w(j) V_j. A = P from tensor memory: 16 bf16 of a row are 8
         columns. B = V, N-major: two 64-column blocks 16 KiB apart, 8-row
         groups 1 KiB apart; a K step is 16 KV rows = 2 KiB. */
      /* `k_next`: the scores that follow use K tile j + 1 for the first time;
         its barrier is polled together with the two this product needs, so
         that the three round trips to the barriers overlap. */
      auto weighted = [&](int w, int j, bool wait, bool release,
                          bool k_next) -> bool {
        const int s = j & (RING - 1);
        const int sk = (j + 1) & (RING - 1);
        const bool p_in = __all_sync(~0u, ptx::mbar_try_wait(&bars->p_full[w], j & 1));
        const bool v_in =
            !wait || __all_sync(~0u, ptx::mbar_try_wait(&bars->v_full[s], (j / RING) & 1));
        const bool k_in =
            !k_next ||
            __all_sync(~0u, ptx::mbar_try_wait(&bars->k_full[sk], ((j + 1) / RING) & 1));
        if (!v_in && !ptx::mbar_wait_warp(&bars->v_full[s], (j / RING) & 1, stop)) {
          GIVE_UP(F2_V_FULL);
          return false;
        }
        if (!p_in && !ptx::mbar_wait_warp(&bars->p_full[w], j & 1, stop)) {
          GIVE_UP(F2_P_FULL);
          return false;
        }
        if (!k_in && !ptx::mbar_wait_warp(&bars->k_full[sk], ((j + 1) / RING) & 1, stop)) {
          GIVE_UP(F2_K_FULL);
          return false;
        }
        ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
          const uint64_t vd = s ? v_desc[1] : v_desc[0];
#pragma unroll
          for (int kk = 0; kk < BKV / 16; ++kk)
            ptx::umma_f16_ts(tmem + w * 256 + 128, tmem + w * 256 + kk * 8,
                             vd + kk * (2048 >> 4), idesc_o, (j | kk) != 0);
          ptx::umma_commit(&bars->pv_done[w]);
          if (release)
            ptx::umma_commit(&bars->v_free[s]);
        }
        __syncwarp();
        return true;
      };
      /* Tile 0 leads, tile 1 follows; each P V is followed at once by the next
         scores of the same Q tile, so that its softmax runs under the other
         tile's products. Tile 1 is the last user of every K and V tile, and
         the first user of the one tile 0 does not meet. A CTA of one Q tile
         has no tile 1. */
      ok = ok && scores(0, 0, true, !two) && (!two || scores(1, 0, false, true));
      for (int j = 0; ok && j < n_max; ++j) {
        if (j < n0) {
          ok = weighted(0, j, true, !two, j + 1 < n0);
          if (ok && j + 1 < n0)
            ok = scores(0, j + 1, false, !two); /* K polled with the product */
        }
        if (!two)
          continue;
        const bool k_first = j + 1 < n1 && j + 1 >= n0;
        ok = ok && weighted(1, j, j >= n0, true, k_first);
        if (ok && j + 1 < n1)
          ok = scores(1, j + 1, false, true);
      }
    }
  } else {
    /* ------------------------------------------------ softmax warpgroups
       Four warps per Q tile, one thread per query row. */
    const int w = (warp - 2) / 4;  /* which Q tile */
    const int quarter = warp & 3;  /* TMEM lanes this warp may touch */
    const int row = quarter * 32 + lane;
    const int q_row = q_base + w * BQ + row;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_tmem = tmem + lane_base + w * 256; /* P goes over it */
    const uint32_t o_tmem = s_tmem + 128;
    const int n_mine = w ? n1 : n0;
    /* scores of unit-variance inputs stay within 2^8 of zero: start from a
       maximum of zero and let the check below catch what does not */
    float m_used = kBy64 ? -INFINITY : 0.0f, l_sum = 0.0f;
    HalfSums halves;
    bool ok = true;

    for (int j = 0; ok && j < n_mine; ++j) {
      if (!ptx::mbar_wait(&bars->s_full[w], j & 1, stop)) {
        GIVE_UP(F2_S_FULL);
        ok = false;
        break;
      }
      ptx::tc_fence_after_sync();
      const int limit = q_row - j * BKV; /* causal: columns above it are out */
      const bool diagonal = causal && j * BKV + BKV - 1 > q_base + w * BQ;
      uint32_t packed[BKV / 2];
      float rel_max = 0.0f, sum = 0.0f;
      if (diagonal)
        mask_scores(s_tmem, limit);
      /* First guess: the maximum in use still holds, so one pass over the
         scores gives P, its row sum and, on the side, the row maximum. If
         some row of this warp outgrew its maximum by more than 2^8 (or this
         is the first tile), take the maximum first, rescale what has been
         accumulated, and make the pass again: the scores are still in tensor
         memory, P has not been stored yet. (Written as a loop over two
         attempts, the compiler kept P live across the back edge and spilled:
         586 instead of 925 TFLOP/s.) */
      bool redo;
      const HalfSums before = halves;
      if (kBy64) {
        if (j == 0) {
          const float mx = row_max<64>(s_tmem) * scale_log2;
          m_used = mx > m_used ? mx : m_used;
        }
        probabilities_by64(s_tmem, scale_log2, -m_used, packed, rel_max, halves);
        /* a little below 8: what has grown is decided from the scores */
        redo = __any_sync(0xffffffffu, rel_max > 7.99f);
      } else {
        probabilities(s_tmem, scale_log2, -m_used, packed, rel_max, sum);
        redo = __any_sync(0xffffffffu, rel_max > 8.0f || (j == 0 && rel_max < -8.0f));
      }
      if (redo) {
        float m_new = m_used;
        if (kBy64) {
          const float m0 = row_max<64>(s_tmem) * scale_log2;
          const float m1 = row_max<64>(s_tmem + 64) * scale_log2;
          m_new = m0 > m_new + 8.0f ? m0 : m_new;
          m_new = m1 > m_new + 8.0f ? m1 : m_new;
        } else {
          const float mx = row_max<BKV>(s_tmem) * scale_log2;
          m_new = mx > m_used + 8.0f || (j == 0 && mx < m_used - 8.0f) ? mx : m_used;
        }
        const float fix = m_new != m_used ? ex2(m_used - m_new) : 1.0f;
        if (j > 0) {
          if (!ptx::mbar_wait(&bars->pv_done[w], (j - 1) & 1, stop)) {
            GIVE_UP(F2_PV_DONE);
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
#pragma unroll 1
          for (int c = 0; c < HD / 32; ++c) {
            uint32_t o[32];
            ptx::tmem_ld_32x32b_x32(o_tmem + c * 32, o);
            ptx::tmem_ld_wait_for(o);
#pragma unroll
            for (int e = 0; e < 32; ++e)
              o[e] = __float_as_uint(__uint_as_float(o[e]) * fix);
            ptx::tmem_st_32x32b_x32(o_tmem + c * 32, o);
          }
          ptx::tmem_st_wait();
        }
        m_used = m_new;
        if (kBy64) {
          halves = before;
          probabilities_by64_stored(s_tmem, scale_log2, -m_used, fix, halves);
        } else {
          l_sum *= fix;
          sum = probabilities_stored(s_tmem, scale_log2, -m_used);
        }
      } else {
        /* P, two bf16 per column, over the first half of the score columns. */
        ptx::tmem_st_32x32b_x32(s_tmem,
                                *reinterpret_cast<uint32_t(*)[32]>(&packed[0]));
        ptx::tmem_st_32x32b_x32(s_tmem + 32,
                                *reinterpret_cast<uint32_t(*)[32]>(&packed[32]));
      }
      l_sum += sum;
      ptx::tmem_st_wait();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->p_full[w]);
    }

    if (ok && n_mine > 0) {
      if (!ptx::mbar_wait(&bars->pv_done[w], (n_mine - 1) & 1, stop)) {
        GIVE_UP(F2_PV_DONE);
      } else {
        ptx::tc_fence_after_sync();
        const float inv = 1.0f / (kBy64 ? halves.l[0] + halves.l[1] : l_sum);
        __nv_bfloat16 *dst = out + ((int64_t)head_row + q_row) * HD;
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          ptx::tmem_ld_32x32b_x32(o_tmem + c * 32, o);
          ptx::tmem_ld_wait_for(o);
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t pk[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __nv_bfloat162 pr = __floats2bfloat162_rn(
                  __uint_as_float(o[q4 * 8 + 2 * e]) * inv,
                  __uint_as_float(o[q4 * 8 + 2 * e + 1]) * inv);
              pk[e] = *reinterpret_cast<const uint32_t *>(&pr);
            }
            *reinterpret_cast<uint4 *>(dst + c * 32 + q4 * 8) =
                make_uint4(pk[0], pk[1], pk[2], pk[3]);
          }
        }
      }
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, 512);
  }
}

} // namespace

/* q, k, v, out [B*H*S, 128] bf16. */
const char *flash_attention_fwd(const void *q, const void *k, const void *v,
                                void *out, int B, int H, int S, int D,
                                float scale, bool causal, cudaStream_t stream) {
  if (D != HD)
    return "flash attention is built for head_dim 128";
  if (B <= 0 || H <= 0 || S <= 0)
    return nullptr;
  if (S % BQ != 0)
    return "the sequence length must be a multiple of 128";
  if ((int64_t)B * H > 65535)
    return "more than 65535 (batch, head) pairs";
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)out) & 15)
    return "q, k, v and out must be 16-byte aligned";
  const int64_t rows = (int64_t)B * H * S;
  CUtensorMap mq, mk, mv;
  if (!make_map_16(&mq, q, HD, rows, HD, 64, BQ, true) ||
      !make_map_16(&mk, k, HD, rows, HD, 64, BKV, true) ||
      !make_map_16(&mv, v, HD, rows, HD, 64, BKV, true))
    return "cuTensorMapEncodeTiled refused q, k or v";
  auto kernel = S % (BQ * NQ) ? flash_kernel<true> : flash_kernel<false>;
  if (allow_dynamic_smem((const void *)kernel, SMEM_BYTES) != cudaSuccess)
    return "flash attention could not get its shared memory";
  /* Of an odd number of tiles the last is alone; all are where each finds an SM of its
     own: [1, 8, 640, 128] without a mask 14.4 us, 17.9 in pairs. */
  const int64_t tiles = S / BQ;
  const int pairs = tiles % 2 && B * H * tiles <= sm_count() ? 0 : (int)(tiles / 2);
  const int64_t blocks = (int64_t)B * H * (tiles - pairs);
  if (blocks > INT32_MAX)
    return "flash attention is asked for too many tiles";
  const dim3 grid((unsigned)blocks);
  const cudaError_t e =
      launch_chained(kernel, grid, dim3(THREADS), SMEM_BYTES, stream, mq, mk, mv,
                     (__nv_bfloat16 *)out, S, pairs, scale * 1.4426950408889634f,
                     causal ? 1 : 0);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

int flash_status(cudaStream_t stream) {
  int v = 0, zero = 0;
  if (cudaStreamSynchronize(stream) != cudaSuccess)
    return -1;
  if (cudaMemcpyFromSymbol(&v, g_flash_status, sizeof v) != cudaSuccess)
    return -1;
  if (v)
    cudaMemcpyToSymbol(g_flash_status, &zero, sizeof zero);
  return v;
}

} // namespace vxb
