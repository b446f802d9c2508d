/* gemm_f32_tile.cu -- C = A B in f32 on the tensor cores, in one launch.
 *
 * An f32 value is the exact sum of three bf16 terms (8 + 8 + 8 mantissa bits,
 * the remainders are exact in f32), so
 *   a b = a1 b1 + (a1 b2 + a2 b1) + (a2 b2 + a1 b3 + a3 b1) + (below 2^-24 |a b|)
 * with every product exact in f32.  The terms are made inside the kernel: sixteen
 * warps read a 128 x 64 tile of A and a 64 x 128 tile of B from global memory
 * (any stride, any alignment, any edge: what lies outside is zero), split them and
 * write the terms into two stages of 128-byte-swizzled shared memory; one thread
 * issues the products.  B is used as stored (an N-major operand), so that b1 and b2
 * lie side by side and a1 [b1 | b2] is one instruction of N = 256.
 *
 * The tensor core's own f32 sums lose a little with their length, so a1 b1 has an
 * accumulator of its own (the others are 2^-8 of it), and after kSegment blocks of
 * K the accumulators are added, in f32, to sums in registers.
 *
 * A cluster of Z blocks shares a tile, each a run of K; the runs' sums meet through
 * distributed shared memory in run order, so the result does not depend on timing,
 * and no scratch is needed.
 *
 * Both operands are multiplied by 2^24 before they are split, which is exact, so that the
 * smallest f32 value has three normal terms; the sums are multiplied by 2^-48.  (Without
 * it a softmax weight below 2^-109 would lose its third term.)  Values that are then too
 * large -- infinities, NaN, magnitudes whose products could overflow, from 2^34 on for
 * 1024 of K -- are noticed while they are read; a block that met one computes its run with
 * plain f32 multiply-adds as well, as gemm_f32 (gemm_simt.cu) would.  The price of one such
 * value, which the slowest block pays: 257 x 300 x 190 takes 21 us instead of 14, 1000^3 97
 * instead of 27 (on the FP32 pipe alone 31 and 118).
 */
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "plain_tile.cuh"
#include "ptx.cuh"

#include <cuda_bf16.h>

#include <cmath>

namespace vxb {
namespace {

constexpr int BM = 128, BN = 128, BK = 64, UK = 16;
constexpr int STAGES = 2;
constexpr int TERM_BYTES = BM * BK * 2; /* 16 KiB: one term of A or of B */
constexpr int STAGE_BYTES = 6 * TERM_BYTES;
constexpr int LOADERS = 512; /* threads that read, split and, at the end, add up */
constexpr int THREADS = LOADERS + 32;
constexpr int PITCH = BN + 4; /* floats between rows of the block's own sums */
/* Blocks of K between two transfers to registers. The tensor core cuts its sums off
   where an f32 addition rounds them: values of one sign lose 2.2e-8 a K step of 16. With
   eight blocks 1500 x 1300 x 1000 of values in [0, 1) was 7.0e-7 off, on the FP32 pipe
   4.2e-7; with two it is 1.4e-7, and 1024^3 takes 25.3 us instead of 25.2. */
constexpr int kSegment = 2;
constexpr float kUp = 0x1p24f, kDown = 0x1p-48f; /* of an operand, of a sum */

enum { T_EMPTY = 0x81, T_FULL, T_DONE, T_DRAINED };
__device__ int g_tile_status; /* first wait that ran out since the last read */

struct Bars {
  uint64_t full[STAGES], empty[STAGES];
  uint64_t done, drained[2]; /* drained: one for each set of accumulators */
  uint32_t tmem_base;
  int stop;
  int plain; /* a value was met that the split cannot carry */
};
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + (int)sizeof(Bars) + 64;
static_assert((BM * PITCH + kPlainFloats) * 4 <= STAGES * STAGE_BYTES,
              "the sums and the plain product reuse the stages");
static_assert(LOADERS == kPlainThreads && BM == 128 && BN == 128, "plain_tile");

/* Eight values, 2^24 of each, as three words of four bf16 pairs; most: the largest
   magnitude met, as a bit pattern. */
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ void split8(const float (&v)[8], uint8_t *at, uint32_t &most) {
  uint32_t w[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = v[2 * j] * kUp, y = v[2 * j + 1] * kUp;
    most = max(most, max(__float_as_uint(x) & 0x7fffffffu, __float_as_uint(y) & 0x7fffffffu));
    const uint32_t p1 = pack(x, y);
    const float rx = x - __uint_as_float(p1 << 16);
    const float ry = y - __uint_as_float(p1 & 0xffff0000u);
    const uint32_t p2 = pack(rx, ry);
    w[0][j] = p1;
    w[1][j] = p2;
    w[2][j] = pack(rx - __uint_as_float(p2 << 16), ry - __uint_as_float(p2 & 0xffff0000u));
  }
#pragma unroll
  for (int t = 0; t < 3; ++t)
    *reinterpret_cast<uint4 *>(at + t * TERM_BYTES) =
        make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
}

struct TileGemm {
  const float *a, *b;
  float *c;
  int64_t lda, ldb, ldc;
  int m, n, k, z; /* z: blocks that share a tile */
  int vec_a, vec_b, vec_c;
  uint32_t too_large; /* bits of the first magnitude, times 2^24, whose products could
                         overflow in a sum of k */
};

__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tile_kernel(const TileGemm g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Bars *bars = reinterpret_cast<Bars *>(smem + STAGES * STAGE_BYTES);
  const int tid = threadIdx.x, warp = ptx::warp_index(), lane = tid % 32;
  const int rank = g.z > 1 ? (int)ptx::cluster_ctarank() : 0;
  const int row0 = blockIdx.y * BM, col0 = (int)(blockIdx.x / g.z) * BN;
  /* this block's run of the blocks of K */
  const int k_blocks = (g.k + BK - 1) / BK;
  const int kb0 = (int)((int64_t)rank * k_blocks / g.z);
  const int kb1 = (int)((int64_t)(rank + 1) * k_blocks / g.z);

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&bars->full[s], LOADERS / 32);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    ptx::mbar_init(&bars->done, 1);
    for (int a = 0; a < 2; ++a)
      ptx::mbar_init(&bars->drained[a], LOADERS / 32);
    bars->stop = 0;
    bars->plain = 0;
    ptx::fence_barrier_init();
  }
  if (warp == LOADERS / 32)
    ptx::tmem_alloc(&bars->tmem_base, 512);
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  const uint32_t tmem = bars->tmem_base;
  volatile int *stop = &bars->stop;
  chain_release();
  chain_wait(); /* set up under the tail of the kernel before */

  /* the sums of a loader thread: row 32 (warp % 4) + lane of the tile, 32 columns */
  float acc[32];
#pragma unroll
  for (int i = 0; i < 32; ++i)
    acc[i] = 0.0f;

  if (warp < LOADERS / 32) {
    /* a thread's share of the tiles: two runs of eight values of each. A: rows of
       64 values, eight lanes a row; B: rows of 128 values, sixteen lanes a row */
    const int ar = tid >> 3, ac = (tid & 7) * 8;
    const int br = tid >> 4, bc = (tid & 15) * 8;
    uint8_t *const a_at = smem + ar * 128 + (((tid & 7) ^ (ar & 7)) << 4);
    uint8_t *const b_at = smem + 3 * TERM_BYTES + ((tid & 15) >> 3) * (64 * BK * 2) +
                          br * 128 + (((tid & 7) ^ (br & 7)) << 4);
    float va[2][8], vb[2][8];
    auto read_a = [&](int kb) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = row0 + ar + 64 * i;
        read8(va[i], g.a + (int64_t)r * g.lda, kb * BK + ac, g.k, r < g.m, g.vec_a);
      }
    };
    auto read_b = [&](int kb) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = kb * BK + br + 32 * i;
        read8(vb[i], g.b + (int64_t)r * g.ldb, col0 + bc, g.n, r < g.k, g.vec_b);
      }
    };
    /* the sums of segment `seg` from tensor memory to registers */
    auto drain = [&](int seg) -> bool {
      if (!ptx::mbar_wait(&bars->done, seg & 1, stop)) {
        atomicCAS(&g_tile_status, 0, T_DONE);
        *stop = 1;
        return false;
      }
      ptx::tc_fence_after_sync();
      const uint32_t at = tmem + (seg & 1) * 256 + ((uint32_t)((warp & 3) * 32) << 16) +
                          (warp >> 2) * 32;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t v[8], w[8];
        ptx::tmem_ld_32x32b_x8(at + q * 8, v);
        ptx::tmem_ld_32x32b_x8(at + BN + q * 8, w);
        ptx::tmem_ld_wait_for(v);
        ptx::tmem_ld_wait_for(w);
#pragma unroll
        for (int e = 0; e < 8; ++e)
          acc[q * 8 + e] += __uint_as_float(v[e]) + __uint_as_float(w[e]);
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->drained[seg & 1]);
      return true;
    };
    uint32_t most = 0;
    if (kb0 < kb1) {
      read_a(kb0);
      read_b(kb0);
    }
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, s = it % STAGES;
      /* the segment before is taken over one block into this one, while the tensor
         core is busy, and in any case before this one's last block goes out: the
         barrier tells two segments apart, not three */
      if (it >= kSegment &&
          (it % kSegment == 1 || (it % kSegment == 0 && kb + 1 == kb1)) &&
          !drain(it / kSegment - 1)) {
        ok = false;
        break;
      }
      if (!ptx::mbar_wait(&bars->empty[s], ((it / STAGES) & 1) ^ 1, stop)) {
        atomicCAS(&g_tile_status, 0, T_EMPTY);
        *stop = 1;
        ok = false;
        break;
      }
      /* each half's next values are asked for as soon as its registers are free */
#pragma unroll
      for (int i = 0; i < 2; ++i) /* 64 rows further: the swizzle is the same */
        split8(va[i], a_at + s * STAGE_BYTES + i * 64 * 128, most);
      if (kb + 1 < kb1)
        read_a(kb + 1);
#pragma unroll
      for (int i = 0; i < 2; ++i)
        split8(vb[i], b_at + s * STAGE_BYTES + i * 32 * 128, most);
      if (kb + 1 < kb1)
        read_b(kb + 1);
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->full[s]);
    }
    if (ok && kb0 < kb1)
      drain((kb1 - kb0 - 1) / kSegment);
    if (most >= g.too_large)
      bars->plain = 1;
  } else {
    const uint32_t wide = ptx::idesc_f16(true, false, true, BM, 2 * BN);
    const uint32_t narrow = ptx::idesc_f16(true, false, true, BM, BN);
    for (int kb = kb0; kb < kb1; ++kb) {
      const int it = kb - kb0, s = it % STAGES;
      const int seg = it / kSegment;
      const bool first = it % kSegment == 0;
      /* Two sets of accumulators alternate. Each has a barrier of its own: this warp may
         come here so late that the segment before has been drained as well, and a shared
         one would then be two phases on, which its parity does not tell from none. This
         set's next phase is this segment's, so it cannot run ahead. */
      if (first && seg > 1 &&
          !ptx::mbar_wait_warp(&bars->drained[seg & 1], ((seg >> 1) - 1) & 1, stop)) {
        atomicCAS(&g_tile_status, 0, T_DRAINED);
        *stop = 1;
        break;
      }
      if (!ptx::mbar_wait_warp(&bars->full[s], (it / STAGES) & 1, stop)) {
        atomicCAS(&g_tile_status, 0, T_FULL);
        *stop = 1;
        break;
      }
      ptx::tc_fence_after_sync();
      const uint32_t sa = ptx::smem_addr(smem + s * STAGE_BYTES);
      const uint32_t sb = sa + 3 * TERM_BYTES;
      const uint32_t sum = tmem + (seg & 1) * 256, rest = sum + BN;
      if (ptx::elect_one()) {
#pragma unroll
        for (int kk = 0; kk < BK / UK; ++kk) {
          const uint64_t a1 = ptx::smem_desc_sw128(sa + kk * UK * 2, 16, 1024);
          const uint64_t b1 = ptx::smem_desc_sw128(sb + kk * UK * 128, 64 * BK * 2, 1024);
          const uint64_t term = TERM_BYTES >> 4; /* in the address field's units */
          ptx::umma_f16_ss(sum, a1, b1, wide, !first || kk != 0); /* a1 b1 | a1 b2 */
          ptx::umma_f16_ss(rest, a1 + term, b1, narrow, 1);
          ptx::umma_f16_ss(rest, a1 + term, b1 + term, narrow, 1);
          ptx::umma_f16_ss(rest, a1, b1 + 2 * term, narrow, 1);
          ptx::umma_f16_ss(rest, a1 + 2 * term, b1, narrow, 1);
        }
        ptx::umma_commit(&bars->empty[s]);
        if ((it + 1) % kSegment == 0 || kb + 1 == kb1)
          ptx::umma_commit(&bars->done);
      }
      __syncwarp();
    }
  }

  /* the products are done with the stages (every loader waited for the last of
     them); the block's sums go where the stages were */
  __syncthreads();
  float *sums = reinterpret_cast<float *>(smem);
  if (bars->plain && warp < LOADERS / 32) {
    const PlainTile t{g.a, g.b, g.lda, g.ldb, g.m, g.n, g.vec_a, g.vec_b};
    plain_tile(t, row0, col0, kb0 * BK, min(kb1 * BK, g.k), tid, sums + BM * PITCH, acc);
    const int ty = tid / 32, tx = tid % 32;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<float4 *>(sums + (ty * 8 + i) * PITCH + tx * 4) =
          make_float4(acc[i * 4], acc[i * 4 + 1], acc[i * 4 + 2], acc[i * 4 + 3]);
  } else if (warp < LOADERS / 32) {
    float *mine = sums + ((warp & 3) * 32 + lane) * PITCH + (warp >> 2) * 32;
#pragma unroll
    for (int j = 0; j < 32; j += 4)
      *reinterpret_cast<float4 *>(mine + j) =
          make_float4(acc[j] * kDown, acc[j + 1] * kDown, acc[j + 2] * kDown,
                      acc[j + 3] * kDown);
  }
  if (g.z > 1)
    ptx::cluster_sync_all();
  else
    __syncthreads();

  /* this block's share of the tile's rows: the runs' sums in run order */
  if (warp < LOADERS / 32) {
    const int rows = BM / g.z, first_row = rank * rows;
    const uint32_t base = ptx::smem_addr(sums);
    for (int r = first_row + warp; r < first_row + rows; r += LOADERS / 32) {
      if (row0 + r >= g.m)
        break;
      float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (g.vec_c) {
        for (int q = 0; q < g.z; ++q) {
          float4 v;
          const uint32_t from = base + (r * PITCH + lane * 4) * 4;
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                       : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                       : "r"(g.z > 1 ? ptx::map_to_cta(from, q) : from)
                       : "memory");
          s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        float *dst = g.c + (int64_t)(row0 + r) * g.ldc + col0 + lane * 4;
        if (col0 + lane * 4 + 4 <= g.n) {
          *reinterpret_cast<float4 *>(dst) = s;
        } else {
          const float e[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (col0 + lane * 4 + j < g.n)
              dst[j] = e[j];
        }
      } else {
        /* neighbouring lanes, neighbouring columns: C's rows may begin anywhere */
        float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int q = 0; q < g.z; ++q)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float v;
            const uint32_t from = base + (r * PITCH + lane + 32 * j) * 4;
            asm volatile("ld.shared::cluster.f32 %0, [%1];"
                         : "=f"(v)
                         : "r"(g.z > 1 ? ptx::map_to_cta(from, q) : from)
                         : "memory");
            e[j] += v;
          }
        float *dst = g.c + (int64_t)(row0 + r) * g.ldc + col0 + lane;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col0 + lane + 32 * j < g.n)
            dst[32 * j] = e[j];
      }
    }
  }
  /* nobody leaves while another block of the cluster may still read its sums */
  if (g.z > 1)
    ptx::cluster_sync_all();
  else
    __syncthreads();
  if (warp == LOADERS / 32) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, 512);
  }
}

constexpr int64_t kMostRowTiles = 65535; /* in a grid's second dimension */

/* How many clusters of z blocks the GPU holds at once: they do not divide the SMs of a
   GPC. */
int64_t clusters_at_once(int z) {
  if (allow_dynamic_smem((const void *)gemm_f32_tile_kernel, SMEM_BYTES) == cudaSuccess) {
    const int n = resident_clusters((const void *)gemm_f32_tile_kernel, z, THREADS, SMEM_BYTES);
    if (n > 0)
      return n;
  }
  return sm_count() / z > 1 ? sm_count() / z : 1;
}

/* How many blocks share a tile: more while the chip has room for them, each keeps a block
   of K, and all are resident at once; but for that last wish none gets so much of K that
   the tensor core's sums grow longer (128 of K). 768^3 as 36 clusters of four, of which
   not all are resident: 26.9 us; of two 18.3. */
int blocks_of_tile(int64_t m, int64_t n, int64_t k) {
  const int64_t tiles = ((m + BM - 1) / BM) * ((n + BN - 1) / BN);
  const int64_t k_blocks = (k + BK - 1) / BK;
  int z = 1;
  while (z < 8 && tiles * z * 2 <= sm_count() && k_blocks >= 2 * z &&
         (k_blocks < 3 * z || tiles <= clusters_at_once(2 * z)))
    z *= 2;
  return z;
}

} // namespace

/* Microseconds, about: 1.7 for a block of K of a tile (96 KiB of terms written to shared
   memory and 176 KiB read from it, and sixteen warps splitting) and 7.4 for a tile's start
   and end, as many rounds as the tiles need. Measured 24.6 / 51.4 / 126 / 365 / 65.6 / 38.8
   at 1024^3, 1536^3, 2048^3, 3072^3, 2944 x 2944 x 320, 128 x 128 x 8192, where this gives
   24.6 / 51.8 / 127 / 360 / 67 / 38.2. (A call by itself, of which 3.4 go under the tail
   of the call before where there is one.) */
double gemm_f32_tile_us(int64_t m, int64_t n, int64_t k) {
  if ((m + BM - 1) / BM > kMostRowTiles)
    return HUGE_VAL;
  const int64_t z = blocks_of_tile(m, n, k);
  const int64_t tiles = ((m + BM - 1) / BM) * ((n + BN - 1) / BN);
  const int64_t at_once = z > 1 ? clusters_at_once((int)z) : sm_count();
  const int64_t k_blocks = ((k + BK - 1) / BK + z - 1) / z;
  return 3.6 + (double)((tiles + at_once - 1) / at_once) * (7.4 + 1.7 * k_blocks);
}

const char *gemm_f32_tile(const float *a, int64_t lda, const float *b, int64_t ldb,
                          float *c, int64_t ldc, int64_t m, int64_t n, int64_t k,
                          cudaStream_t stream) {
  if (m <= 0 || n <= 0)
    return nullptr;
  if (m > INT32_MAX - BM || n > INT32_MAX - BN || k > INT32_MAX - BK)
    return "a dimension does not fit in 32 bits";
  if ((m + BM - 1) / BM > kMostRowTiles)
    return "more than 65535 row tiles";
  TileGemm g{};
  g.a = a; g.b = b; g.c = c;
  g.lda = lda; g.ldb = ldb; g.ldc = ldc;
  g.m = (int)m; g.n = (int)n; g.k = (int)k;
  auto vec = [](const void *p, int64_t ld) {
    return ((uintptr_t)p & 15) == 0 && ld % 4 == 0 ? 4
           : ((uintptr_t)p & 7) == 0 && ld % 2 == 0 ? 2 : 1;
  };
  g.vec_a = vec(a, lda);
  g.vec_b = vec(b, ldb);
  g.vec_c = vec(c, ldc) == 4;
  /* k products of two such values, as their terms add up to them, stay below 2^127 */
  int log2_k = 0;
  while (((int64_t)1 << log2_k) < k)
    ++log2_k;
  g.too_large = (uint32_t)(127 + (126 - log2_k) / 2) << 23;
  const int z = blocks_of_tile(m, n, k);
  g.z = z;
  if (allow_dynamic_smem((const void *)gemm_f32_tile_kernel, SMEM_BYTES) != cudaSuccess)
    return "the f32 GEMM could not get its shared memory";
  const dim3 grid((unsigned)((n + BN - 1) / BN * z), (unsigned)((m + BM - 1) / BM));
  const cudaError_t e =
      z > 1 ? launch_chained_cluster_smem(gemm_f32_tile_kernel, grid, dim3(THREADS), z,
                                          SMEM_BYTES, stream, g)
            : launch_chained(gemm_f32_tile_kernel, grid, dim3(THREADS), SMEM_BYTES, stream, g);
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

int gemm_f32_tile_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_tile_status, sizeof v) != cudaSuccess)
    return -1;
  if (v)
    cudaMemcpyToSymbol(g_tile_status, &zero, sizeof zero);
  return v;
}

} // namespace vxb
