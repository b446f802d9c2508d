/* gemm_f32_split.cu -- C = A B in f32 on the tensor cores.
 *
 * The reference sends an f32 matmul to cuBLAS Sgemm (cuda_dispatch.cpp:988-1023),
 * which runs on the FP32 pipe. A B200 has twenty times more bf16 tensor
 * throughput than FP32, and an f32 value is the exact sum of three bf16 terms
 * (8 + 8 + 8 mantissa bits, the remainders are exact in f32), so
 *   a b = (a1 + a2 + a3)(b1 + b2 + b3)
 *       = a1 b1 + a1 b2 + a2 b1 + a1 b3 + a2 b2 + a3 b1 + (terms below 2^-24 |a b|)
 * with every product bf16 x bf16 exact in f32 and the sums in f32. Laid out
 * as ONE bf16 GEMM over K' = 6 k:
 *   A' [m, 6k] = a3 | a2 | a1 | a2 | a1 | a1
 *   B' [n, 6k] = b1 | b2 | b3 | b1 | b2 | b1      (B transposed on the way)
 * (of each run of K by itself, one run after another) -- the small products first: the tensor core cuts its sum off at every K step of 16, by
 * up to 2^-24 of what the sum then is, so only the k / 16 steps of a1 b1 count.  With a1 b1
 * first 3072^3 in one run was 3.4e-5 off (2.0e-5 of values in [0, 1)), so it is 2.9e-6
 * (8.9e-6).  It runs on the CTA-pair kernel of the prefill (tcgen05.mma.cta_group::2,
 * f32 partial sums per run of K', added in run order).
 *
 * The range is that of gemm_f32_tile.cu: both operands times 2^24, the sums times 2^-48,
 * and a flag for each 128 rows of A and 128 columns of B in which a value was met that is
 * too large then (infinities and NaN among them).  A last launch computes the tiles of
 * flagged rows and columns with plain multiply-adds; where there is none it adds 1.4
 * to 3 us (3072 x 3072 x 1024: 103.7 -> 105.1, 3072 x 3072 x 64: 30.0 -> 33.0).
 */
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "plain_tile.cuh"

#include <cuda_bf16.h>

#include <algorithm>

namespace vxb {
namespace {

constexpr float kUp = 0x1p24f, kDown = 0x1p-48f; /* of an operand, of a sum */
constexpr int TILE = 128; /* rows, or columns, behind a flag */
/* Where values too large for the terms were met. split_bt leaves a word for each of its
   blocks and clears the rows' words; split_a, after it, sets those and gathers the others. */
struct Flags {
  int *rows, *columns; /* for each TILE of them */
  int *blocks;         /* [down][across]: of 32 x 32 values of B */
  int row_tiles, down, across;
};
__device__ __forceinline__ uint32_t magnitude(float x) {
  return __float_as_uint(x) & 0x7fffffffu;
}
/* bits of the first magnitude, times 2^24, whose products could overflow: k products of
   two such values, as their terms add up to them, stay below 2^127 */
uint32_t too_large(int64_t k) {
  int log2_k = 0;
  while (((int64_t)1 << log2_k) < k)
    ++log2_k;
  return (uint32_t)(127 + (126 - log2_k) / 2) << 23;
}

__device__ __forceinline__ void three_terms(float v, __nv_bfloat16 &t1,
                                            __nv_bfloat16 &t2, __nv_bfloat16 &t3) {
  t1 = __float2bfloat16(v);
  const float r1 = v - __bfloat162float(t1);
  t2 = __float2bfloat16(r1);
  t3 = __float2bfloat16(r1 - __bfloat162float(t2));
}

/* Where the terms of a block of 64 of K lie: the first is block `first` of K', the next one
   is `step` further. Run r of `runs` has the blocks r * blocks / runs .. of K. */
struct Place {
  int64_t first;
  int step;
};
template <typename Int> __device__ __forceinline__ Place place_in(int block, int blocks, int runs) {
  const int r = (int)(((Int)(block + 1) * runs - 1) / blocks);
  const int begin = (int)((Int)r * blocks / runs);
  const int end = (int)((Int)(r + 1) * blocks / runs);
  return Place{6 * (int64_t)begin + (block - begin), end - begin};
}
__device__ __forceinline__ Place place_of(int block, int blocks, int runs) {
  if (runs == 1)
    return Place{block, blocks};
  /* three 64-bit divisions cost a thread as much as the rest of its work */
  return (uint64_t)(blocks + 1) * runs < (1ull << 32) ? place_in<uint32_t>(block, blocks, runs)
                                                     : place_in<uint64_t>(block, blocks, runs);
}

/* A' from A: one thread per eight consecutive values of a row (k is a
   multiple of 64), six 16-byte stores. The last blocks gather the flags that split_bt's
   blocks left, one block for each 128 columns. */
__global__ void __launch_bounds__(256)
split_a_kernel(__nv_bfloat16 *out, const float *a, int64_t lda, int m, int k,
               int runs, uint32_t limit, const Flags f) {
  chain_release();
  chain_wait();
  const int gatherers = (f.across + 3) / 4;
  const int column = (int)blockIdx.x - (int)gridDim.x + gatherers;
  if (column >= 0) {
    int any = 0;
    for (int i = threadIdx.x; i < 4 * f.down; i += blockDim.x)
      if (4 * column + i % 4 < f.across)
        any |= f.blocks[i / 4 * f.across + 4 * column + i % 4];
    any = __syncthreads_or(any);
    if (threadIdx.x == 0)
      f.columns[column] = any;
    return;
  }
  const int per_row = k / 8;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)m * per_row)
    return;
  const int64_t r = idx / per_row;
  const int c = (int)(idx - r * per_row) * 8;
  const float *src = a + r * lda + c;
  uint32_t w1[4], w2[4], w3[4], most = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __nv_bfloat16 x1, x2, x3, y1, y2, y3;
    const float x = src[2 * j] * kUp, y = src[2 * j + 1] * kUp;
    most = max(most, max(magnitude(x), magnitude(y)));
    three_terms(x, x1, x2, x3);
    three_terms(y, y1, y2, y3);
    w1[j] = (uint32_t)__bfloat16_as_ushort(x1) | (uint32_t)__bfloat16_as_ushort(y1) << 16;
    w2[j] = (uint32_t)__bfloat16_as_ushort(x2) | (uint32_t)__bfloat16_as_ushort(y2) << 16;
    w3[j] = (uint32_t)__bfloat16_as_ushort(x3) | (uint32_t)__bfloat16_as_ushort(y3) << 16;
  }
  const uint4 t1 = make_uint4(w1[0], w1[1], w1[2], w1[3]);
  const uint4 t2 = make_uint4(w2[0], w2[1], w2[2], w2[3]);
  const uint4 t3 = make_uint4(w3[0], w3[1], w3[2], w3[3]);
  if (most >= limit)
    f.rows[r / TILE] = 1;
  const Place at = place_of(c / 64, k / 64, runs);
  const int64_t step = (int64_t)at.step * 64;
  __nv_bfloat16 *row = out + r * 6 * k + at.first * 64 + c % 64;
  *reinterpret_cast<uint4 *>(row) = t3;
  *reinterpret_cast<uint4 *>(row + step) = t2;
  *reinterpret_cast<uint4 *>(row + 2 * step) = t1;
  *reinterpret_cast<uint4 *>(row + 3 * step) = t2;
  *reinterpret_cast<uint4 *>(row + 4 * step) = t1;
  *reinterpret_cast<uint4 *>(row + 5 * step) = t1;
}

/* B' from B [k, n]: a block transposes a 32 x 32 tile through shared memory,
   so that B is read along n and B' written along k. */
__global__ void __launch_bounds__(256)
split_bt_kernel(__nv_bfloat16 *out, const float *b, int64_t ldb, int k, int n,
                int runs, uint32_t limit, const Flags f) {
  __shared__ __nv_bfloat16 tile[3][32][34];
  chain_release();
  chain_wait();
  const int k0 = blockIdx.y * 32, n0 = blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5; /* 32 x 8 */
  int large = 0;
  for (int r = ty; r < 32; r += 8) {
    __nv_bfloat16 t1, t2, t3;
    const float v =
        (k0 + r < k && n0 + tx < n) ? b[(int64_t)(k0 + r) * ldb + n0 + tx] * kUp : 0.0f;
    large |= magnitude(v) >= limit;
    three_terms(v, t1, t2, t3);
    tile[0][r][tx] = t1;
    tile[1][r][tx] = t2;
    tile[2][r][tx] = t3;
  }
  large = __syncthreads_or(large);
  if (threadIdx.x == 0)
    f.blocks[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = large;
  for (int64_t i = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
       i < f.row_tiles; i += (int64_t)gridDim.x * gridDim.y * blockDim.x)
    f.rows[i] = 0;
  const Place at = place_of(k0 / 64, k / 64, runs); /* 32 of K are of one block */
  const int64_t step = (int64_t)at.step * 64;
  for (int j = ty; j < 32; j += 8) {
    if (n0 + j >= n || k0 + tx >= k)
      continue;
    __nv_bfloat16 *row = out + (int64_t)(n0 + j) * 6 * k + at.first * 64 + k0 % 64 + tx;
    const __nv_bfloat16 t1 = tile[0][tx][j], t2 = tile[1][tx][j], t3 = tile[2][tx][j];
    row[0] = t1;
    row[step] = t2;
    row[2 * step] = t3;
    row[3 * step] = t1;
    row[4 * step] = t2;
    row[5 * step] = t1;
  }
}

/* C = the runs' partial sums, in run order; four values per thread (n is a
   multiple of 4). vec: C's rows are 16-byte aligned. */
__global__ void __launch_bounds__(256)
sum_runs_kernel(float *c, int64_t ldc, const float *partials, int splits, int m,
                int n, int vec) {
  chain_release();
  chain_wait();
  const int per_row = n / 4;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)m * per_row)
    return;
  const int64_t r = idx / per_row;
  const int j = (int)(idx - r * per_row) * 4;
  const int64_t at = r * n + j;
  float4 s = *reinterpret_cast<const float4 *>(partials + at);
  for (int q = 1; q < splits; ++q) {
    const float4 v =
        *reinterpret_cast<const float4 *>(partials + (int64_t)q * m * n + at);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  float *dst = c + r * ldc + j;
  if (vec) {
    *reinterpret_cast<float4 *>(dst) = s;
  } else {
    dst[0] = s.x; dst[1] = s.y; dst[2] = s.z; dst[3] = s.w;
  }
}

/* The tiles whose rows or columns are flagged, again, with plain multiply-adds. */
__global__ void __launch_bounds__(kPlainThreads, 1)
plain_tiles_kernel(const PlainTile g, float *c, int64_t ldc, int k, const int *row_flags,
                   const int *column_flags) {
  extern __shared__ __align__(16) float room[];
  chain_release();
  chain_wait();
  const int row_tiles = (g.m + TILE - 1) / TILE, column_tiles = (g.n + TILE - 1) / TILE;
  for (int64_t t = blockIdx.x; t < (int64_t)row_tiles * column_tiles; t += gridDim.x) {
    const int tm = (int)(t / column_tiles), tn = (int)(t - (int64_t)tm * column_tiles);
    if (!row_flags[tm] && !column_flags[tn])
      continue;
    float acc[32];
    plain_tile(g, tm * TILE, tn * TILE, 0, k, threadIdx.x, room, acc);
    const int row = tm * TILE + threadIdx.x / 32 * 8, col = tn * TILE + threadIdx.x % 32 * 4;
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (row + i / 4 < g.m && col + i % 4 < g.n)
        c[(int64_t)(row + i / 4) * ldc + col + i % 4] = acc[i];
    __syncthreads(); /* the next tile's first stage may be this one's last */
  }
}

size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }
Flags flags_of(void *at, int64_t m, int64_t n, int64_t k) {
  Flags f;
  f.row_tiles = (int)((m + TILE - 1) / TILE);
  f.down = (int)((k + 31) / 32);
  f.across = (int)((n + 31) / 32);
  f.rows = (int *)at;
  f.columns = f.rows + f.row_tiles;
  f.blocks = f.columns + (n + TILE - 1) / TILE;
  return f;
}
size_t flag_bytes(int64_t m, int64_t n, int64_t k) {
  const Flags f = flags_of(nullptr, m, n, k);
  return up256((size_t)(f.row_tiles + (n + TILE - 1) / TILE + (int64_t)f.down * f.across) *
               sizeof(int));
}

bool direct(int splits, int64_t n, int64_t ldc) { return splits == 1 && ldc == n; }

/* How many runs the K blocks are cut into: the number, up to 12, that leaves the
   last wave of pairs fullest. Many short runs rather than the fewest that are as
   fast: the tensor core's own f32 sums lose a little with their length, and none is
   longer than 12288 of K: 768 cuts of up to 2^-24 are 4.6e-5, where the reference's
   check of a product allows 1e-4. */
int runs_of(int64_t m, int64_t n, int64_t k) {
  const int tiles = (int)(((m + 255) / 256) * ((n + 255) / 256));
  const int blocks = (int)(k / 64), pairs = 74;
  const int least = (int)((k + 12287) / 12288);
  int best = least;
  double best_fill = 0.0;
  for (int s = least; s <= std::max(12, least) && s <= blocks; ++s) {
    const int items = tiles * s;
    const double fill = (double)items / (((items + pairs - 1) / pairs) * pairs);
    if (fill > best_fill + 0.02) {
      best_fill = fill;
      best = s;
    }
  }
  return best;
}

} // namespace

/* Microseconds, about: the six products at 1.5 PFLOP/s, or 0.34 for a block of K' of each
   pair's items where there are few, the terms (12 bytes a value) and the runs' partial sums
   (8) written and read, five launches. Measured 154 / 105 / 290 / 40.6 at 2048^3, 3072 x
   3072 x 1024, 3072^3 and 128 x 128 x 8192, where this gives 174 / 110 / 295 / 45. */
double gemm_f32_split_us(int64_t m, int64_t n, int64_t k, int64_t ldc) {
  const int64_t runs = runs_of(m, n, k), pairs = 74;
  const int64_t items = (m + 255) / 256 * ((n + 255) / 256) * runs;
  const double sums = direct((int)runs, n, ldc) ? 0.0 : 8.0e-6 * runs * m * n / 4.0;
  const double longest =
      0.34 * (double)((items + pairs - 1) / pairs * ((6 * k / 64 + runs - 1) / runs));
  return 18.0 + std::max(12.0e-9 * m * n * k / 1.5, longest) + 24.0e-6 * (m + n) * k / 10.0 +
         sums;
}

size_t gemm_f32_split_scratch_bytes(int64_t m, int64_t n, int64_t k, int64_t ldc) {
  /* n % 4: the GEMM stores its f32 results four at a time */
  if (k % 64 != 0 || n % 4 != 0 || m < 128 || n < 128 || m > (1 << 30) || n > (1 << 30) ||
      6 * k > (1ll << 31) - 1 || m * n * k < (1ll << 24))
    return 0;
  const int splits = runs_of(m, n, k);
  size_t bytes = flag_bytes(m, n, k) + up256((size_t)(m + n) * 6 * k * 2);
  if (!direct(splits, n, ldc))
    bytes += (size_t)splits * m * n * 4;
  return bytes;
}

const char *gemm_f32_split(const float *a, int64_t lda, const float *b, int64_t ldb,
                           float *c, int64_t ldc, int64_t m, int64_t n, int64_t k,
                           void *scratch, cudaStream_t stream) {
  if (!gemm_f32_split_scratch_bytes(m, n, k, ldc) || !scratch)
    return "the shape is not for the tensor-core f32 product";
  const Flags f = flags_of(scratch, m, n, k);
  __nv_bfloat16 *a6 = (__nv_bfloat16 *)((char *)scratch + flag_bytes(m, n, k));
  __nv_bfloat16 *b6 = a6 + m * 6 * k;
  float *partials = (float *)((char *)a6 + up256((size_t)(m + n) * 6 * k * 2));
  const uint32_t limit = too_large(k);
  int splits = runs_of(m, n, k);
  launch_chained(split_bt_kernel, dim3((unsigned)f.across, (unsigned)f.down), dim3(256), 0,
                 stream, b6, b, ldb, (int)k, (int)n, splits, limit, f);
  launch_chained(split_a_kernel,
                 dim3((unsigned)((m * (k / 8) + 255) / 256 + (n + TILE - 1) / TILE)),
                 dim3(256), 0, stream, a6, a, lda, (int)m, (int)k, splits, limit, f);
  if (cudaGetLastError() != cudaSuccess)
    return "the term-splitting launches failed";
  float *out = direct(splits, n, ldc) ? c : partials;
  if (const char *why = rows_gemm_of(a6, 6 * k, b6, 6 * k, (int)m, (int)n, out, &splits,
                                     stream, splits, kDown, 6))
    return why;
  if (out != c) {
    const int vec = ldc % 4 == 0 && ((uintptr_t)c & 15) == 0;
    launch_chained(sum_runs_kernel, dim3((unsigned)((m * (n / 4) + 255) / 256)),
                   dim3(256), 0, stream, c, ldc, partials, splits, (int)m, (int)n, vec);
    if (cudaGetLastError() != cudaSuccess)
      return "the launch that adds the runs failed";
  }
  constexpr int room = kPlainFloats * 4;
  if (allow_dynamic_smem((const void *)plain_tiles_kernel, room) != cudaSuccess)
    return "the plain tiles could not get their shared memory";
  auto vec = [](const float *p, int64_t ld) {
    return ((uintptr_t)p & 15) == 0 && ld % 4 == 0 ? 4
           : ((uintptr_t)p & 7) == 0 && ld % 2 == 0 ? 2 : 1;
  };
  const int64_t tiles = ((m + TILE - 1) / TILE) * ((n + TILE - 1) / TILE);
  launch_chained(plain_tiles_kernel, dim3((unsigned)std::min<int64_t>(tiles, sm_count())),
                 dim3(kPlainThreads), room, stream,
                 PlainTile{a, b, lda, ldb, (int)m, (int)n, vec(a, lda), vec(b, ldb)}, c, ldc,
                 (int)k, (const int *)f.rows, (const int *)f.columns);
  if (cudaGetLastError() != cudaSuccess)
    return "the launch of the plain tiles failed";
  return nullptr;
}

} // namespace vxb
