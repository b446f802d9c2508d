/* gemm_f32_small.cu -- C = A B in f32 where there is little of it, on the FP32 pipe.
 *
 * The tensor-core kernel of gemm_f32_tile.cu splits every value into three terms and has
 * tiles of 128 x 128: nine of them for 257 x 300 x 190, which took 13.4 us, most of it a
 * tile's start and end.  Here a tile is 32 x 32, so that the same product has 90 blocks, and
 * a block's eight warps share it: two take the halves of its rows, four such pairs a quarter
 * of every 128 of K each, with a lane's 4 x 4 results in registers (eight loads from shared
 * memory for 64 multiply-adds), and the pairs' sums meet in shared memory at the end.  Where
 * there are few tiles, K is divided over a cluster of up to eight blocks as well, whose sums
 * meet through distributed shared memory in run order.
 * A and B come by cp.async into three stages of 128 of K.
 *
 * Four products are added in f32, two such sums, and those sums with what an addition rounds
 * off kept beside the sum: all of it where the sum so far is the larger, all but 2^-24 of the
 * eight products where they are (with 16 products in a row it was 9.8e-8 from 64 bits
 * at 257 x 300 x 190, where the terms are 9.3e-8; so 5.7e-8, and 2e-8 to 3e-8 for values of
 * one sign, where the terms are 7e-8 to 1.5e-7).  Groups of warps and blocks add up in 64
 * bits.  B is multiplied by 2^24, which keeps products below the smallest f32; a tile in
 * which something became infinite is made once more as the values are.
 *
 * What bounds it: of few tiles the trips to memory and the launch, of many the FP32 pipe,
 * 1.7 us for 128 of K of each tile of an SM.  In a graph, us, the terms' kernel in
 * brackets: 64^3 4.1 (5.8), 257 x 300 x 190 8.8 (10.5), 64 x 64 x 2048 7.7 (12.9), 512 x 512
 * x 128 6.9 (8.3), 512^3 17.1 (18.3); 1024 x 1024 x 512 would take 54 (13.9).
 */
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "ptx.cuh"

#include <cooperative_groups.h>

#include <cmath>
#include <cstdint>

namespace vxb {
namespace {

constexpr int TILE = 32, KC = 128, STAGES = 3, WARPS = 8, THREADS = WARPS * 32;
constexpr int PITCH_A = KC + 4; /* floats: four rows apart by one land in four banks */
constexpr int A_FLOATS = TILE * PITCH_A, B_FLOATS = KC * TILE;
constexpr int SMEM_BYTES = STAGES * (A_FLOATS + B_FLOATS) * 4;
constexpr int K_GROUPS = 4; /* of warps: two take the halves of a tile's rows */
static_assert((K_GROUPS + 1) * TILE * TILE * 2 <= STAGES * (A_FLOATS + B_FLOATS), "the sums");

struct SmallGemm {
  const float *a, *b;
  float *c;
  int64_t lda, ldb, ldc;
  int m, n, k, z;
  int run;          /* of K a block, a multiple of 4 */
  int vec_c;
};

/* V floats from src to shared memory, of which `bytes` are there and the rest zeros. */
template <int V> __device__ __forceinline__ void copy(uint32_t dst, const float *src, int bytes) {
  if (V == 4)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src),
                 "n"(V * 4), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(d)
      : "l"(*reinterpret_cast<const unsigned long long *>(&a)),
        "l"(*reinterpret_cast<const unsigned long long *>(&b)));
  return *reinterpret_cast<float2 *>(&d);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long d;
  const float2 one = make_float2(-1.0f, -1.0f);
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<const unsigned long long *>(&b)),
        "l"(*reinterpret_cast<const unsigned long long *>(&one)),
        "l"(*reinterpret_cast<const unsigned long long *>(&a)));
  return *reinterpret_cast<float2 *>(&d);
}
/* sum + x, and what its rounding takes off is added to `rest` (Dekker's sum of two: exact
   where x is the smaller; else t - sum may round, by at most 2^-24 of x. The form that is
   exact for any order takes three more operations, and the products in x have lost as much
   by then). */
__device__ __forceinline__ void add_with_rest(float2 &sum, float2 &rest, const float2 x) {
  const float2 t = add2(sum, x);
  rest = add2(rest, sub2(x, sub2(t, sum)));
  sum = t;
}
__device__ __forceinline__ float4 times(const float4 v, float f) {
  return make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
}
/* (an infinity's rest is not a number) */
__device__ __forceinline__ double whole(float sum, float rest) {
  return isfinite(sum) ? (double)sum + (double)rest : (double)sum;
}

/* VA, VB: how many floats of a row the rows' alignment lets a copy take. */
template <int VA, int VB>
__global__ void __launch_bounds__(THREADS, 2) gemm_f32_small_kernel(const SmallGemm g) {
  extern __shared__ __align__(16) float room[];
  __shared__ int any_large;
  namespace cg = cooperative_groups;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int rank = blockIdx.x % g.z;
  const int row0 = blockIdx.y * TILE, col0 = blockIdx.x / g.z * TILE;
  const int k0 = min(g.k, rank * g.run), k1 = min(g.k, k0 + g.run);
  const int chunks = (k1 - k0 + KC - 1) / KC;
  chain_release();
  chain_wait();

  auto fetch = [&](int chunk) {
    if (chunk < chunks) {
      const int k = k0 + chunk * KC;
      float *sa = room + chunk % STAGES * (A_FLOATS + B_FLOATS), *sb = sa + A_FLOATS;
      const uint32_t at_a = ptx::smem_addr(sa), at_b = ptx::smem_addr(sb);
#pragma unroll
      for (int i = 0; i < TILE * KC / VA / THREADS; ++i) {
        const int at = threadIdx.x + i * THREADS;
        const int r = at / (KC / VA), c = at % (KC / VA) * VA;
        const int left = row0 + r < g.m ? min(max(k1 - k - c, 0), VA) : 0;
        copy<VA>(at_a + (r * PITCH_A + c) * 4,
                 left ? g.a + (row0 + r) * g.lda + k + c : g.a, left * 4);
      }
#pragma unroll
      for (int i = 0; i < KC * TILE / VB / THREADS; ++i) {
        const int at = threadIdx.x + i * THREADS;
        const int r = at / (TILE / VB), c = at % (TILE / VB) * VB;
        const int left = k + r < k1 ? min(max(g.n - col0 - c, 0), VB) : 0;
        copy<VB>(at_b + (r * TILE + c) * 4,
                 left ? g.b + (int64_t)(k + r) * g.ldb + col0 + c : g.b, left * 4);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  /* rows first + 4 i, columns 4 cq .. of a quarter of each 128 of K */
  const int first = warp % 2 * (TILE / 2) + lane / 8, cq = lane % 8, group = warp / 2;
  cg::cluster_group cluster = cg::this_cluster();
  /* Everything times 2^24, so that products below the smallest f32 are not lost before
     they are added; and once more as it is where that made something too large. */
  float up = 0x1p24f;
again:
  float2 sum[4][2] = {}, rest[4][2] = {};
  for (int s = 0; s < STAGES - 1; ++s)
    fetch(s);
  for (int chunk = 0; chunk < chunks; ++chunk) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads(); /* this chunk is here, and the one before has been read */
    fetch(chunk + STAGES - 1);
    const float *sa = room + chunk % STAGES * (A_FLOATS + B_FLOATS), *sb = sa + A_FLOATS;
    sa += first * PITCH_A + group * (KC / K_GROUPS);
    sb += group * (KC / K_GROUPS) * TILE + cq * 4;
#pragma unroll 1
    for (int k = 0; k < KC / K_GROUPS; k += 8) {
      float2 eight[4][2]; /* the sum of two sums of four products */
#pragma unroll
      for (int o = 0; o < 8; o += 4) {
        float4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          b[j] = times(*reinterpret_cast<const float4 *>(sb + (k + o + j) * TILE), up);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 a = *reinterpret_cast<const float4 *>(sa + 4 * i * PITCH_A + k + o);
          const float av[4] = {a.x, a.y, a.z, a.w};
          float2 four[2] = {make_float2(a.x * b[0].x, a.x * b[0].y),
                            make_float2(a.x * b[0].z, a.x * b[0].w)};
#pragma unroll
          for (int j = 1; j < 4; ++j) {
            four[0].x = fmaf(av[j], b[j].x, four[0].x);
            four[0].y = fmaf(av[j], b[j].y, four[0].y);
            four[1].x = fmaf(av[j], b[j].z, four[1].x);
            four[1].y = fmaf(av[j], b[j].w, four[1].y);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)
            eight[i][h] = o ? add2(eight[i][h], four[h]) : four[h];
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          add_with_rest(sum[i][h], rest[i][h], eight[i][h]);
    }
  }

  /* ---- the groups' sums, then the runs', in 64 bits ---- */
  __syncthreads();
  double2 *pairs = reinterpret_cast<double2 *>(room);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      pairs[(group * TILE + first + 4 * i) * (TILE / 2) + cq * 2 + h] =
          make_double2(whole(sum[i][h].x, rest[i][h].x), whole(sum[i][h].y, rest[i][h].y));
  __syncthreads();
  auto add = [](double2 &x, const double2 y) {
    x.x += y.x;
    x.y += y.y;
  };
  auto store = [&](int pair, const double2 v) {
    const int row = row0 + pair / (TILE / 2), col = col0 + pair % (TILE / 2) * 2;
    if (row >= g.m)
      return;
    float *dst = g.c + row * g.ldc + col;
    if (g.vec_c && col + 2 <= g.n) {
      *reinterpret_cast<float2 *>(dst) = make_float2((float)v.x, (float)v.y);
    } else {
      if (col < g.n)
        dst[0] = (float)v.x;
      if (col + 1 < g.n)
        dst[1] = (float)v.y;
    }
  };
  constexpr int PAIRS = TILE * TILE / 2;
  double2 *mine = pairs + K_GROUPS * PAIRS;
  int large = 0;
  for (int p = threadIdx.x; p < PAIRS; p += THREADS) {
    double2 total = pairs[p];
#pragma unroll
    for (int w = 1; w < K_GROUPS; ++w) /* fixed order */
      add(total, pairs[w * PAIRS + p]);
    large |= !isfinite(total.x) || !isfinite(total.y);
    mine[p] = total;
  }
  large = __syncthreads_or(large);
  if (g.z > 1) {
    if (threadIdx.x == 0)
      any_large = large;
    cluster.sync();
    for (int r = 0; r < g.z; ++r)
      large |= *cluster.map_shared_rank(&any_large, r);
  }
  if (large && up != 1.0f) {
    up = 1.0f;
    if (g.z > 1)
      cluster.sync(); /* the others have read this block's word */
    goto again;
  }
  const double down = 1.0 / up;
  const int share = PAIRS / g.z;
  for (int p = rank * share + threadIdx.x; p < (rank + 1) * share; p += THREADS) {
    double2 total = mine[p];
    if (g.z > 1) {
      total = *cluster.map_shared_rank(mine + p, 0);
      for (int r = 1; r < g.z; ++r) /* fixed order */
        add(total, *cluster.map_shared_rank(mine + p, r));
    }
    store(p, make_double2(total.x * down, total.y * down));
  }
  if (g.z > 1)
    cluster.sync(); /* nobody leaves while another may still read its sums */
}

int runs_of(int64_t m, int64_t n, int64_t k) {
  const int64_t tiles = ((m + TILE - 1) / TILE) * ((n + TILE - 1) / TILE);
  int z = 1;
  while (z < 8 && tiles * z * 2 <= sm_count() && k >= 2 * KC * z)
    z *= 2;
  return z;
}

} // namespace

/* Microseconds, about, one call after another: 1.73 for 128 of K of each tile that an SM has,
   3.2 for a launch, 1.5 for the meeting of a cluster, 0.9 for each tile an SM has after its
   first two. From half as many blocks as SMs on, some SM has two: blocks begin beside those of
   the call before, on what SMs that leaves. Measured 4.1 / 5.9 / 8.7 / 8.8 / 6.9 / 17.1 / 14.2 /
   32.0 at 64^3, 64 x 64 x 1024, 320 x 320 x 256, 257 x 300 x 190, 512 x 512 x 128, 512^3,
   576 x 576 x 256 and 768 x 768 x 512, where this gives 4.9 / 6.4 / 10.1 / 10.1 / 6.7 / 17.0 /
   14.5 / 32.7. */
double gemm_f32_small_us(int64_t m, int64_t n, int64_t k) {
  if (m > 65535ll * TILE || n > INT32_MAX - TILE || k > INT32_MAX - 4 * KC)
    return HUGE_VAL;
  const int64_t z = runs_of(m, n, k);
  const int64_t blocks = ((m + TILE - 1) / TILE) * ((n + TILE - 1) / TILE) * z;
  const int64_t chunks = ((k + z - 1) / z + KC - 1) / KC;
  const int64_t rounds = (blocks + sm_count() - 1) / sm_count();
  const int64_t on_an_sm = 2 * blocks <= sm_count() ? 1 : rounds < 2 ? 2 : rounds;
  return 3.2 + (z > 1 ? 1.5 : 0.0) + 1.73 * (double)(on_an_sm * chunks) +
         (on_an_sm > 2 ? 0.9 * (double)(on_an_sm - 2) : 0.0);
}

const char *gemm_f32_small(const float *a, int64_t lda, const float *b, int64_t ldb, float *c,
                           int64_t ldc, int64_t m, int64_t n, int64_t k, cudaStream_t stream) {
  if (m <= 0 || n <= 0)
    return nullptr;
  if (m > 65535ll * TILE || n > INT32_MAX - TILE || k > INT32_MAX - 4 * KC)
    return "a dimension is too large for the small f32 product";
  SmallGemm g{};
  g.a = a; g.b = b; g.c = c;
  g.lda = lda; g.ldb = ldb; g.ldc = ldc;
  g.m = (int)m; g.n = (int)n; g.k = (int)k;
  g.z = runs_of(m, n, k);
  g.run = (int)(((k + g.z - 1) / g.z + 3) / 4 * 4);
  auto vec = [](const void *p, int64_t ld) {
    return ((uintptr_t)p & 15) == 0 && ld % 4 == 0 ? 4
           : ((uintptr_t)p & 7) == 0 && ld % 2 == 0 ? 2 : 1;
  };
  g.vec_c = vec(c, ldc) >= 2;
  auto go = [&](auto kernel) -> const char * {
    if (allow_dynamic_smem((const void *)kernel, SMEM_BYTES) != cudaSuccess)
      return "the small f32 product could not get its shared memory";
    const dim3 grid((unsigned)((n + TILE - 1) / TILE * g.z), (unsigned)((m + TILE - 1) / TILE));
    const cudaError_t e =
        g.z > 1 ? launch_chained_cluster_smem(kernel, grid, dim3(THREADS), g.z, SMEM_BYTES,
                                              stream, g)
                : launch_chained(kernel, grid, dim3(THREADS), SMEM_BYTES, stream, g);
    return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
  };
  auto of_b = [&](auto va) -> const char * {
    constexpr int VA = decltype(va)::value;
    const int vb = vec(b, ldb);
    return vb == 4   ? go(gemm_f32_small_kernel<VA, 4>)
           : vb == 2 ? go(gemm_f32_small_kernel<VA, 2>)
                     : go(gemm_f32_small_kernel<VA, 1>);
  };
  const int va = vec(a, lda);
  return va == 4   ? of_b(std::integral_constant<int, 4>())
         : va == 2 ? of_b(std::integral_constant<int, 2>())
                   : of_b(std::integral_constant<int, 1>());
}

} // namespace vxb
