/* gemm_umma.cu -- C[m,n] = A[m,k] * B[k,n] for bf16/f16 inputs on the sm_100a
 * tensor cores, f32 accumulation in tensor memory, output of the input type.
 *
 * This is the arithmetic of the reference's cublasGemmEx call for 16-bit
 * tensors (runtime/cuda_dispatch.cpp:1014-1022: CUBLAS_COMPUTE_32F, C of the
 * input type), on row-major operands as the dispatch plan describes them.
 *
 * One persistent CTA per SM, 192 threads, three roles:
 *   warp 0      one thread issues TMA loads of A (128x64) and B (64x256) tiles
 *               into a 4-deep ring of 128-byte-swizzled shared memory stages;
 *   warp 1      allocates the 512 TMEM columns; one thread issues
 *               tcgen05.mma (M=128, N=256, K=16, four per stage) and commits
 *               each stage back to the loader and each finished tile to the
 *               epilogue;
 *   warps 2-5   read a finished 128x256 f32 accumulator out of TMEM (each warp
 *               its own 32 lanes), round to the output type and store.
 * TMEM holds two accumulators, so the epilogue of tile i overlaps the MMAs of
 * tile i+1.  Tiles are visited in groups of 16 row-tiles so that the CTAs that
 * run together share A and B panels in L2.
 *
 * A is K-major as stored.  B, stored [k, n] with n contiguous, is given to the
 * tensor core as an N-major operand: four 64x64 TMA boxes per stage, leading
 * byte offset 8 KiB between 64-column blocks, stride byte offset 1 KiB between
 * 8-row groups.  (Route 2 instead transposes B first and uses a K-major B.)
 *
 * Edges: TMA zero-fills loads past m, n or k, and the epilogue guards its
 * stores, so any m, n, k work as long as the bases are 16-byte aligned and the
 * row strides are multiples of 8 elements.
 */
#include "gemm_store.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdlib>
#include <algorithm>
#include <mutex>
#include <type_traits>

namespace vxb {

bool tensor_maps_available();
bool make_map_16(CUtensorMap *map, const void *base, int64_t inner, int64_t rows,
                 int64_t ld, int box_inner, int box_rows, bool is_bf16);

const char *gemm_16_plain(bool is_bf16, const void *a, int64_t lda,
                          const void *b, int64_t ldb, void *c, int64_t ldc,
                          int64_t m, int64_t n, int64_t k, cudaStream_t stream);
/* gemm_umma_pair.cu: the same product on CTA pairs (256x256 tiles). */
const char *gemm_16_pair(int route, bool is_bf16, const void *a, int64_t lda,
                         const void *b, int64_t ldb, void *c, int64_t ldc,
                         int64_t m, int64_t n, int64_t k, cudaStream_t stream);
int gemm_pair_status();
int gemm_f32_tile_status(); /* gemm_f32_tile.cu */

namespace {

constexpr int BM = 128, BK = 64, UK = 16;
constexpr int A_BYTES = BM * BK * 2; /* 16 KiB */
/* Tiles of 256 columns, or of 128 where 256 would leave most SMs without one. */
template <int BN> struct Shape {
  static constexpr int stages = BN == 256 ? 4 : 6;
  static constexpr int b_bytes = BN * BK * 2;
  static constexpr int stage_bytes = A_BYTES + b_bytes;
  static constexpr int smem_bytes =
      stages * stage_bytes + 1024 /* align */ + 256 + 4 * kTurnWords * 4;
};
constexpr int THREADS = 192;
constexpr int GROUP_M = 16;

/* Where a wait ran out: role * 16 + which barrier. */
enum { ST_OK = 0, ST_LOADER_EMPTY = 0x11, ST_MMA_FULL = 0x21,
       ST_MMA_TMEM_EMPTY = 0x22, ST_EPI_TMEM_FULL = 0x31 };

__device__ int g_status; /* first failure of any CTA since the last read */

struct Barriers {
  uint64_t full[6];
  uint64_t empty[6];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int stop;
};

__device__ inline void tile_coords(int tile, int m_tiles, int n_tiles, int &tm,
                                   int &tn) {
  const int per_group = GROUP_M * n_tiles;
  const int group = tile / per_group;
  const int first = group * GROUP_M;
  const int rows = min(m_tiles - first, GROUP_M);
  const int in_group = tile - group * per_group;
  tm = first + in_group % rows;
  tn = in_group / rows;
}

/* Where the sums go: to C, rounded, or, with the blocks of K cut into several runs, to
   partials[run][m][pitch] as they are (finish16_kernel adds the runs up). */
template <typename T> struct Out {
  T *c;
  int64_t ldc;
  int vec;         /* C's rows are 16-byte aligned */
  int runs;        /* of the blocks of K */
  float *partials; /* runs > 1 */
  int64_t pitch;   /* a multiple of 8 */
};

/* kBNMajor: B tiles are [64 k][64 n] boxes (B as stored); otherwise B was
   transposed beforehand and tiles are [BN n][64 k]. */
template <typename T, bool kBNMajor, int BN>
__global__ void __launch_bounds__(THREADS, 1)
umma_gemm_kernel(const __grid_constant__ CUtensorMap map_a,
                 const __grid_constant__ CUtensorMap map_b, const Out<T> out, int m,
                 int n, int k) {
  constexpr int STAGES = Shape<BN>::stages, STAGE_BYTES = Shape<BN>::stage_bytes;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Barriers *bars = reinterpret_cast<Barriers *>(smem + STAGES * STAGE_BYTES);

  const int warp = ptx::warp_index(), lane = threadIdx.x % 32;
  const int m_tiles = (m + BM - 1) / BM, n_tiles = (n + BN - 1) / BN;
  const int items = m_tiles * n_tiles * out.runs;
  const int k_blocks = (k + BK - 1) / BK;
  /* item -> tile and the run's blocks of K: the runs of a tile are neighbours */
  auto first_block = [&](int item) {
    return (int)((int64_t)(item % out.runs) * k_blocks / out.runs);
  };
  auto end_block = [&](int item) {
    return (int)((int64_t)(item % out.runs + 1) * k_blocks / out.runs);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      ptx::mbar_init(&bars->full[s], 1);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      ptx::mbar_init(&bars->tmem_full[a], 1);
      ptx::mbar_init(&bars->tmem_empty[a], 4);
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
    /* ---------------------------------------------------------- loader */
    if (lane == 0) {
      ptx::tma_prefetch_desc(&map_a);
      ptx::tma_prefetch_desc(&map_b);
      int it = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        int tm, tn;
        tile_coords(item / out.runs, m_tiles, n_tiles, tm, tn);
        const int kb1 = end_block(item);
        for (int kb = first_block(item); kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t phase = (it / STAGES) & 1;
          if (!ptx::mbar_wait(&bars->empty[s], phase ^ 1, stop)) {
            atomicCAS(&g_status, 0, ST_LOADER_EMPTY);
            *stop = 1;
            ok = false;
            break;
          }
          uint8_t *sa = smem + s * STAGE_BYTES, *sb = sa + A_BYTES;
          ptx::mbar_expect_tx(&bars->full[s], STAGE_BYTES);
          ptx::tma_load_2d(sa, &map_a, kb * BK, tm * BM, &bars->full[s]);
          if (kBNMajor) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              ptx::tma_load_2d(sb + j * (64 * BK * 2), &map_b, tn * BN + j * 64,
                               kb * BK, &bars->full[s]);
          } else {
            ptx::tma_load_2d(sb, &map_b, kb * BK, tn * BN, &bars->full[s]);
          }
        }
      }
      /* Do not leave while a copy may still land in this CTA's memory. */
      for (int back = 0; back < STAGES && back < it; ++back) {
        const int j = it - 1 - back;
        ptx::mbar_wait_alone(&bars->full[j % STAGES], (j / STAGES) & 1);
      }
    }
  } else if (warp == 1) {
    /* ------------------------------------------------------ MMA issuer */
    {
      const uint32_t idesc =
          ptx::idesc_f16(sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value,
                         false, kBNMajor, BM, BN);
      int it = 0, t = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x, ++t) {
        const int acc = t & 1;
        const uint32_t acc_phase = (t >> 1) & 1;
        if (!ptx::mbar_wait_warp(&bars->tmem_empty[acc], acc_phase ^ 1, stop)) {
          atomicCAS(&g_status, 0, ST_MMA_TMEM_EMPTY);
          *stop = 1;
          break;
        }
        ptx::tc_fence_after_sync();
        const uint32_t d_tmem = tmem + acc * BN;
        const int kb0 = first_block(item), kb1 = end_block(item);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % STAGES;
          if (!ptx::mbar_wait_warp(&bars->full[s], (it / STAGES) & 1, stop)) {
            atomicCAS(&g_status, 0, ST_MMA_FULL);
            *stop = 1;
            ok = false;
            break;
          }
          ptx::tc_fence_after_sync();
          const uint32_t sa = ptx::smem_addr(smem + s * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
          if (ptx::elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / UK; ++kk) {
              /* A: K-major, rows of 128 bytes, 8-row groups 1 KiB apart; a K
                 step of 16 elements is 32 bytes along the row. */
              const uint64_t da = ptx::smem_desc_sw128(sa + kk * UK * 2, 16, 1024);
              /* B N-major: 64-column blocks 8 KiB apart (leading offset), 8-row
                 K groups 1 KiB apart (stride offset); a K step is 16 rows.
                 B K-major: as A. */
              const uint64_t db =
                  kBNMajor ? ptx::smem_desc_sw128(sb + kk * UK * 128, 64 * BK * 2,
                                                  1024)
                           : ptx::smem_desc_sw128(sb + kk * UK * 2, 16, 1024);
              ptx::umma_f16_ss(d_tmem, da, db, idesc, kb != kb0 || kk != 0);
            }
            ptx::umma_commit(&bars->empty[s]);
          }
          __syncwarp();
        }
        if (ok && ptx::elect_one())
          ptx::umma_commit(&bars->tmem_full[acc]);
        __syncwarp();
      }
    }
  } else {
    /* ---------------------------------------------------------- epilogue */
    const int quarter = warp & 3; /* the TMEM lanes this warp may read */
    uint32_t *turn = reinterpret_cast<uint32_t *>(smem + STAGES * STAGE_BYTES + 256) +
                     quarter * kTurnWords;
    int t = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x, ++t) {
      int tm, tn;
      tile_coords(item / out.runs, m_tiles, n_tiles, tm, tn);
      const int acc = t & 1;
      if (!ptx::mbar_wait(&bars->tmem_full[acc], (t >> 1) & 1, stop)) {
        atomicCAS(&g_status, 0, ST_EPI_TMEM_FULL);
        *stop = 1;
        break;
      }
      ptx::tc_fence_after_sync();
      const int row0 = tm * BM + quarter * 32;
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + acc * BN;
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(taddr + c * 32, v);
        ptx::tmem_ld_wait();
        const int col = tn * BN + c * 32;
        if (out.runs > 1) {
          if (row0 + lane < m) {
            float *dst = out.partials +
                         ((int64_t)(item % out.runs) * m + row0 + lane) * out.pitch + col;
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if (col + 4 * q < out.pitch)
                reinterpret_cast<uint4 *>(dst)[q] =
                    make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
          }
        } else if (row0 < m) {
          store_block<T>(v, out.c, out.ldc, row0, col, m, n, lane, out.vec, turn);
        }
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0)
        ptx::mbar_arrive(&bars->tmem_empty[acc]);
    }
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, 512);
  }
}

/* C = the runs' sums, added in run order and rounded; neighbouring threads, neighbouring
   columns. */
template <typename T>
__global__ void __launch_bounds__(256)
finish16_kernel(const Out<T> out, int m, int n) {
  chain_wait();
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t r = idx / out.pitch;
  const int c = (int)(idx - r * out.pitch);
  if (r >= m || c >= n)
    return;
  const float *at = out.partials + r * out.pitch + c;
  float s = at[0];
  for (int q = 1; q < out.runs; ++q)
    s += at[q * (int64_t)m * out.pitch];
  const uint32_t w = pack2<T>(s, 0.0f);
  reinterpret_cast<uint16_t *>(out.c)[r * out.ldc + c] = (uint16_t)w;
}

/* Matrices whose rows TMA cannot describe (a base off the 16-byte grid, a stride that is
   no multiple of 8), copied to rows of `pitch` elements, a multiple of 8: A, B or both in
   one launch. Eight elements a thread: whole words of the source, moved half a word where
   the row begins on an odd element, so that a row is read once in wide accesses (4096^2:
   33 us with two elements a thread). */
struct Pack16 {
  const uint16_t *src;
  uint4 *dst;
  int64_t ld;
  int rows, cols, groups; /* groups: of eight, in a row of dst */
  int blocks;
};
__global__ void __launch_bounds__(256)
pack16_kernel(const Pack16 first, const Pack16 second) {
  const bool one = (int)blockIdx.x < first.blocks;
  const Pack16 &p = one ? first : second;
  const int64_t idx =
      (int64_t)(blockIdx.x - (one ? 0 : first.blocks)) * blockDim.x + threadIdx.x;
  const int64_t r = idx / p.groups;
  const int c = (int)(idx - r * p.groups) * 8;
  if (r >= p.rows)
    return;
  const uint16_t *at = p.src + r * p.ld + c;
  uint32_t w[4];
  if (c + 8 <= p.cols) {
    if (((uintptr_t)at & 3) == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        w[j] = reinterpret_cast<const uint32_t *>(at)[j];
    } else {
      const uint32_t *in = reinterpret_cast<const uint32_t *>(at + 1);
      uint32_t low = at[0];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t next = j < 3 ? in[j] : (uint32_t)at[7];
        w[j] = low | next << 16;
        low = next >> 16;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      w[j] = (uint32_t)(c + 2 * j < p.cols ? at[2 * j] : 0) |
             (uint32_t)(c + 2 * j + 1 < p.cols ? at[2 * j + 1] : 0) << 16;
  }
  p.dst[idx] = make_uint4(w[0], w[1], w[2], w[3]);
}

/* ---- host side ------------------------------------------------------------- */
template <typename T, bool kBNMajor, int BN>
const char *launch_umma(const CUtensorMap &ma, const CUtensorMap &mb, const Out<T> &out,
                        int m, int n, int k, cudaStream_t stream) {
  auto kernel = umma_gemm_kernel<T, kBNMajor, BN>;
  constexpr int bytes = Shape<BN>::smem_bytes;
  if (allow_dynamic_smem((const void *)kernel, bytes) != cudaSuccess)
    return "the tcgen05 GEMM could not get its shared memory";
  const int64_t items =
      (int64_t)((m + BM - 1) / BM) * ((n + BN - 1) / BN) * out.runs;
  const int grid = (int)(items < sm_count() ? items : sm_count());
  launch_chained(kernel, dim3(grid), dim3(THREADS), bytes, stream, ma, mb, out, m, n, k);
  if (out.runs > 1)
    launch_chained(finish16_kernel<T>,
                   dim3((unsigned)(((int64_t)m * out.pitch + 255) / 256)), dim3(256), 0,
                   stream, out, m, n);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? nullptr : cudaGetErrorString(e);
}

bool rows_ok(const void *p, int64_t ld) { return ((uintptr_t)p & 15) == 0 && ld % 8 == 0; }
bool dims_ok(int64_t m, int64_t n, int64_t k) {
  return m < (1 << 30) && n < (1 << 30) && k < (1 << 30) && k >= 1;
}
bool umma_shape_ok(const void *a, int64_t lda, const void *b, int64_t ldb,
                   const void *c, int64_t ldc, int64_t m, int64_t n, int64_t k) {
  return rows_ok(a, lda) && rows_ok(b, ldb) && rows_ok(c, ldc) && dims_ok(m, n, k);
}

/* The one-CTA kernel with B as stored. */
template <typename T>
const char *run_umma(int bn, const void *a, int64_t lda, const void *b, int64_t ldb,
                     const Out<T> &out, int64_t m, int64_t n, int64_t k,
                     cudaStream_t stream) {
  constexpr bool bf16 = std::is_same<T, __nv_bfloat16>::value;
  CUtensorMap ma, mb;
  if (!make_map_16(&ma, a, k, m, lda, BK, BM, bf16))
    return "cuTensorMapEncodeTiled refused the A matrix";
  if (!make_map_16(&mb, b, n, k, ldb, 64, BK, bf16))
    return "cuTensorMapEncodeTiled refused the B matrix";
  return bn == 256
             ? launch_umma<T, true, 256>(ma, mb, out, (int)m, (int)n, (int)k, stream)
             : launch_umma<T, true, 128>(ma, mb, out, (int)m, (int)n, (int)k, stream);
}

/* How a 16-bit product of this size runs. */
struct Plan16 {
  bool pair; /* on CTA pairs, 256 x 256 */
  int bn;    /* else: columns of a one-CTA tile */
  int runs;  /* of the blocks of K, whose sums another kernel adds */
  double us; /* about */
};
int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
Plan16 plan_16(int64_t m, int64_t n, int64_t k, bool scratch) {
  const int sms = sm_count();
  const int64_t kb = ceil_div(k, BK);
  /* One CTA per 128x256 tile, or a CTA pair per 256x256 tile. The single CTA's
     MMA is held to 77 % of the tensor pipe by its operand fetch and the pair's
     runs near the full rate, so a pair finishes its tile (twice the work on
     two SMs) in about 0.82 of the time one CTA needs for its own; but there
     are half as many pair tiles, so for a small product the last wave decides,
     and below two waves of pair tiles the cluster's start-up shows (2048^3:
     823 against 912 TFLOP/s). */
  const int64_t t1 = ceil_div(m, 128) * ceil_div(n, 256);
  const int64_t t2 = ceil_div(m, 256) * ceil_div(n, 256);
  const double block = 0.42; /* microseconds of a block of K of a 128 x 256 tile */
  const double one = (double)(ceil_div(t1, sms) * kb) * block;
  const double two = (double)(ceil_div(t2, sms / 2) * kb) * block * 0.82;
  Plan16 plan{two < one && t2 >= sms, 256, 1, two};
  if (!plan.pair)
    plan.us = one;
  /* Tiles of 128 columns (0.32 us a block: 32 KiB of operands come from L2 for half the
     work, 512 x 11008 x 4096 takes 70 us with them and 60 with 256 columns) and runs of K
     fill the SMs that few tiles leave idle; runs cost a second launch (about 3 us) and
     their sums' way through L2 (8 bytes a sum at 4 TB/s). 100 x 100 x 8000: 736 us on the
     plain kernel, 21 in 16 runs; 1664 x 128 x 4160: 28 and 18. */
  for (int bn = 256; bn >= 128; bn -= 128) {
    const int64_t tiles = ceil_div(m, 128) * ceil_div(n, bn);
    for (int runs = 1; runs <= 16 && runs <= kb; ++runs) {
      if (runs > 1 && (!scratch || tiles * runs > sms))
        break;
      const double us = (double)(ceil_div(tiles * runs, sms) * ceil_div(kb, runs)) *
                            (bn == 256 ? block : 0.32) +
                        (runs > 1 ? 4.0 + 2.0e-6 * runs * m * n : 0.0);
      if (us < plan.us)
        plan = Plan16{false, bn, runs, us};
    }
  }
  plan.us += 5.0;
  return plan;
}
/* The plain kernel: 1.5 us for 16 of K whatever the size, up to four 64 x 64 tiles an SM.
   It reads any strides, so it is the one for short products that would have to be copied
   first (a copy: 4 us and more). 300 x 260 x 136: 19 us, 26 on the tensor cores. A call
   with a copy takes the host 16.5 us, scratch and a launch more than the plain one's 13.5,
   so up to 128 of K the plain kernel is done before: 292 x 591 x 77 13.6 against 16.5,
   65 x 129 x 100 13.5 against 16.3; 170 x 846 x 292 31 against 17. */
double plain16_us(int64_t m, int64_t n, int64_t k) {
  return 4.0 + 1.5 * (double)(ceil_div(k, 16) *
                              ceil_div(ceil_div(m, 64) * ceil_div(n, 64), 4 * sm_count()));
}
bool plain16(bool a_ok, bool b_ok, int64_t m, int64_t n, int64_t k, const Plan16 &plan) {
  return plain16_us(m, n, k) < (a_ok && b_ok ? plan.us : std::max(plan.us + 4.0, 16.1));
}
int64_t up8(int64_t v) { return (v + 7) / 8 * 8; }
size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

} // namespace

const char *gemm_16_route(int route, bool is_bf16, const void *a, int64_t lda,
                          const void *b, int64_t ldb, void *c, int64_t ldc,
                          int64_t m, int64_t n, int64_t k, void *scratch,
                          cudaStream_t stream) {
  if (m <= 0 || n <= 0)
    return nullptr;
  if (route == 3)
    return gemm_16_plain(is_bf16, a, lda, b, ldb, c, ldc, m, n, k, stream);
  if (!umma_shape_ok(a, lda, b, ldb, c, ldc, m, n, k))
    return "the tcgen05 GEMM needs 16-byte aligned bases and row strides that "
           "are multiples of 8 elements";
  if (route == 4)
    return gemm_16_pair(4, is_bf16, a, lda, b, ldb, c, ldc, m, n, k, stream);
  if (route == 5) {
    if (!scratch || ((uintptr_t)scratch & 15) || k % 8 != 0)
      return "the transposed-B route needs a 16-byte aligned scratch matrix "
             "and k a multiple of 8";
    if (const char *why = transpose_16(b, ldb, scratch, k, k, n, stream))
      return why;
    return gemm_16_pair(5, is_bf16, a, lda, scratch, k, c, ldc, m, n, k, stream);
  }
  if (route == 2) {
    if (!scratch || ((uintptr_t)scratch & 15) || k % 8 != 0)
      return "the transposed-B route needs a 16-byte aligned scratch matrix "
             "and k a multiple of 8";
    if (const char *why = transpose_16(b, ldb, scratch, k, k, n, stream))
      return why;
    CUtensorMap ma, mb;
    if (!make_map_16(&ma, a, k, m, lda, BK, BM, is_bf16))
      return "cuTensorMapEncodeTiled refused the A matrix";
    if (!make_map_16(&mb, scratch, k, n, k, BK, 256, is_bf16))
      return "cuTensorMapEncodeTiled refused the transposed B matrix";
    return is_bf16
               ? launch_umma<__nv_bfloat16, false, 256>(
                     ma, mb, Out<__nv_bfloat16>{(__nv_bfloat16 *)c, ldc, 1, 1, nullptr, 0},
                     (int)m, (int)n, (int)k, stream)
               : launch_umma<__half, false, 256>(
                     ma, mb, Out<__half>{(__half *)c, ldc, 1, 1, nullptr, 0}, (int)m, (int)n,
                     (int)k, stream);
  }
  return is_bf16
             ? run_umma(256, a, lda, b, ldb,
                        Out<__nv_bfloat16>{(__nv_bfloat16 *)c, ldc, 1, 1, nullptr, 0}, m, n,
                        k, stream)
             : run_umma(256, a, lda, b, ldb, Out<__half>{(__half *)c, ldc, 1, 1, nullptr, 0},
                        m, n, k, stream);
}

/* What gemm_16 can use: room for A and B where TMA cannot read them as they are, and for
   the sums of several runs of K. */
size_t gemm_16_scratch_bytes(const void *a, int64_t lda, const void *b, int64_t ldb,
                             int64_t m, int64_t n, int64_t k) {
  if (m <= 0 || n <= 0 || !dims_ok(m, n, k))
    return 0;
  const bool a_ok = rows_ok(a, lda), b_ok = rows_ok(b, ldb);
  const Plan16 plan = plan_16(m, n, k, true);
  if (plain16(a_ok, b_ok, m, n, k, plan))
    return 0;
  return (a_ok ? 0 : up256((size_t)(m * up8(k)) * 2)) +
         (b_ok ? 0 : up256((size_t)(k * up8(n)) * 2)) +
         (plan.runs > 1 ? (size_t)(plan.runs * m * up8(n)) * 4 : 0);
}

const char *gemm_16(bool is_bf16, const void *a, int64_t lda, const void *b,
                    int64_t ldb, void *c, int64_t ldc, int64_t m, int64_t n,
                    int64_t k, void *scratch, cudaStream_t stream) {
  if (m <= 0 || n <= 0)
    return nullptr;
  const bool a_ok = rows_ok(a, lda), b_ok = rows_ok(b, ldb);
  /* Without scratch, strides that TMA cannot describe are the plain kernel's. */
  if (!dims_ok(m, n, k) || !tensor_maps_available() || (!scratch && !(a_ok && b_ok)))
    return gemm_16_plain(is_bf16, a, lda, b, ldb, c, ldc, m, n, k, stream);
  Plan16 plan = plan_16(m, n, k, scratch != nullptr);
  if (plain16(a_ok, b_ok, m, n, k, plan))
    return gemm_16_plain(is_bf16, a, lda, b, ldb, c, ldc, m, n, k, stream);
  char *room = (char *)scratch;
  if (!a_ok || !b_ok) {
    Pack16 part[2] = {};
    auto packed = [&](Pack16 &q, const void *&p, int64_t &ld, int64_t rows, int64_t cols) {
      const int64_t pitch = up8(cols);
      q = Pack16{(const uint16_t *)p, (uint4 *)room, ld, (int)rows, (int)cols,
                 (int)(pitch / 8), (int)ceil_div(rows * (pitch / 8), 256)};
      p = room;
      ld = pitch;
      room += up256((size_t)(rows * pitch) * 2);
    };
    if (!a_ok)
      packed(part[0], a, lda, m, k);
    if (!b_ok)
      packed(part[1], b, ldb, k, n);
    pack16_kernel<<<(unsigned)(part[0].blocks + part[1].blocks), 256, 0, stream>>>(part[0],
                                                                                 part[1]);
    if (cudaGetLastError() != cudaSuccess)
      return "the launch that copies the operands failed";
  }
  /* VXB_GEMM_ROUTE=1 or 4 pins the choice (for measurements). */
  const char *force = getenv("VXB_GEMM_ROUTE");
  if (force && (force[0] == '1' || force[0] == '4'))
    plan = Plan16{force[0] == '4', 256, 1, 0.0};
  if (plan.pair)
    return gemm_16_pair(4, is_bf16, a, lda, b, ldb, c, ldc, m, n, k, stream);
  const int vec = rows_ok(c, ldc);
  float *partials = plan.runs > 1 ? (float *)room : nullptr;
  return is_bf16 ? run_umma(plan.bn, a, lda, b, ldb,
                            Out<__nv_bfloat16>{(__nv_bfloat16 *)c, ldc, vec, plan.runs,
                                               partials, up8(n)},
                            m, n, k, stream)
                 : run_umma(plan.bn, a, lda, b, ldb,
                            Out<__half>{(__half *)c, ldc, vec, plan.runs, partials, up8(n)},
                            m, n, k, stream);
}

int gemm_status(cudaStream_t stream) {
  int v = 0, zero = 0;
  if (cudaStreamSynchronize(stream) != cudaSuccess)
    return -1;
  if (cudaMemcpyFromSymbol(&v, g_status, sizeof v) != cudaSuccess)
    return -1;
  if (v)
    cudaMemcpyToSymbol(g_status, &zero, sizeof zero);
  const int pair = gemm_pair_status(), tile = gemm_f32_tile_status();
  return v ? v : pair ? pair : tile;
}

} // namespace vxb
