/* q4_tiles.cu -- products of many rows of activations with Q4_0 matrices on tcgen05: the
 * expert projections of many positions.
 *
 *   D[r, j] = sum over c of ((code[r, c] - 8) * scale[r, c / 32]) * x[j, c]
 *
 * A block takes 128 weight rows and up to 128 of one expert's pairs.  A weight has 4 + 11
 * significant bits: two bf16 terms hold it exactly, and they are made on the way into
 * tensor memory, the A operand; x is three bf16 terms in shared memory.  Of the six
 * products the smallest (below 2^-24 of the first) is left out.  The tensor core's own
 * sums lose a little with their length: the first product has an accumulator of its own,
 * which is added to f32 registers after 128 columns, while the other products of the next
 * block run (the layer's error against 64 bits is 3.5e-7; with 512 columns it was 9.1e-7, on
 * mma.sync with a sum per 32 columns 5.9e-7); the others, 2^-8 of it, stay in theirs to the
 * end.
 *
 * Sixteen warps, persistent over (segment of pairs, row tile), with rings of three blocks
 * of 64 columns:
 *   warp 0       TMA: the terms of the pairs into shared memory (made beforehand, an
 *                expert's pairs one after another: group_terms_kernel);
 *   warp 1       issues the products, twenty instructions a block;
 *   warp 2       TMA: the codes, 128 rows of 256 columns at a time;
 *   warps 4-15   three sets of 128 threads, a row a thread: set k makes the terms of every
 *                third block, and keeps the sums of every third run of columns.
 * SwiGLU takes 64 gate rows and the 64 up rows beside them, which meet in shared memory
 * at the end.
 *
 * What bounds it: with 128 pairs the tensor pipe for two thirds of the time (1 280 of
 * 2 000 cycles a block of 64 columns) and the round of barriers between it and the sets for
 * the rest; with few pairs that round alone, 1 250 cycles.  The gate and up rows of 8
 * experts of 14336 x 4096 take 0.93 ms for 1000 pairs, 2.5 ms on mma.sync (moe_grouped.cu).
 *
 * A scale of infinity makes its 32 weights NaN (its second term is infinity minus
 * infinity); moe_grouped.cu, which applies the scale to the sum of the 32, gives infinity.
 *
 * What was slower: the codes alone as A (exact, three products) and the scale applied to
 * the sums of each 32 columns, 1 850 cycles a block of few pairs and 2 500 of 128, since
 * sums then leave tensor memory twice a block; codes fetched by their own threads, 32 bytes
 * of 32 rows a load.  The loops are not unrolled over the rings or the columns: straight-
 * line code of four kinds of warps on an SM runs at the pace of instruction fetches.
 */
#include "kernels.h"
#include "launch.cuh"
#include "launch_util.h"
#include "ptx.cuh"
#include "terms.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace vxb {

bool tensor_maps_available();
bool make_map_16(CUtensorMap *map, const void *base, int64_t inner, int64_t rows,
                 int64_t ld, int box_inner, int box_rows, bool is_bf16);

namespace {

constexpr int ROWS = 128, PAIRS = 128, BK = 64, GROUP = 32, RING = 3, SETS = 3;
constexpr int WIDE = 4;   /* blocks of codes, and of scales, that are fetched together */
constexpr int CODE_RING = 2, SCALE_RING = 2;
constexpr int SEGMENT = 2; /* blocks between two transfers to registers */
constexpr int MOST = 48;   /* columns of a set: a third of 128, in sixteens */
constexpr int TERM_BYTES = PAIRS * BK * 2, HALF_BYTES = TERM_BYTES / 2;
constexpr int STAGE_BYTES = 3 * TERM_BYTES;
constexpr int MEET_BYTES = (ROWS / 2) * PAIRS * 4;
constexpr int CODES_STAGE = ROWS * WIDE * BK / 2; /* 128-byte rows, swizzled */
constexpr int CODES_BYTES = CODE_RING * CODES_STAGE;
constexpr int SCALES_BYTES = SCALE_RING * SETS * ROWS * WIDE * 4; /* 16 bytes a thread */
static_assert(WIDE * BK / 2 == 128, "a row of codes is a swizzled row");
static_assert(RING == SETS, "a set fills a place of the ring of its own");
constexpr int THREADS = 512;
constexpr int A_COL = 0, A_COLS = BK, D_COL = RING * A_COLS; /* two terms of a block */
static_assert(D_COL + 2 * PAIRS <= 512, "tensor memory");

enum { Q_EMPTY_B = 0xa1, Q_FULL_B, Q_FULL_A, Q_EMPTY_A, Q_FULL_D, Q_EMPTY_D, Q_EMPTY_C,
       Q_FULL_C };
__device__ int g_q4_status; /* first wait that ran out since the last read */

struct Bars {
  uint64_t b_full[RING], a_full[RING], empty[RING], d_full, d_empty;
  uint64_t c_full[CODE_RING], c_empty[CODE_RING];
  uint32_t tmem_base;
  int stop;
};
constexpr int SMEM_BYTES = RING * STAGE_BYTES + MEET_BYTES + CODES_BYTES + SCALES_BYTES +
                           1024 + (int)sizeof(Bars) + 64;

/* Pairs first .. first + count of the grouped order, all of one expert. */
struct Segment {
  int expert, first, count, unused;
};

struct Q4Tiles {
  const uint32_t *w;       /* [experts * expert_rows, cols / 8] */
  const __half *scales;    /* [experts * expert_rows, cols / 32] */
  const Segment *segments;
  const int32_t *segment_count;
  const int32_t *order;
  float *out;              /* pair p: row p, out_pitch apart */
  int64_t out_pitch;
  const float *pair_scale; /* null: 1 */
  int pairs, rows, cols;
  int64_t expert_rows;     /* 2 * rows (gate then up) or rows */
  int scale_words;         /* how many words of scales a row's alignment lets a thread
                              fetch at once: 4, 2 or 1 */
};

#define WAIT(bar, parity, code)                                                          \
  do {                                                                                   \
    if (!ptx::mbar_wait((bar), (parity), stop)) {                                        \
      atomicCAS(&g_q4_status, 0, (code));                                                \
      *stop = 1;                                                                         \
    }                                                                                    \
  } while (0)

/* Codes 2 i and 2 i + 1 of a word, times the scale s1 + s2 (bf16 pairs of equal halves),
   as the two terms of their values. (code - 8) * s2 is exact (4 and 3 bits), so t1 is the
   value rounded once; what is left of it has at most 7 bits and comes out exactly. */
__device__ __forceinline__ void two_weights(uint32_t word, int i, uint32_t s1, uint32_t s2,
                                            uint32_t &t1, uint32_t &t2) {
  const uint32_t byte = __byte_perm(word, 0, 0x4440 + i);
  uint32_t c, low, rest;
  asm("sub.rn.bf16x2 %0, %1, %2;"
      : "=r"(c)
      : "r"(((byte * 4097u) & 0x000f000fu) | 0x43004300u), "r"(0x43084308u));
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(low) : "r"(c), "r"(s2));
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(t1) : "r"(c), "r"(s1), "r"(low));
  asm("{.reg .b32 n;\n\tneg.bf16x2 n, %3;\n\tfma.rn.bf16x2 %0, %1, %2, n;}"
      : "=r"(rest)
      : "r"(c), "r"(s1), "r"(t1));
  asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(t2) : "r"(rest), "r"(low));
}
/* the value rounded to bf16, in both halves */
__device__ __forceinline__ uint32_t bf16_pair(float x) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, x);
  return *reinterpret_cast<const uint32_t *>(&v);
}
template <int COLUMNS> __device__ __forceinline__ void move_down(float (&sums)[MOST]) {
#pragma unroll
  for (int i = 0; i + COLUMNS < MOST; ++i)
    sums[i] = sums[i + COLUMNS];
}
__device__ __forceinline__ float gated(float gate, float up) {
  return gate / (1.0f + expf(0.0f - gate)) * up;
}
/* Up to four words of scales: as wide as the alignment allows, none past the row. */
__device__ __forceinline__ void fetch_scales(uint32_t *to, const uint32_t *from, int left,
                                             int words) {
  const uint32_t dst = ptx::smem_addr(to);
  if (words == 4) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(from)
                 : "memory");
  } else if (words == 2) {
    for (int i = 0; i < WIDE && i < left; i += 2)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 4 * i),
                   "l"(from + i)
                   : "memory");
  } else {
    for (int i = 0; i < WIDE && i < left; ++i)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * i),
                   "l"(from + i)
                   : "memory");
  }
}
__device__ __forceinline__ void copies_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int LEFT> __device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

template <bool SWIGLU>
__global__ void __launch_bounds__(THREADS, 1)
q4_tiles_kernel(const __grid_constant__ CUtensorMap map_x,
                const __grid_constant__ CUtensorMap map_w, const Q4Tiles a) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float *meet = reinterpret_cast<float *>(smem + RING * STAGE_BYTES);
  uint8_t *codes_at = smem + RING * STAGE_BYTES + MEET_BYTES;
  uint8_t *scales_at = codes_at + CODES_BYTES;
  Bars *bars = reinterpret_cast<Bars *>(scales_at + SCALES_BYTES);
  const int warp = ptx::warp_index(), lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RING; ++s) {
      ptx::mbar_init(&bars->b_full[s], 1);
      ptx::mbar_init(&bars->a_full[s], 4);
      ptx::mbar_init(&bars->empty[s], 1);
    }
    ptx::mbar_init(&bars->d_full, 1);
    ptx::mbar_init(&bars->d_empty, 4 * SETS);
    for (int c = 0; c < CODE_RING; ++c) {
      ptx::mbar_init(&bars->c_full[c], 1);
      ptx::mbar_init(&bars->c_empty[c], 4 * SETS);
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
  chain_wait();

  constexpr int TILE = SWIGLU ? ROWS / 2 : ROWS;
  const int row_tiles = (a.rows + TILE - 1) / TILE;
  const int items = *a.segment_count * row_tiles, blocks = a.cols / BK;
  auto segment_of = [&](int item) { return a.segments[item / row_tiles]; };
  /* the matrix row behind row `l` of an item's tile; one past the end reads row 0 */
  auto matrix_row = [&](int item, int l) -> int64_t {
    const int r = item % row_tiles * TILE + (SWIGLU ? l & 63 : l);
    return segment_of(item).expert * a.expert_rows + (r < a.rows ? r : 0) +
           (SWIGLU && l >= 64 ? a.rows : 0);
  };

  if (warp == 0) {
    if (lane == 0) {
      ptx::tma_prefetch_desc(&map_x);
      int it = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        const Segment seg = segment_of(item);
        const int halves = seg.count > PAIRS / 2 ? 2 : 1;
        for (int kb = 0; kb < blocks; ++kb, ++it) {
          const int s = it % RING;
          if (!ptx::mbar_wait(&bars->empty[s], ((it / RING) & 1) ^ 1, stop)) {
            atomicCAS(&g_q4_status, 0, Q_EMPTY_B);
            *stop = 1;
            ok = false;
            break;
          }
          ptx::mbar_expect_tx(&bars->b_full[s], 3 * halves * HALF_BYTES);
          for (int t = 0; t < 3; ++t)
            for (int h = 0; h < halves; ++h)
              ptx::tma_load_2d(smem + s * STAGE_BYTES + t * TERM_BYTES + h * HALF_BYTES,
                               &map_x, t * a.cols + kb * BK, seg.first + h * (PAIRS / 2),
                               &bars->b_full[s]);
        }
      }
      for (int back = 0; back < RING && back < it; ++back) {
        const int j = it - 1 - back;
        ptx::mbar_wait_alone(&bars->b_full[j % RING], (j / RING) & 1);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    int s = 0;
    uint32_t phase = 0, d_phase = 1;
    const uint64_t b_desc = ptx::smem_desc_sw128(ptx::smem_addr(smem), 16, 1024);
    const uint32_t sum = tmem + D_COL, rest = sum + PAIRS;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const int n = (segment_of(item).count + 15) & ~15;
      const uint32_t idesc = ptx::idesc_f16(true, false, false, ROWS, n);
#pragma unroll 1
      for (int kb = 0; kb < blocks; ++kb) {
        const bool first = kb % SEGMENT == 0;
        const bool last = kb % SEGMENT == SEGMENT - 1 || kb + 1 == blocks;
        WAIT(&bars->b_full[s], phase, Q_FULL_B);
        WAIT(&bars->a_full[s], phase, Q_FULL_A);
        if (kb == 0) { /* both accumulators of the item before have been read */
          WAIT(&bars->d_empty, d_phase, Q_EMPTY_D);
          d_phase ^= 1;
        }
        __syncwarp();
        ptx::tc_fence_after_sync();
        if (ptx::elect_one()) {
          const uint32_t w1 = tmem + A_COL + s * A_COLS, w2 = w1 + BK / 2;
          const uint64_t x1 = b_desc + (s * STAGE_BYTES >> 4);
          const uint64_t x2 = x1 + (TERM_BYTES >> 4), x3 = x2 + (TERM_BYTES >> 4);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) {
            const int k8 = kk * 8, k2 = kk * 2; /* tensor memory columns, 16 bytes */
            ptx::umma_f16_ts(rest, w1 + k8, x3 + k2, idesc, kb != 0 || kk != 0);
            ptx::umma_f16_ts(rest, w2 + k8, x2 + k2, idesc, 1);
            ptx::umma_f16_ts(rest, w2 + k8, x1 + k2, idesc, 1);
            ptx::umma_f16_ts(rest, w1 + k8, x2 + k2, idesc, 1);
          }
        }
        __syncwarp();
        if (first && kb != 0) {
          WAIT(&bars->d_empty, d_phase, Q_EMPTY_D);
          d_phase ^= 1;
          __syncwarp();
          ptx::tc_fence_after_sync();
        }
        if (ptx::elect_one()) {
          const uint32_t w1 = tmem + A_COL + s * A_COLS;
          const uint64_t x1 = b_desc + (s * STAGE_BYTES >> 4);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            ptx::umma_f16_ts(sum, w1 + kk * 8, x1 + kk * 2, idesc, !first || kk != 0);
          ptx::umma_commit(&bars->empty[s]);
          if (last)
            ptx::umma_commit(&bars->d_full);
        }
        __syncwarp();
        if (++s == RING) {
          s = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 2) {
    if (lane == 0) {
      /* 128 rows of 256 columns at a time; rows past the matrix are some other's, or zero,
         and are not stored */
      ptx::tma_prefetch_desc(&map_w);
      int it = 0;
      bool ok = true;
      for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
        const int row = (int)(segment_of(item).expert * a.expert_rows) +
                        item % row_tiles * TILE;
        for (int kb = 0; kb < blocks; kb += WIDE, ++it) {
          const int c = it % CODE_RING;
          if (!ptx::mbar_wait(&bars->c_empty[c], ((it / CODE_RING) & 1) ^ 1, stop)) {
            atomicCAS(&g_q4_status, 0, Q_EMPTY_C);
            *stop = 1;
            ok = false;
            break;
          }
          uint8_t *to = codes_at + c * CODES_STAGE;
          ptx::mbar_expect_tx(&bars->c_full[c], CODES_STAGE);
          ptx::tma_load_2d(to, &map_w, kb * (BK / 4), row, &bars->c_full[c]);
          ptx::tma_load_2d(to + CODES_STAGE / 2, &map_w, kb * (BK / 4),
                           row + (SWIGLU ? a.rows : ROWS / 2), &bars->c_full[c]);
        }
      }
      for (int back = 0; back < CODE_RING && back < it; ++back) {
        const int j = it - 1 - back;
        ptx::mbar_wait_alone(&bars->c_full[j % CODE_RING], (j / CODE_RING) & 1);
      }
    }
    __syncwarp();
  } else if (warp >= 4) {
    const int set = warp / 4 - 1, quarter = warp & 3, l = quarter * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16);
    uint32_t *const own =
        reinterpret_cast<uint32_t *>(scales_at) + (threadIdx.x - ROWS) * WIDE;
    int turn = 0, c = 0; /* whose block an item's first is; the place of a stage of codes */
    uint32_t phase = 1, c_phase = 0, d_phase = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
      const Segment seg = segment_of(item);
      const int n = (seg.count + 15) & ~15, part = (n + SETS * 16 - 1) / (SETS * 16) * 16;
      const int from = set * part, mine = max(0, min(n - from, part)); /* columns */
      const uint32_t *scale_of = reinterpret_cast<const uint32_t *>(
          a.scales + matrix_row(item, l) * (a.cols / GROUP));
      const int r = item % row_tiles * TILE + (SWIGLU ? l & 63 : l);
      const bool stored = r < a.rows, up = SWIGLU && quarter >= 2;
      /* Of gate and up each hands the other half of its columns over at the end: the
         gate's threads finish the first half, the up's the second. Lane i knows the pairs
         of the columns i and 32 + i that this warp finishes. */
      const int share = SWIGLU ? mine / 2 : mine, skip = up ? share : 0;
      int pair[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int slot = from + skip + i * 32 + lane;
        pair[i] = -1;
        if (i * 32 + lane < share && slot < seg.count)
          pair[i] = __ldg(a.order + seg.first + slot);
        if (pair[i] >= a.pairs)
          pair[i] = -1;
      }
      float sums[MOST];
#pragma unroll
      for (int i = 0; i < MOST; ++i)
        sums[i] = 0.0f;
      auto fetch = [&](int kb) { /* a thread's own scales */
        if (kb < blocks)
          fetch_scales(own + kb / WIDE % SCALE_RING * (SETS * ROWS * WIDE), scale_of + kb,
                       blocks - kb, a.scale_words);
        copies_commit();
      };
      auto take_sums = [&](bool with_rest) {
        WAIT(&bars->d_full, d_phase, Q_FULL_D);
        d_phase ^= 1;
        __syncwarp();
        ptx::tc_fence_after_sync();
#pragma unroll
        for (int q = 0; q < MOST; q += 16) {
          if (q >= mine)
            break;
          uint32_t u[16];
          ptx::tmem_ld_32x32b_x16(lanes + D_COL + from + q, u);
          ptx::tmem_ld_wait_for(u);
#pragma unroll
          for (int e = 0; e < 16; ++e)
            sums[q + e] += __uint_as_float(u[e]);
          if (with_rest) {
            ptx::tmem_ld_32x32b_x16(lanes + D_COL + PAIRS + from + q, u);
            ptx::tmem_ld_wait_for(u);
#pragma unroll
            for (int e = 0; e < 16; ++e)
              sums[q + e] += __uint_as_float(u[e]);
          }
        }
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(&bars->d_empty);
      };
      int stage = 0, taken = 0; /* of the codes; segments whose sums were taken */
      auto enter = [&]() {
        WAIT(&bars->c_full[c], c_phase, Q_FULL_C);
        __syncwarp();
        fetch((stage + 1) * WIDE);
        copies_wait<1>();
      };
      auto leave = [&]() {
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(&bars->c_empty[c]);
        if (++c == CODE_RING) {
          c = 0;
          c_phase ^= 1;
        }
        ++stage;
      };
      fetch(0);
      enter();
#pragma unroll 1
      for (int kb = set - turn + (set < turn ? SETS : 0); kb < blocks; kb += SETS) {
        while (stage < kb / WIDE) {
          leave();
          enter();
        }
        /* the segments before the last: the products of this one wait for them */
        for (; taken < kb / SEGMENT - 1; ++taken)
          take_sums(false);
        const int at = kb % WIDE;
        const uint8_t *src = codes_at + c * CODES_STAGE + l * 128;
        const uint4 c0 = *reinterpret_cast<const uint4 *>(src + (((2 * at) ^ (l & 7)) << 4));
        const uint4 c1 =
            *reinterpret_cast<const uint4 *>(src + (((2 * at + 1) ^ (l & 7)) << 4));
        const uint32_t two = own[stage % SCALE_RING * (SETS * ROWS * WIDE) + at];
        WAIT(&bars->empty[set], phase, Q_EMPTY_A);
        phase ^= 1;
        __syncwarp();
        ptx::tc_fence_after_sync();
        const uint32_t to = lanes + A_COL + set * A_COLS;
#pragma unroll 1
        for (int g = 0; g < 2; ++g) { /* a group of 32 columns, one scale */
          const float scale = __half2float(
              __ushort_as_half((unsigned short)(g ? two >> 16 : two & 0xffffu)));
          const uint32_t s1 = bf16_pair(scale);
          const uint32_t s2 = bf16_pair(scale - __uint_as_float(s1 << 16));
          const uint32_t word[4] = {g ? c1.x : c0.x, g ? c1.y : c0.y, g ? c1.z : c0.z,
                                    g ? c1.w : c0.w};
          uint32_t t1[16], t2[16];
#pragma unroll
          for (int i = 0; i < 16; ++i)
            two_weights(word[i / 4], i % 4, s1, s2, t1[i], t2[i]);
          ptx::tmem_st_32x32b_x16(to + g * 16, t1);
          ptx::tmem_st_32x32b_x16(to + BK / 2 + g * 16, t2);
        }
        ptx::tmem_st_wait();
        ptx::tc_fence_before_sync();
        __syncwarp();
        if (lane == 0)
          ptx::mbar_arrive(&bars->a_full[set]);
        for (; taken < kb / SEGMENT; ++taken)
          take_sums(false);
      }
      while (stage < (blocks - 1) / WIDE) {
        leave();
        enter();
      }
      leave();
      for (; taken < (blocks - 1) / SEGMENT; ++taken)
        take_sums(false);
      take_sums(true);
      turn = (turn + blocks) % SETS;
      if (SWIGLU) {
#pragma unroll
        for (int i = 0; i < MOST; ++i)
          if (i < mine && (up ? i < share : i >= share))
            meet[(from + i) * (ROWS / 2) + (l & 63)] = sums[i];
        asm volatile("bar.sync 1, 384;" ::: "memory");
        if (up) /* its columns first in its registers */
#pragma unroll 1
          for (int i = 0; i < share; i += 8)
            move_down<8>(sums);
      }
      /* the sums move down by eight from one round to the next, so that the code is that
         of eight */
#pragma unroll 1
      for (int i0 = 0; i0 < share; i0 += 8) {
        const int first = from + skip + i0, mine_of = i0 < 32 ? pair[0] : pair[1];
        const float weight = !SWIGLU && a.pair_scale && mine_of >= 0
                                 ? __ldg(a.pair_scale + mine_of) : 1.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int p = __shfl_sync(0xffffffffu, mine_of, (i0 + i) & 31);
          float out = sums[i];
          if (SWIGLU) {
            const float other = meet[(first + i) * (ROWS / 2) + (l & 63)];
            out = gated(up ? other : out, up ? out : other);
          } else {
            out *= __shfl_sync(0xffffffffu, weight, (i0 + i) & 31);
          }
          if (p >= 0 && stored)
            a.out[p * a.out_pitch + r] = out;
        }
        move_down<8>(sums);
      }
      if (SWIGLU)
        asm volatile("bar.sync 1, 384;" ::: "memory");
    }
    copies_wait<0>();
  }
  __syncwarp();
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after_sync();
    ptx::tmem_dealloc(tmem, 512);
  }
}

/* The rows of x behind the grouped pairs as three bf16 terms, [slots, 3 cols], slot by
   slot, eight columns a thread; the last block cuts the runs of tiles of one expert into
   segments of at most 128 slots. */
__global__ void __launch_bounds__(256)
group_terms_kernel(__nv_bfloat16 *terms, Segment *segments, int32_t *segment_count,
                   const float *x, int64_t x_pitch, int x_div, const int32_t *order,
                   const int32_t *tile_expert, int tiles, int align, int experts,
                   int pairs, int cols) {
  chain_release();
  chain_wait();
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ int count;
    if (threadIdx.x == 0)
      count = 0;
    __syncthreads();
    const int per = PAIRS / align;
    for (int t = threadIdx.x; t < tiles; t += blockDim.x) {
      const int e = tile_expert[t];
      if (e < 0 || e >= experts || (t > 0 && tile_expert[t - 1] == e))
        continue;
      int run = 1;
      while (t + run < tiles && tile_expert[t + run] == e)
        ++run;
      const int pieces = (run + per - 1) / per;
      const int at = atomicAdd(&count, pieces);
      for (int i = 0; i < pieces; ++i) {
        const int first = (int)((int64_t)run * i / pieces);
        const int end = (int)((int64_t)run * (i + 1) / pieces);
        segments[at + i] = Segment{e, (t + first) * align, (end - first) * align, 0};
      }
    }
    __syncthreads();
    if (threadIdx.x == 0)
      *segment_count = count;
    return;
  }
  const int eights = cols / 8;
  const int64_t total = (int64_t)tiles * align * eights;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)(gridDim.x - 1) * blockDim.x) {
    const int64_t slot = i / eights;
    const int c = (int)(i - slot * eights) * 8;
    const int e = tile_expert[slot / align];
    if (e < 0 || e >= experts)
      continue; /* no pair has a slot here, and `order` may end before it */
    const int p = order[slot];
    float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v = u;
    if (p >= 0 && p < pairs) {
      const float4 *from = reinterpret_cast<const float4 *>(x + p / x_div * x_pitch + c);
      u = from[0];
      v = from[1];
    }
    const float eight[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    store_terms8(terms, cols, slot, c, eight);
  }
}

template <bool SWIGLU>
const char *launch(Q4Tiles a, const void *terms, int64_t slots, int64_t experts,
                   int64_t most_segments, cudaStream_t stream) {
  a.scale_words = a.cols % 256 == 0 && ((uintptr_t)a.scales & 15) == 0  ? 4
                  : a.cols % 128 == 0 && ((uintptr_t)a.scales & 7) == 0 ? 2
                                                                        : 1;
  CUtensorMap map, map_w; /* four codes count as one 16-bit value of the second */
  if (!make_map_16(&map, terms, 3 * (int64_t)a.cols, slots, 3 * (int64_t)a.cols, BK,
                   PAIRS / 2, true))
    return "cuTensorMapEncodeTiled refused the terms";
  if (!make_map_16(&map_w, a.w, a.cols / 4, experts * a.expert_rows, a.cols / 4,
                   WIDE * BK / 4, ROWS / 2, true))
    return "cuTensorMapEncodeTiled refused the weights";
  if (allow_dynamic_smem((const void *)q4_tiles_kernel<SWIGLU>, SMEM_BYTES) != cudaSuccess)
    return "the Q4_0 product could not get its shared memory";
  const int tile = SWIGLU ? ROWS / 2 : ROWS;
  const int64_t items = most_segments * ((a.rows + tile - 1) / tile);
  if (items > INT32_MAX)
    return "too many rows";
  launch_chained(q4_tiles_kernel<SWIGLU>,
                 dim3((unsigned)std::min<int64_t>(items, sm_count())), dim3(THREADS),
                 SMEM_BYTES, stream, map, map_w, a);
  return check_launch("the Q4_0 product");
}

size_t table_bytes(const MoeGroupedArgs &m) {
  return 256 + ((size_t)m.tiles * sizeof(Segment) + 255) / 256 * 256;
}

} // namespace

/* Where the line lies, measured against moe_grouped.cu: experts of 14336 x 4096 with 8
   pairs each 0.94 of its speed, with 16 0.98, with 32 1.43, with 125 2.0; experts of
   1024 x 1024, where two more launches weigh, with 32 pairs 0.92, with 64 1.38. */
size_t q4_tiles_scratch_bytes(const MoeGroupedArgs &m) {
  if (m.cols % BK != 0 || m.cols < WIDE * BK || ((uintptr_t)m.w & 15) ||
      ((uintptr_t)m.scales & 3) || !tensor_maps_available())
    return 0;
  const int64_t pairs = (int64_t)m.n * m.k, matrix = (int64_t)m.rows * m.cols;
  if (pairs < (matrix >= (1 << 22) ? 32 : 64) * (int64_t)m.experts)
    return 0;
  const size_t need = table_bytes(m) + (size_t)m.tiles * m.align * 3 * m.cols * 2;
  return need <= ((size_t)1 << 30) ? need : 0;
}

const char *q4_tiles_grouped(const MoeGroupedArgs &m, bool swiglu, void *scratch,
                             cudaStream_t stream) {
  int32_t *count = (int32_t *)scratch;
  Segment *segments = (Segment *)((char *)scratch + 256);
  __nv_bfloat16 *terms = (__nv_bfloat16 *)((char *)scratch + table_bytes(m));
  const int64_t slots = (int64_t)m.tiles * m.align;
  const int64_t eights = slots * (m.cols / 8);
  launch_chained(group_terms_kernel,
                 dim3((unsigned)std::min<int64_t>((eights + 255) / 256, 16 * sm_count()) + 1),
                 dim3(256), 0, stream, terms, segments, count, m.x, m.x_pitch,
                 swiglu ? m.k : 1, m.order, m.tile_expert, m.tiles, m.align, m.experts,
                 m.n * m.k, m.cols);
  if (const char *why = check_launch("the grouped terms"))
    return why;
  Q4Tiles a{};
  a.w = (const uint32_t *)m.w;
  a.scales = (const __half *)m.scales;
  a.segments = segments;
  a.segment_count = count;
  a.order = m.order;
  a.out = swiglu ? m.out : m.scratch;
  a.out_pitch = swiglu ? m.out_pitch : m.rows;
  a.pair_scale = swiglu ? nullptr : m.pair_weights;
  a.pairs = m.n * m.k;
  a.rows = m.rows;
  a.cols = m.cols;
  a.expert_rows = swiglu ? 2 * (int64_t)m.rows : m.rows;
  const int64_t most = std::min<int64_t>(m.tiles, m.experts + slots / (PAIRS / 2) + 1);
  return swiglu ? launch<true>(a, terms, slots, m.experts, most, stream)
                : launch<false>(a, terms, slots, m.experts, most, stream);
}

int q4_tiles_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_q4_status, sizeof v) != cudaSuccess)
    return -1;
  if (v)
    cudaMemcpyToSymbol(g_q4_status, &zero, sizeof zero);
  return v;
}

} // namespace vxb
