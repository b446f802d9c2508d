/* plain_tile.cuh -- a 128 x 128 tile of an f32 product with plain multiply-adds: what the
 * f32 kernels on the tensor cores turn to where an operand holds a value that their bf16
 * terms cannot carry.
 *
 * 512 threads, 8 x 4 results each, ascending k, 32 of K at a time through two stages of
 * shared memory; the next 32 are read while these are multiplied.  Bound by the FP32 pipe:
 * 4 096 cycles for 32 of K.
 */
#ifndef VXB_PLAIN_TILE_CUH
#define VXB_PLAIN_TILE_CUH

#include <stdint.h>

namespace vxb {
namespace {

/* Eight consecutive values of a row, zero outside [0, cols) and where !inside.
   vec: how many at a time the row's alignment allows, 4, 2 or 1. */
__device__ __forceinline__ void read8(float (&v)[8], const float *row, int c, int cols,
                                      bool inside, int vec) {
  const bool whole = inside && c + 8 <= cols;
  if (whole && vec == 4) {
    const float4 a = *reinterpret_cast<const float4 *>(row + c);
    const float4 b = *reinterpret_cast<const float4 *>(row + c + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else if (whole && vec == 2) {
#pragma unroll
    for (int e = 0; e < 8; e += 2) {
      const float2 a = *reinterpret_cast<const float2 *>(row + c + e);
      v[e] = a.x;
      v[e + 1] = a.y;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e)
      v[e] = inside && c + e < cols ? row[c + e] : 0.0f;
  }
}

struct PlainTile {
  const float *a, *b; /* A [m, k], B [k, n] */
  int64_t lda, ldb;
  int m, n;
  int vec_a, vec_b; /* read8 */
};
constexpr int kPlainThreads = 512, kPlainK = 32;
constexpr int kPlainPitch = 128 + 4; /* of a row of either operand, in floats */
constexpr int kPlainFloats = 2 * 2 * kPlainK * kPlainPitch; /* two stages of A and B */

/* acc[4 i + j] = row row0 + 8 (tid / 32) + i, column col0 + 4 (tid % 32) + j, over
   k0 <= k < k1 (k0 a multiple of 8); tid 0 .. 511, all of which come here; room:
   kPlainFloats floats of shared memory, 16-byte aligned. */
__device__ __forceinline__ void plain_tile(const PlainTile &g, int row0, int col0, int k0,
                                           int k1, int tid, float *room, float (&acc)[32]) {
  const int ty = tid / 32, tx = tid % 32;
  /* a thread's share of a stage: eight of a row of A, which go down a column of the
     stage (neighbouring lanes, neighbouring rows), and eight of a row of B */
  const int ar = tid % 128, ac = tid / 128 * 8, br = tid / 16, bc = tid % 16 * 8;
  float va[8], vb[8];
  auto read = [&](int k) {
    read8(va, g.a + (int64_t)(row0 + ar) * g.lda, k + ac, k1, row0 + ar < g.m, g.vec_a);
    read8(vb, g.b + (int64_t)(k + br) * g.ldb, col0 + bc, g.n, k + br < k1, g.vec_b);
  };
#pragma unroll
  for (int i = 0; i < 32; ++i)
    acc[i] = 0.0f;
  if (k0 < k1)
    read(k0);
  int s = 0;
#pragma unroll 1
  for (int k = k0; k < k1; k += kPlainK, s ^= 1) {
    float *const sa = room + s * 2 * kPlainK * kPlainPitch;
    float *const sb = sa + kPlainK * kPlainPitch;
#pragma unroll
    for (int e = 0; e < 8; ++e)
      sa[(ac + e) * kPlainPitch + ar] = va[e];
    *reinterpret_cast<float4 *>(sb + br * kPlainPitch + bc) =
        make_float4(vb[0], vb[1], vb[2], vb[3]);
    *reinterpret_cast<float4 *>(sb + br * kPlainPitch + bc + 4) =
        make_float4(vb[4], vb[5], vb[6], vb[7]);
    /* one barrier a step: the stage written next was read before it */
    asm volatile("bar.sync 1, 512;" ::: "memory");
    if (k + kPlainK < k1)
      read(k + kPlainK);
#pragma unroll 4
    for (int kk = 0; kk < kPlainK; ++kk) {
      const float4 x0 = *reinterpret_cast<const float4 *>(sa + kk * kPlainPitch + ty * 8);
      const float4 x1 = *reinterpret_cast<const float4 *>(sa + kk * kPlainPitch + ty * 8 + 4);
      const float4 y = *reinterpret_cast<const float4 *>(sb + kk * kPlainPitch + tx * 4);
      const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        acc[4 * i] = fmaf(x[i], y.x, acc[4 * i]);
        acc[4 * i + 1] = fmaf(x[i], y.y, acc[4 * i + 1]);
        acc[4 * i + 2] = fmaf(x[i], y.z, acc[4 * i + 2]);
        acc[4 * i + 3] = fmaf(x[i], y.w, acc[4 * i + 3]);
      }
    }
  }
}

} // namespace
} // namespace vxb

#endif /* VXB_PLAIN_TILE_CUH */
