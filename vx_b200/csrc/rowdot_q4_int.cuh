/* rowdot_q4_int.cuh -- the Q4_0 projections of ONE sequence as whole-number products
 * (nn_matvec_q4 / nn_swiglu_q4 / nn_qkv_q4, nn.vx:1666-2190). Part of rowdot_quant.cu
 * (included there).
 *
 * A code minus 8 is a whole number, and 32 of them share a scale; so each 32 values of x
 * become fixed-point numbers with one power of two for the 32: a whole number of 30 bits
 * in four signed bytes, and a fifth byte of what that leaves.  mma.sync.m16n8k32 on bytes
 * then gives, for 16 rows and a run of 32 columns, the five sums of (code - 8) * byte,
 * exactly; each times scale * power of two is added to a sum in f32.  So a row of 4096
 * columns has 128 roundings where products with x in f32 have 4096, and x loses what lies
 * below 2^-38 of the largest of its 32.  Off from 64 bits, x from N(0, 1): 4096 x 4096
 * 4.9e-8, 4096 x 11008 6.2e-8 (three bf16 terms of x on bf16 mma.sync, which this
 * replaced: 1.0e-7, 1.4e-7); with one x of 10^6 whose weights are all 0: 1.0e-7, 8.7e-8
 * (1.0e-7, 1.4e-7; four bytes alone: 2.8e-5).  With values further apart the small ones
 * would lose what a row without a weight for the large one shows (all of it where that is
 * 10^12): where four neighbours lie 2^-17 below the largest of their 32, or further, every
 * sum of the launch is made from x in f32 instead (4096 x 4096 in 55 us, not 4.8).  Looking
 * for them takes 0.8 % of a step (sixteen tokens of the 7B-shaped decoder 24.2 -> 24.4 ms).
 *
 * Bytes because of what it takes to unpack a code: eight codes are 4-bit fields of a word;
 * the odd ones in place and the even ones shifted up by four are bytes 16 * code, and
 * an exclusive or with 0x80 makes them 16 * (code - 8): five instructions for eight
 * codes with the shift, where bf16 takes eleven.  m16n8k32 takes an SM 2.2 cycles, as
 * bf16 m16n8k16 does for half of it.
 *
 * The rows of a launch are divided evenly over the SMs, the 256-column steps of a row and
 * the tiles of eight items over a block's eight warps.  A warp walks its steps of its
 * tiles; its loads (cp.async, 16 rows x 128 bytes and their scales, into a ring of its
 * own) run ahead through all of them, and the first ones start before the kernel that
 * makes x has finished.  The warps' sums meet in shared memory once, when the block's
 * tiles are done.  Eight warps, and at most half of an SM's registers and shared memory, so
 * that the block of the next projection is resident, and its ring full, before this one
 * leaves the SM.  (Slower, us a layer where this takes 44.5: one block of 16 warps an SM
 * 49.3, two of 12 warps 49.8, L2 asked for the rest of a block's rows at its start 58.)
 *
 * What bounds it: alone, 90000 x 4096 runs at 5.0 to 5.5 TB/s of weights (38 to 42 us; 81
 * before).  In a layer, a projection takes 1.1 us from the end of the kernel before to its
 * signal, 1.1 (4096 columns) to 3.2 (11008) for x, and then as long as its instructions
 * take: eight warps issue half the time, 8.6 us for the 22016 x 4096 of gate/up, of which
 * HBM would take 7.7.  Back to back in a graph, us: 12288 x 4096 7.8 to 9.3 (13.6 on bf16
 * mma.sync), 4096 x 4096 4.1 to 5.6 (6.7), 22016 x 4096 11.4 to 12.7 (23.1), 4096 x 11008
 * 8.6 to 10.3 (13.3).
 */
#ifndef VXB_ROWDOT_Q4_INT_CUH
#define VXB_ROWDOT_Q4_INT_CUH

constexpr int I_WARPS = 8;
constexpr int I_CODE_BYTES = 16 * 128;             /* of a step: 16 rows, 256 columns */
constexpr int I_STAGE_BYTES = I_CODE_BYTES + 256;  /* and 16 rows x eight f16 scales */

struct Q4IntPlan {
  int steps;  /* of 256 columns in a row */
  int slices; /* warps that share a tile's steps; the other factor of I_WARPS shares tiles */
  int round;  /* tiles between two meetings of the warps: 8 or 16 */
};

__device__ __forceinline__ void copy16_async(uint32_t dst, const void *src, uint64_t policy) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint.L2::128B [%0], [%1], 16, %2;" ::"r"(dst),
               "l"(src), "l"(policy)
               : "memory");
}

/* D = A * B + C on signed bytes; `start`: every element of C. */
__device__ __forceinline__ void mma_s8_from(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                            uint32_t a3, uint32_t b0, uint32_t b1, int start) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 "
               "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(start));
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float m;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
  return m;
}

/* Byte j of each of four words, for j = 0 .. 3, as a word each. */
__device__ __forceinline__ void transpose_bytes(uint32_t (&w)[4]) {
  const uint32_t a = __byte_perm(w[0], w[1], 0x5140), b = __byte_perm(w[2], w[3], 0x5140);
  const uint32_t c = __byte_perm(w[0], w[1], 0x7362), d = __byte_perm(w[2], w[3], 0x7362);
  w[0] = __byte_perm(a, b, 0x5410);
  w[1] = __byte_perm(a, b, 0x7632);
  w[2] = __byte_perm(c, d, 0x5410);
  w[3] = __byte_perm(c, d, 0x7632);
}

/* Shared memory: a ring per warp, then x (of each 64 columns 320 bytes: a byte of the eight
   columns of a lane, of the first 32 and of the second, is 16 bytes; of the four lanes of
   a byte, 64), then a factor for each 32 columns, then the warps' sums. */
__host__ __device__ inline size_t q4_int_ring(int stages) {
  return (size_t)I_WARPS * stages * I_STAGE_BYTES;
}
inline size_t q4_int_smem(int stages, int cols, const Q4IntPlan &plan) {
  return 128 + q4_int_ring(stages) + 5 * (size_t)cols + cols / 8 +
         sizeof(float2) * plan.round * plan.slices * 8;
}

/* The two results of an item with x in f32 as it is; every lane has them. A column of both
   rows to a lane at a time, and rolled: a case that hardly occurs, whose instructions cost
   every launch as they come from HBM with the others (eight columns at a time four times as
   fast here, and 1.5 % of a step). */
template <int EPI>
__device__ __forceinline__ float2 item_of_wide_x(const RowDotParams &p, int item) {
  const ItemRows it = item_rows<Q4W, EPI>(p, item);
  const int lane = threadIdx.x & 31;
  float t[2] = {0.0f, 0.0f};
#pragma unroll 1
  for (int c = lane; c < p.cols; c += 32) {
    float x = p.x[c];
    if (p.norm_w)
      x *= p.norm_bf16 ? bf16_at(p.norm_w, c) : ((const float *)p.norm_w)[c];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const char *codes = h && it.r1 ? it.r1 : it.r0, *scales = h && it.r1 ? it.sc1 : it.sc0;
      const int code = ((const unsigned char *)codes)[c / 2] >> (c % 2 * 4) & 15;
      t[h] = fmaf((float)(code - 8) * __half2float(((const __half *)scales)[c / 32]), x, t[h]);
    }
  }
  return make_float2(warp_sum(t[0]), warp_sum(t[1]));
}

template <int EPI, int STAGES>
__global__ void __launch_bounds__(I_WARPS * 32, 2)
q4_int_kernel(const RowDotParams p, const Q4IntPlan plan) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *smem = smem_raw + ((128 - (ptx::smem_addr(smem_raw) & 127)) & 127);
  __shared__ float ssq[I_WARPS];
  __shared__ __align__(16) int wide[I_WARPS]; /* x too far apart for whole numbers */
  const int cols = p.cols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  unsigned char *ring = smem + warp * (STAGES * I_STAGE_BYTES);
  unsigned char *xs = smem + q4_int_ring(STAGES);
  float *factors = reinterpret_cast<float *>(xs + 5 * (size_t)cols);
  float2 *parts = reinterpret_cast<float2 *>(factors + cols / 32); /* [tile][slice][8] */

  const int first = (int)((int64_t)blockIdx.x * p.items / gridDim.x);
  const int last = (int)((int64_t)(blockIdx.x + 1) * p.items / gridDim.x);
  const int tiles = (last - first + 7) / 8;
  const int apart = I_WARPS / plan.slices; /* a warp's tiles */
  const int slice = warp % plan.slices, tile0 = warp / plan.slices;
  const int u0 = slice * plan.steps / plan.slices;
  const int u1 = (slice + 1) * plan.steps / plan.slices;

  /* ---- the loading side: this lane's 16 bytes of four rows of codes (r0 and r1 of two
     items) and, of the first sixteen lanes, of one row of scales. The rows of a tile lie
     a fixed distance behind those of the warp's tile before (of q, k and v: until the
     half of a head ends). ---- */
  const int64_t row_bytes = cols / 2, scale_bytes = cols / 16;
  const int half = EPI == EPI_QKV ? p.head_dim / 2 : 1;
  struct Row {
    int row0, row1; /* of w0, of w1 or w0 */
    int in_half;    /* q, k and v */
  };
  auto row_of = [&](int item) {
    Row r;
    if (EPI == EPI_QKV) {
      const int head = item / half;
      r.in_half = item - head * half;
      r.row0 = head * p.head_dim + r.in_half;
      r.row1 = r.row0 + half;
    } else if (EPI == EPI_SWIGLU) {
      r.row0 = item;
      r.row1 = p.w1 ? item : p.rows + item;
    } else {
      r.row0 = 2 * item;
      r.row1 = 2 * item + 1;
    }
    return r;
  };
  auto advance = [&](Row &r) {
    const int by = 8 * apart * (EPI == EPI_STORE || EPI == EPI_ADD || EPI == EPI_BIAS ? 2 : 1);
    r.row0 += by;
    r.row1 += by;
    if (EPI == EPI_QKV)
      for (r.in_half += by; r.in_half >= half; r.in_half -= half) {
        r.row0 += half;
        r.row1 += half;
      }
  };
  const char *w0 = (const char *)p.w0 + (lane & 7) * 16;
  const char *w1 = EPI == EPI_SWIGLU && p.w1 ? (const char *)p.w1 + (lane & 7) * 16 : w0;
  const bool second = lane & 8; /* of the scales */
  const char *s0 = second && EPI == EPI_SWIGLU && p.w1
                       ? (const char *)p.s1
                       : (const char *)p.s0 + p.row_base * scale_bytes;
  const bool odd = EPI != EPI_SWIGLU && EPI != EPI_QKV; /* the last row may be missing */
  int ld_tile = tile0, ld_left = 0, ld_stage = 0;
  Row ld_rows[2] = {row_of(first + tile0 * 8 + (lane >> 3)),
                    row_of(first + tile0 * 8 + (lane >> 3) + 4)};
  Row ld_scales = row_of(first + tile0 * 8 + (lane & 7));
  const char *src[4] = {}, *src_scale = nullptr;
  bool have[4] = {}, have_scale = false;
  auto open_tile = [&]() {
    const int left = last - (first + ld_tile * 8); /* items of the tile */
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      have[h] = (lane >> 3) + 4 * h < left;
      have[2 + h] = have[h] && (!odd || ld_rows[h].row1 < p.rows);
      src[h] = w0 + ld_rows[h].row0 * row_bytes + u0 * 128;
      src[2 + h] = w1 + ld_rows[h].row1 * row_bytes + u0 * 128;
      advance(ld_rows[h]);
    }
    const int row = second ? ld_scales.row1 : ld_scales.row0;
    have_scale = lane < 16 && (lane & 7) < left && (!odd || row < p.rows);
    src_scale = s0 + row * scale_bytes + u0 * 16;
    advance(ld_scales);
    ld_left = u1 - u0;
  };
  /* 16-byte run c of a row sits at c ^ (row mod 8): no two of the eight rows that ldmatrix
     reads together share a bank */
  const uint32_t ring_at = ptx::smem_addr(ring);
  const uint32_t to0 = ring_at + (lane >> 3) * 128 + (((lane & 7) ^ (lane >> 3)) << 4);
  const uint32_t to1 = ring_at + ((lane >> 3) + 4) * 128 +
                       (((lane & 7) ^ ((lane >> 3) + 4)) << 4);
  const uint32_t to_scale = ring_at + I_CODE_BYTES + lane * 16;
  const uint64_t policy = ptx::evict_first();
  auto issue_next = [&]() {
    if (ld_tile < tiles) {
      const uint32_t at = ld_stage * I_STAGE_BYTES;
      if (have[0])
        copy16_async(to0 + at, src[0], policy);
      if (have[1])
        copy16_async(to1 + at, src[1], policy);
      if (have[2])
        copy16_async(to0 + at + 1024, src[2], policy);
      if (have[3])
        copy16_async(to1 + at + 1024, src[3], policy);
      if (have_scale)
        copy16_async(to_scale + at, src_scale, policy);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        src[i] += 128;
      src_scale += 16;
      ld_stage = ld_stage + 1 == STAGES ? 0 : ld_stage + 1;
      if (--ld_left == 0) {
        ld_tile += apart;
        if (ld_tile < tiles)
          open_tile();
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (u0 == u1)
    ld_tile = tiles;
  else if (ld_tile < tiles)
    open_tile();
  /* Settled weights do not depend on the kernel before this one: start them. */
  if (!p.weights_settled)
    chain_wait();
  for (int s = 0; s < STAGES; ++s)
    issue_next();
  chain_release();
  if (p.norm_w) /* nor do the norm's gains, which come from HBM once a step */
    for (int at = threadIdx.x * 128; at < cols * (p.norm_bf16 ? 2 : 4); at += I_WARPS * 32 * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)p.norm_w + at));
  chain_wait();

  /* ---- x, times the norm's gains if any, as whole numbers: a thread takes eight
     columns, four threads the 32 that share a factor ---- */
  float ss = 0.0f;
  bool far = false;
  constexpr int kApart = I_WARPS * 32 * 8;
  for (int c0 = threadIdx.x * 8; c0 < cols; c0 += 2 * kApart) {
    /* two runs' loads in flight at once: a trip to L2 is half a microsecond */
    float vs[2][8], ws[2][8];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = c0 + k * kApart;
      if (c >= cols)
        break;
      *reinterpret_cast<float4 *>(&vs[k][0]) = *reinterpret_cast<const float4 *>(p.x + c);
      *reinterpret_cast<float4 *>(&vs[k][4]) = *reinterpret_cast<const float4 *>(p.x + c + 4);
      if (!p.norm_w)
        continue;
      float *w = ws[k];
      if (p.norm_bf16) {
        /* (gains on an 8-byte boundary, as the other projection kernels take them) */
        const uint2 *b2 = reinterpret_cast<const uint2 *>((const uint16_t *)p.norm_w + c);
        const uint2 a = b2[0], b = b2[1];
        w[0] = bf_lo(a.x); w[1] = bf_hi(a.x); w[2] = bf_lo(a.y); w[3] = bf_hi(a.y);
        w[4] = bf_lo(b.x); w[5] = bf_hi(b.x); w[6] = bf_lo(b.y); w[7] = bf_hi(b.y);
      } else {
        *reinterpret_cast<float4 *>(&w[0]) =
            *reinterpret_cast<const float4 *>((const float *)p.norm_w + c);
        *reinterpret_cast<float4 *>(&w[4]) =
            *reinterpret_cast<const float4 *>((const float *)p.norm_w + c + 4);
      }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = c0 + k * kApart;
      if (c >= cols)
        break;
      float(&v)[8] = vs[k];
      if (p.norm_w)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          ss = fmaf(v[j], v[j], ss);
          v[j] *= ws[k][j];
        }
      float four[2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        four[h] = max_nan(max_nan(fabsf(v[4 * h]), fabsf(v[4 * h + 1])),
                          max_nan(fabsf(v[4 * h + 2]), fabsf(v[4 * h + 3])));
      float top = max_nan(four[0], four[1]);
      top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, 2));
      /* 2^s brings the largest into [2^29, 2^30). Below 2^-117 s stays: what is cut then
         lies below the smallest f32. In two factors: 2^s itself may be above the largest
         f32. Infinities and NaN make the factor, and so every result, NaN. */
      const int e = max((int)(__float_as_uint(top) >> 23 & 255u), 10);
      /* four neighbours, not all 0, that lie 2^-17 below the largest or further: the sums
         are then made from x itself */
      const uint32_t low = e == 255 ? 0u : (uint32_t)max(e - 16, 0) << 23;
      far |= __float_as_uint(four[0]) - 1u < low || __float_as_uint(four[1]) - 1u < low;
      if (e < 64)
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[j] *= 0x1p64f;
      const float up = __uint_as_float((uint32_t)(283 - e - (e < 64 ? 64 : 0)) << 23);
      uint32_t even[4], odd[4], even_rest = 0, odd_rest = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        /* signed bytes: 0x80 carried into the next one makes each byte its digit + 0x80;
           the fifth byte, of what the whole number leaves, is at most 127 / 256 */
        const float y = v[2 * j] * up, z = v[2 * j + 1] * up;
        const int yi = __float2int_rn(y), zi = __float2int_rn(z);
        const int yr = min(__float2int_rn((y - (float)yi) * 256.0f), 127);
        const int zr = min(__float2int_rn((z - (float)zi) * 256.0f), 127);
        even[j] = (uint32_t)yi + 0x00808080u;
        odd[j] = (uint32_t)zi + 0x00808080u;
        even_rest |= ((uint32_t)yr & 255u) << (8 * j);
        odd_rest |= ((uint32_t)zr & 255u) << (8 * j);
      }
      transpose_bytes(even);
      transpose_bytes(odd);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        even[j] ^= 0x80808080u;
        odd[j] ^= 0x80808080u;
      }
      unsigned char *at = xs + (c >> 6) * 320 + ((c >> 3) & 3) * 16 + ((c >> 5) & 1) * 8;
      *reinterpret_cast<uint2 *>(at) = make_uint2(even_rest, odd_rest);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint2 *>(at + 64 + j * 64) = make_uint2(even[j], odd[j]);
      /* 2^-s, less the 16 of the codes' bytes, times the 2^24 of the fourth byte */
      if ((c & 31) == 0)
        factors[c >> 5] = e == 255 ? __uint_as_float(0x7fc00000u)
                                   : __uint_as_float((uint32_t)(e - 9) << 23);
    }
  }
  far = __any_sync(0xffffffffu, far);
  if (lane == 0)
    wide[warp] = far;
  if (p.norm_w) {
    ss = warp_sum(ss);
    if (lane == 0)
      ssq[warp] = ss;
  }
  __syncthreads();
  float inv = 1.0f;
  if (p.norm_w) {
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < I_WARPS; ++w) /* fixed order */
      total += ssq[w];
    inv = 1.0f / sqrtf(total / (float)cols + p.eps);
  }

  /* what the results are added to or turned by: asked for now, not when they are there */
  float2 read = make_float2(0.0f, 0.0f);
  if ((int)threadIdx.x < plan.round * 8 && first + (int)threadIdx.x < last)
    read = before_item<EPI>(p, first + threadIdx.x);

  /* A lane has columns 2 t and 2 t + 1 of the results: the bytes of X from the fifth on
     (columns 5 to 7 are the largest byte's again, and not used). */
  const float d0 = t == 0 ? 0x1p-32f : t == 1 ? 0x1p-16f : t == 2 ? 1.0f : 0.0f;
  const float d1 = t == 0 ? 0x1p-24f : t == 1 ? 0x1p-8f : 0.0f;
  /* sums of 32 products are below 2^20: added to the bits of 1.5 * 2^23 they are the
     last bits of a float */
  constexpr int kMagic = 0x4B400000;
  const float2 magic = make_float2(-12582912.0f, -12582912.0f);
  const uint32_t matrix_at = (uint32_t)(((lane & 7) + (lane & 8)) * 128 +
                                        ((((lane >> 4) & 1) ^ (lane & 7)) << 4));
  const unsigned char *xb = xs + min(g, 4) * 64 + t * 16;
  int stage = 0;
  for (int round = 0; round < tiles; round += plan.round) {
    const int end = min(round + plan.round, tiles);
    /* round is a multiple of `apart` */
    for (int tile = round + tile0; tile < end; tile += apart) {
      float2 lo = make_float2(0.0f, 0.0f), hi = lo;
      for (int u = u0; u < u1; ++u) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory");
        __syncwarp();
        const unsigned char *st = ring + stage * I_STAGE_BYTES;
        const uint32_t codes = ptx::smem_addr(st) + matrix_at;
        const uint4 sl = *reinterpret_cast<const uint4 *>(st + I_CODE_BYTES + g * 16);
        const uint4 sh = *reinterpret_cast<const uint4 *>(st + I_CODE_BYTES + 128 + g * 16);
        const uint32_t slw[4] = {sl.x, sl.y, sl.z, sl.w};
        const uint32_t shw[4] = {sh.x, sh.y, sh.z, sh.w};
        float f[8];
        *reinterpret_cast<float4 *>(&f[0]) = *reinterpret_cast<const float4 *>(factors + u * 8);
        *reinterpret_cast<float4 *>(&f[4]) =
            *reinterpret_cast<const float4 *>(factors + u * 8 + 4);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          uint32_t r[4];
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                       : "r"(codes ^ (uint32_t)(m << 5))
                       : "memory");
          const uint4 bx = *reinterpret_cast<const uint4 *>(xb + (u * 4 + m) * 320);
          const float2 scale_lo = __half22float2(*reinterpret_cast<const __half2 *>(&slw[m]));
          const float2 scale_hi = __half22float2(*reinterpret_cast<const __half2 *>(&shw[m]));
          constexpr uint32_t M = 0xF0F0F0F0u, S = 0x80808080u;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t a = r[2 * h], b = r[2 * h + 1];
            int d[4];
            mma_s8_from(d, ((a << 4) & M) ^ S, ((b << 4) & M) ^ S, (a & M) ^ S, (b & M) ^ S,
                        h ? bx.z : bx.x, h ? bx.w : bx.y, kMagic);
            const float s_lo = (h ? scale_lo.y : scale_lo.x) * f[2 * m + h];
            const float s_hi = (h ? scale_hi.y : scale_hi.x) * f[2 * m + h];
            fma_pair(lo, add_pair(make_float2(__int_as_float(d[0]), __int_as_float(d[1])), magic),
                     make_float2(s_lo, s_lo));
            fma_pair(hi, add_pair(make_float2(__int_as_float(d[2]), __int_as_float(d[3])), magic),
                     make_float2(s_hi, s_hi));
          }
        }
        __syncwarp(); /* every lane has read the stage: it may be filled again */
        issue_next();
        stage = stage + 1 == STAGES ? 0 : stage + 1;
      }
      float v = fmaf(d1, lo.y, d0 * lo.x), w = fmaf(d1, hi.y, d0 * hi.x);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      w += __shfl_xor_sync(0xffffffffu, w, 1);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      w += __shfl_xor_sync(0xffffffffu, w, 2);
      if (t == 0)
        parts[((tile - round) * plan.slices + slice) * 8 + g] = make_float2(v, w);
    }
    __syncthreads();
    const int4 far0 = *reinterpret_cast<const int4 *>(&wide[0]);
    const int4 far1 = *reinterpret_cast<const int4 *>(&wide[4]);
    if (far0.x | far0.y | far0.z | far0.w | far1.x | far1.y | far1.z | far1.w) {
#pragma unroll 1
      for (int i = round * 8 + warp; i < end * 8 && first + i < last; i += I_WARPS) {
        const float2 t = item_of_wide_x<EPI>(p, first + i);
        if (lane < plan.slices) /* whose sum over the slices it is then */
          parts[((i / 8 - round) * plan.slices + lane) * 8 + i % 8] =
              lane ? make_float2(0.0f, 0.0f) : t;
      }
      __syncthreads();
    }
    const int item = first + round * 8 + threadIdx.x;
    if ((int)threadIdx.x < plan.round * 8 && item < last) {
      const float2 *at = parts + (threadIdx.x >> 3) * plan.slices * 8 + (threadIdx.x & 7);
      float2 total = at[0];
      for (int s = 1; s < plan.slices; ++s) { /* fixed order */
        total.x += at[s * 8].x;
        total.y += at[s * 8].y;
      }
      finish_item_with<EPI>(p, item, total.x * inv, total.y * inv, read);
      if (item + plan.round * 8 < last)
        read = before_item<EPI>(p, item + plan.round * 8);
    }
    if (end < tiles)
      __syncthreads();
  }
}

/* nullptr: launched; "": this projection is not for this kernel (the caller takes the one
   on the FMA pipe); anything else: an error. */
template <int EPI> const char *launch_q4_int(RowDotParams &p, cudaStream_t stream) {
  static const bool wanted = [] {
    const char *e = getenv("VXB_QUANT_MMA");
    return !(e && e[0] == '0');
  }();
  if (!wanted || p.batch != 1 || p.expert_ids || p.items < 1 || p.cols % 256 != 0)
    return "";
  if (EPI == EPI_QKV &&
      (p.rope_mode != 0 || p.w1 || p.w2 || (p.head_dim / 2) % 8 != 0))
    return "";
  if (((uintptr_t)p.w0 | (uintptr_t)p.w1 | (uintptr_t)p.s0 | (uintptr_t)p.s1) & 15)
    return "";
  Q4IntPlan plan;
  plan.steps = p.cols / 256;
  const int blocks = sm_count() < p.items ? sm_count() : p.items;
  /* the division of warps that leaves the busiest one the fewest steps */
  const int tiles = ((p.items + blocks - 1) / blocks + 7) / 8;
  int least = INT_MAX;
  for (int n = 1; n <= I_WARPS && n <= plan.steps; ++n) {
    const int apart = I_WARPS / n;
    if (n * apart != I_WARPS)
      continue;
    const int busiest = (tiles + apart - 1) / apart * ((plan.steps + n - 1) / n);
    if (busiest < least) {
      least = busiest;
      plan.slices = n;
    }
  }
  /* Two projections one after another share an SM's 228 KB, two blocks of one projection
     must not: another SM would be without. (Attention leaves SMs uneven. With 111 KB for
     all, gate/up took 14.7 us on SMs with two blocks, 8.5 on those with one, and the SMs
     with none waited: 58 us a layer of the 7B shape at 1000 positions, so 44.5.) So what
     follows attention or gate/up takes 115 KB, q/k/v and gate/up at most 111. */
  const size_t floor_bytes = EPI == EPI_QKV || EPI == EPI_SWIGLU ? 0 : 115 * 1024;
  const size_t share = EPI == EPI_QKV || EPI == EPI_SWIGLU ? 111 * 1024 : 115 * 1024;
  const size_t most = 226 * 1024;
  auto go = [&](auto kernel, size_t smem) -> const char * {
    if (allow_dynamic_smem((const void *)kernel, (int)most) != cudaSuccess)
      return "a Q4_0 projection could not get its shared memory on this GPU";
    prefer_shared_memory((const void *)kernel);
    launch_chained(kernel, dim3(blocks), dim3(I_WARPS * 32), std::max(smem, floor_bytes), stream, p,
                   plan);
    return check_launch("a Q4_0 projection launch");
  };
  plan.round = 16;
  if (q4_int_smem(3, p.cols, plan) > share)
    plan.round = 8;
  const size_t four = q4_int_smem(4, p.cols, plan), three = q4_int_smem(3, p.cols, plan);
  if (three > most)
    return "";
  if (four <= share || (three > share && four <= most))
    return go(q4_int_kernel<EPI, 4>, four);
  return go(q4_int_kernel<EPI, 3>, three);
}

#endif /* VXB_ROWDOT_Q4_INT_CUH */
