// y[M, N] = x[M, K] . W[N, K]^T of 32-bit values on the tensor cores, as exact as the fp32 pipes.
//
// Each value is the exact sum of three bfloat16 pieces (high, middle, low: 8 bits of significand each, rounded to
// nearest).  Of the nine products of pieces six are kept; the three left out are below 2^-26 of the product.  The tensor
// core multiplies pieces exactly but cuts its sums off (towards zero), a bias that would grow along K.  So:
//
//   * the products of high pieces (chunks of 32 k: two instructions from zero) leave the accumulator after every chunk and
//     are added up in registers, rounded to nearest;
//   * the five others, 2^-8 of the whole and less, keep two accumulators of their own over a span (an eighth of K, a multiple
//     of 64): high by middle with middle by high, and high by low, middle by middle, low by high.  The bits that these cut
//     off lie 2^-8 lower.
//
// A span's value is the first plus the sum of the two others, and the spans are added in order.  This order is fixed by K
// alone, so a row's result does not depend on the rows beside it, nor on the tile's width or the number of blocks that
// share K.  It is another order than that of the fp32 pipes, and a little nearer to the exact sum.  Measured against 64 bits,
// relative error of 300 rows of N(0, 1) with N(0, 0.02) (the fp32 pipes): K 2048 9.2e-8 (1.58e-7), K 8192 1.29e-7 (2.95e-7),
// K 14336 1.58e-7 (3.84e-7); where all products have one sign the bias shows, 6.0e-8 (4.5e-8) and 6.5e-8 (5.8e-8).
// An infinity, or a value that rounds to one, has pieces that are no numbers.  An output that comes out as NaN is therefore
// summed again on the fp32 pipes, by the thread that would store it.
#pragma once
#include <cooperative_groups.h>

#include "common.cuh"
#include "tcgen05.cuh"

namespace dlgo {

constexpr int SPLIT_SPANS = 8, SPLIT_K = 64;
__host__ __device__ __forceinline__ int split_span_length(int K) { return (K + SPLIT_SPANS * SPLIT_K - 1) / (SPLIT_SPANS * SPLIT_K) * SPLIT_K; }

__device__ int g_gemm_split_error = 0;      // set when a bounded wait ran out

// two neighbours of k -> their pieces, packed (the lower k in the lower half)
struct Pieces {
  uint32_t h, m, l;
};
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// {a, b} minus the two bfloat16 of h, exact where h is their rounding
__device__ __forceinline__ void less_bf16(float& a, float& b, uint32_t h) {
  asm("{\n\t"
      ".reg .b64 v, w, n;\n\t"
      ".reg .b32 lo, hi;\n\t"
      "mov.b64 v, {%0, %1};\n\t"
      "shl.b32 lo, %2, 16;\n\t"
      "and.b32 hi, %2, 0xffff0000;\n\t"
      "mov.b64 w, {lo, hi};\n\t"
      "mov.b64 n, 0xbf800000bf800000;\n\t"
      "fma.rn.f32x2 v, w, n, v;\n\t"
      "mov.b64 {%0, %1}, v;\n\t"
      "}\n"
      : "+f"(a), "+f"(b)
      : "r"(h));
}
__device__ __forceinline__ Pieces split_two(float a, float b) {
  Pieces p;
  p.h = pack_bf16(a, b);
  less_bf16(a, b, p.h);
  p.m = pack_bf16(a, b);
  less_bf16(a, b, p.m);
  p.l = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);        // (7 bits are left)
  return p;
}

__device__ __forceinline__ void add_two(float& a, float& b, float x, float y) {
  asm("{\n\t"
      ".reg .b64 v, w;\n\t"
      "mov.b64 v, {%0, %1};\n\t"
      "mov.b64 w, {%2, %3};\n\t"
      "add.rn.f32x2 v, v, w;\n\t"
      "mov.b64 {%0, %1}, v;\n\t"
      "}\n"
      : "+f"(a), "+f"(b)
      : "f"(x), "f"(y));
}

// the sum on the fp32 pipes, for outputs whose pieces are no numbers (inlined: a call costs the kernel registers, and 366 x
// 16384 x 2048 8 %)
__device__ __forceinline__ float split_plain_sum(const float* a, const float* w, int K) {
  float sum = 0.f;
#pragma unroll 1
  for (int k = 0; k < K; ++k) sum = fmaf(a[k], w[k], sum);
  return sum;
}

template <bool ADD>
__device__ __forceinline__ void split_finish(float* out, const float* A, const float* W, int K, int lda, int ldw, int ldo, int m, int n, float v) {
  if (v != v) v = split_plain_sum(A + (size_t)m * lda, W + (size_t)n * ldw, K);
  float* o = out + (size_t)m * ldo + n;
  *o = ADD ? *o + v : v;
}

// four values k .. k + 3 of a row (K is a multiple of 4), zero from K on and where the row does not exist
__device__ __forceinline__ float4 split_fetch(const float* row, int k, int K, bool live, bool aligned) {
  if (!live || k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (aligned) return *reinterpret_cast<const float4*>(row + k);
  return make_float4(row[k], row[k + 1], row[k + 2], row[k + 3]);
}

// x is split once, by a kernel of its own, into the tiles that the product copies: for every BN rows and 64 k the three
// pieces as they will lie in shared memory (rows of 128 bytes, 128-byte swizzle), zero where rows or k end.
template <int BN>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* A, uint8_t* tiles, int M, int K, int lda, int a_aligned) {
  pdl_launch_dependents();
  pdl_wait();
  const int chunks = gridDim.x, c = blockIdx.x, mt = blockIdx.y;
  uint8_t* tile = tiles + ((size_t)mt * chunks + c) * (3 * BN * 128);
#pragma unroll
  for (int i = 0; i < BN * 8 / 256; ++i) {
    const int at = threadIdx.x + 256 * i, r = at >> 3, u = at & 7, m = mt * BN + r, k = c * SPLIT_K + u * 8;
    const float* row = A + (size_t)m * lda;
    const float4 v = split_fetch(row, k, K, m < M, a_aligned != 0), w = split_fetch(row, k + 4, K, m < M, a_aligned != 0);
    const Pieces p0 = split_two(v.x, v.y), p1 = split_two(v.z, v.w), p2 = split_two(w.x, w.y), p3 = split_two(w.z, w.w);
    uint8_t* o = tile + r * 128 + ((u ^ (r & 7)) << 4);
    *reinterpret_cast<uint4*>(o) = make_uint4(p0.h, p1.h, p2.h, p3.h);
    *reinterpret_cast<uint4*>(o + BN * 128) = make_uint4(p0.m, p1.m, p2.m, p3.m);
    *reinterpret_cast<uint4*>(o + 2 * BN * 128) = make_uint4(p0.l, p1.l, p2.l, p3.l);
  }
}

// A block takes 128 weight rows (the MMA's M) times BN rows of x (its N) of a share of K's spans: all eight, or two or one of
// them, whose blocks are then a cluster and meet through distributed shared memory, each finishing a part of the tile.
//   warps 0-7   read the sums of a chunk out of tensor memory (a warp's own 32 lanes, half of the columns) into registers
//   warps 8-15  fetch the weight, two blocks of 64 k ahead, split it and lay the pieces out with the 128-byte swizzle
//   warp 16     one thread issues the MMAs of high pieces
//   warp 18     one thread issues the others: per 16 k high by middle | low (one instruction, twice as wide), middle by
//               high | middle, low by high; sums that take part in the same instruction lie side by side.  (One thread for
//               all waited for the chunk's sums to be read before it issued what does not need that: 200 -> 182 us)
//   warp 17     one thread copies the tiles of x
// Tensor memory: the sums of high products, the two others, and a place for the spans before.
// Bound by the chain weight -> pieces -> MMAs in two stages of shared memory, in which pieces are written and read at the
// same time (without the writes 10 % less; the tensor pipe is 40 % busy).  Measured on a B200, us a product in a row of them
// with x's split (on the fp32 pipes): 17 x 16384 x 2048 47 (121), 64 x 3072 x 2048 22 (53), 64 x 2048 x 8192 54 (177), 128 x
// 16384 x 2048 61 (226), 366 x 3072 x 2048 57 (142), 366 x 16384 x 2048 170 (613), 366 x 2048 x 8192 125 (340), 1500 x 2048 x
// 8192 362 (1,196: 139 TFLOP/s against 42, where the fp32 pipes give 74 at most).  Stages of 32 k (four, rows of 64 bytes)
// took 23 % longer for 128 rows a tile and 48 % for 64; 64 rows a tile for all sizes 30 % longer; the weight hinted into L2
// ahead, or fetched past L1, changed nothing or lost.
template <int BN> struct SplitShape {
  static constexpr int STAGES = BN >= 128 ? 2 : 3;
  static constexpr int W_PIECE = 128 * 128, X_PIECE = BN * 128;               // bytes: rows of 64 bfloat16
  static constexpr int STAGE = 3 * (W_PIECE + X_PIECE);
  static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
  static constexpr int TMEM = BN >= 128 ? 512 : 256;                           // 4 x BN columns
  static_assert(4 * BN <= TMEM && 2 * BN * 128 * 4 <= STAGES * STAGE, "");
};
constexpr int SPLIT_THREADS = 19 * 32;

// contiguous bytes into shared memory, counted on `bar` (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void split_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sm100::smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(sm100::smem_u32(bar))
               : "memory");
}

template <int BN, bool ADD>
__global__ void __launch_bounds__(SPLIT_THREADS, 1)
gemm_split_kernel(const float* A, const uint8_t* x_tiles, const float* W, float* out, int M, int N, int K, int lda, int ldw, int ldo,
                  int block_spans, int static_w) {
  namespace cg = cooperative_groups;
  using namespace sm100;
  using S = SplitShape<BN>;
  constexpr int STAGES = S::STAGES;
  extern __shared__ uint8_t split_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)split_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * S::STAGE);
  uint64_t* empty = full + STAGES;
  uint64_t* high_full = empty + STAGES;
  uint64_t* high_empty = high_full + 1;
  uint64_t* rest_full = high_empty + 1;
  uint64_t* rest_empty = rest_full + 1;
  uint32_t* tmem_slot = (uint32_t*)(rest_empty + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  pdl_launch_dependents();
  cg::cluster_group cl = cg::this_cluster();
  const int blocks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tile = (int)blockIdx.x / blocks;
  const int m_tiles = (M + BN - 1) / BN;                      // blocks of the same weight rows follow one another
  const int m0 = (tile % m_tiles) * BN, n0 = (tile / m_tiles) * 128;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int span = split_span_length(K), span_chunks = span / SPLIT_K;
  const int k_begin = rank * block_spans * span, k_end = min(K, k_begin + block_spans * span);
  const int chunks = (k_end - k_begin + SPLIT_K - 1) / SPLIT_K;                                  // (no block without k)

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 9);
      mbar_init(&empty[s], 2);
    }
    mbar_init(high_full, 1);
    mbar_init(high_empty, 8);
    mbar_init(rest_full, 1);
    mbar_init(rest_empty, 8);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 16) {
    tmem_alloc(tmem_slot, S::TMEM);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const uint32_t t_rest = tmem + BN, t_before = tmem + 3 * BN;

  if (warp >= 8 && warp < 16) {
    // a lane: four k at 16 j + 4 (lane & 3) of rows `row` + 8 i; half a warp's rows are two apart, so that its 8-byte pieces
    // fill all banks
    const int quad = lane & 3, row = (warp - 8) * 16 + ((lane >> 2) & 3) * 2 + (lane >> 4);
    float4 wv[2][2][4];
    const float* w_row = W + (size_t)(n0 + row) * ldw + k_begin + 4 * quad;
    const bool rows_whole = n0 + 128 <= N;
    auto fetch = [&](int c, float4 (&v)[2][4]) {
      const float* at = w_row + c * SPLIT_K;
      if (rows_whole && k_begin + (c + 1) * SPLIT_K <= k_end) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) v[i][j] = *reinterpret_cast<const float4*>(at + (size_t)i * 8 * ldw + 16 * j);
        return;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[i][j] = split_fetch(at + (size_t)i * 8 * ldw + 16 * j - 4 * quad, 4 * quad, k_end - k_begin - c * SPLIT_K - 16 * j, n0 + row + i * 8 < N, true);
    };
    auto put = [&](int c, const float4 (&v)[2][4]) {
      const int s = c % STAGES;
      if (c >= STAGES && !mbar_wait(&empty[s], ((c / STAGES) & 1) ^ 1, abort_flag)) return false;
      uint8_t* at = smem + s * S::STAGE + row * 128 + ((quad & 1) << 3);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const Pieces a = split_two(v[i][j].x, v[i][j].y), b = split_two(v[i][j].z, v[i][j].w);
          uint8_t* p = at + i * 1024 + (((2 * j + (quad >> 1)) ^ (row & 7)) << 4);
          *reinterpret_cast<uint2*>(p) = make_uint2(a.h, b.h);
          *reinterpret_cast<uint2*>(p + S::W_PIECE) = make_uint2(a.m, b.m);
          *reinterpret_cast<uint2*>(p + 2 * S::W_PIECE) = make_uint2(a.l, b.l);
        }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[s]);
      return true;
    };
    if (!static_w) pdl_wait();      // (W may come from the launch before)
    fetch(0, wv[0]);
    if (chunks > 1) fetch(1, wv[1]);
    for (int c = 0; c < chunks; c += 2) {
      if (!put(c, wv[0])) break;
      if (c + 2 < chunks) fetch(c + 2, wv[0]);
      if (c + 1 >= chunks || !put(c + 1, wv[1])) break;
      if (c + 3 < chunks) fetch(c + 3, wv[1]);
    }
  } else if (warp == 17) {
    if (elect_one()) {
      pdl_wait();
      const uint8_t* src = x_tiles + ((size_t)(m0 / BN) * ((K + SPLIT_K - 1) / SPLIT_K) + k_begin / SPLIT_K) * (3 * S::X_PIECE);
      for (int c = 0; c < chunks; ++c) {
        const int s = c % STAGES;
        if (c >= STAGES && !mbar_wait(&empty[s], ((c / STAGES) & 1) ^ 1, abort_flag)) break;
        mbar_expect_tx(&full[s], 3 * S::X_PIECE);
        split_bulk_load(smem + s * S::STAGE + 3 * S::W_PIECE, src + (size_t)c * (3 * S::X_PIECE), 3 * S::X_PIECE, &full[s]);
      }
    }
  } else if (warp == 16) {
    if (elect_one()) {                                        // the products of high pieces
      constexpr uint32_t one = umma_idesc_bf16(128, BN);
      const uint64_t dw0 = umma_desc_k_sw128(smem_u32(smem)), dx0 = umma_desc_k_sw128(smem_u32(smem + 3 * S::W_PIECE));
      bool ok = true;
      for (int c = 0, s = 0, turn = 0; c < chunks && ok; ++c) {
        if (!mbar_wait(&full[s], turn, abort_flag)) break;
        const uint64_t at = (uint64_t)(s * (S::STAGE >> 4));
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          if (c + half > 0 && !mbar_wait(high_empty, half ^ 1, abort_flag)) { ok = false; break; }
          tc_fence_after_sync();
#pragma unroll
          for (int k = 0; k < 2; ++k) umma_bf16(tmem, dw0 + at + 2 * (2 * half + k), dx0 + at + 2 * (2 * half + k), one, k != 0);
          umma_commit(high_full);
        }
        umma_commit(&empty[s]);
        if (++s == STAGES) { s = 0; turn ^= 1; }
      }
    }
  } else if (warp == 18) {
    if (elect_one()) {                                        // the others
      constexpr uint32_t one = umma_idesc_bf16(128, BN), two = umma_idesc_bf16(128, 2 * BN);
      const uint64_t dw0 = umma_desc_k_sw128(smem_u32(smem)), dx0 = umma_desc_k_sw128(smem_u32(smem + 3 * S::W_PIECE));
      constexpr uint64_t WP = S::W_PIECE >> 4, XP = S::X_PIECE >> 4;
      int in_span = 0, sp = 0;
      for (int c = 0, s = 0, turn = 0; c < chunks; ++c) {
        if (!mbar_wait(&full[s], turn, abort_flag)) break;
        if (in_span == 0 && c > 0 && !mbar_wait(rest_empty, (sp - 1) & 1, abort_flag)) break;
        tc_fence_after_sync();
        const uint64_t dw = dw0 + (uint64_t)(s * (S::STAGE >> 4)), dx = dx0 + (uint64_t)(s * (S::STAGE >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          umma_bf16(t_rest, dw + 2 * k, dx + XP + 2 * k, two, (k | in_span) != 0);
          umma_bf16(t_rest, dw + WP + 2 * k, dx + 2 * k, two, true);
          umma_bf16(t_rest + BN, dw + 2 * WP + 2 * k, dx + 2 * k, one, true);
        }
        umma_commit(&empty[s]);
        if (in_span == span_chunks - 1 || c == chunks - 1) umma_commit(rest_full);
        if (++in_span == span_chunks) {
          in_span = 0;
          ++sp;
        }
        if (++s == STAGES) { s = 0; turn ^= 1; }
      }
    }
  } else {
    constexpr int COLS = BN / 2;                              // of this warp, 16 at a time
    const int col0 = (warp >> 2) * COLS;
    const uint32_t mine = ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
    float run[COLS];
    bool ok = true;
    int in_span = 0, sp = 0;
    for (int c = 0; c < chunks && ok; ++c) {
      if (in_span == 0) {
#pragma unroll
        for (int j = 0; j < COLS; ++j) run[j] = 0.f;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if (!mbar_wait(high_full, half, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
#pragma unroll
        for (int g = 0; g < COLS; g += 16) {
          float v[16];
          tmem_ld_32x16(tmem + mine + g, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; j += 2) add_two(run[g + j], run[g + j + 1], v[j], v[j + 1]);
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(high_empty);
      }
      if (!ok) break;
      if (in_span == span_chunks - 1 || c == chunks - 1) {
        if (!mbar_wait(rest_full, sp & 1, abort_flag)) { ok = false; break; }
        tc_fence_after_sync();
#pragma unroll
        for (int g = 0; g < COLS; g += 8) {                   // (16 at a time and the sums do not fit 96 registers)
          float v[8], u[8];
          tmem_ld_32x8(t_rest + mine + g, v);
          tmem_ld_32x8(t_rest + BN + mine + g, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) run[g + j] += v[j] + u[j];
          if (sp > 0 && blocks == 1) {                        // one block adds its spans up; more keep them apart
            tmem_ld_32x8(t_before + mine + g, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j) run[g + j] = v[j] + run[g + j];
          }
          if (c != chunks - 1) tmem_st_32x8(t_before + mine + g, run + g);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(rest_empty);
      }
      if (++in_span == span_chunks) {
        in_span = 0;
        ++sp;
      }
    }
    if (ok) {
      // every MMA has finished: the ring becomes the tile [span][BN][128]
      float* sums = reinterpret_cast<float*>(smem) + (warp & 3) * 32 + lane;
      const int last = blocks == 1 ? 0 : (chunks - 1) / span_chunks;
#pragma unroll
      for (int j = 0; j < COLS; ++j) sums[(last * BN + col0 + j) * 128] = run[j];
      if (last > 0) {                                         // (two spans a block)
#pragma unroll
        for (int g = 0; g < COLS; g += 16) {
          float v[16];
          tmem_ld_32x16(t_before + mine + g, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) sums[(col0 + g + j) * 128] = v[j];
        }
      }
    }
  }
  __syncwarp();
  pdl_wait();
  tc_fence_before_sync();
  if (*abort_flag)                  // what may still be running gets time to finish before its memory is handed on
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  if (blocks > 1) cl.sync(); else __syncthreads();
  if (warp == 16) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, S::TMEM);
  }
  if (*abort_flag) {
    if (tid == 0) atomicExch(&g_gemm_split_error, 1);
  } else if (tid < 512) {
    // lane: output, then row of x; this block's part of the rows
    float* sums = reinterpret_cast<float*>(smem);
    const int r = tid & 127, n = n0 + r, spans = blocks == 1 ? 1 : (K + span - 1) / span;
    for (int t = rank * 4 + (tid >> 7); t < BN; t += 4 * blocks) {
      const int m = m0 + t;
      if (m >= M) break;
      float v;
      if (blocks == 1) {
        v = sums[t * 128 + r];
      } else {
        v = *cl.map_shared_rank(sums + t * 128 + r, 0);
        for (int q = 1; q < spans; ++q) v += *cl.map_shared_rank(sums + ((q % block_spans) * BN + t) * 128 + r, q / block_spans);
      }
      if (n < N) split_finish<ADD>(out, A, W, K, lda, ldw, ldo, m, n, v);
    }
  }
  if (blocks > 1) cl.sync();        // nobody leaves while its sums may still be read
}

}  // namespace dlgo
