// y[M, N] = x[M, K] . W[N, K]^T on the fp32 pipes (FFMA), for every size.
//
// This is the contraction of the true 32-bit path (no tensor cores, no
// reduced-precision matrix mode), the plain counterpart the tensor-core kernel
// is checked against, and the stand-in where the tensor-core kernel refuses a
// size.  The reference contracts one weight row with the activation vector per
// output (blas/blas.go:152-196, models/llm/forward.go:224,286,296-298).
//
// The order of an output's sum is fixed by K alone and the same in both kernels below, so a row's result does not
// depend on the other rows of the launch, nor on which kernel ran.  K is cut into 16 spans of equal length (a multiple of
// 32; the last ones may be short or empty).  Within a span the products of even k and those of odd k are two running
// sums: one packed fp32 pair, since fma.rn.f32x2 takes two neighbours of k straight from rows as they lie, so nothing is
// transposed or duplicated.  A span's value is their sum; four spans are added up in order, and so are the four quarters.
//
// Epilogues: store in the activation type, store fp32 (logits), or add into an
// fp32 residual in place (models/llm/forward.go:163,169).
#include <cooperative_groups.h>

#include <atomic>

#include "async_copy.cuh"
#include "common.cuh"

namespace dlgo {

enum { EPI_STORE = 0, EPI_STORE_F32 = 1, EPI_ADD_F32 = 2 };
constexpr int SPANS = 16, QUARTER = SPANS / 4;
__host__ __device__ __forceinline__ int span_length(int K) { return (K + SPANS * 32 - 1) / (SPANS * 32) * 32; }

// acc (even k, odd k) += a * b over two, and over four, neighbours of k
__device__ __forceinline__ void fma_two(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ void fma_four(unsigned long long& acc, const ulonglong2& a, const ulonglong2& b) {
  fma_two(acc, a.x, b.x);
  fma_two(acc, a.y, b.y);
}
__device__ __forceinline__ float pair_sum(unsigned long long acc) {
  float even, odd;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(even), "=f"(odd) : "l"(acc));
  return even + odd;
}

// Four values k .. k + 3 of a row into shared memory as fp32, zero from K on or where the row does not exist.
// VEC: fp32 rows whose pieces of four are aligned and whole; the copy is asynchronous.
template <typename T, bool VEC>
__device__ __forceinline__ void stage_four(float* dst, const T* row, int k, int K, bool live) {
  if constexpr (VEC) {
    if (live && k < K) copy16_async(dst, (const float*)row + k);
    else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) {
      if (k < K) v.x = to_float(row[k]);
      if (k + 1 < K) v.y = to_float(row[k + 1]);
      if (k + 2 < K) v.z = to_float(row[k + 2]);
      if (k + 3 < K) v.w = to_float(row[k + 3]);
    }
    *reinterpret_cast<float4*>(dst) = v;
  }
}

template <typename T, int EPI>
__device__ __forceinline__ void finish(void* out, size_t at, float v) {
  if (EPI == EPI_STORE) ((T*)out)[at] = from_float<T>(v);
  else if (EPI == EPI_STORE_F32) ((float*)out)[at] = v;
  else ((float*)out)[at] += v;
}

// ------------------------------------------------------------------ many rows
// Bound by the fp32 pipes and, as closely, by what shared memory delivers to registers (128 bytes a clock, broadcast or
// not): 8 x 8 outputs per thread need 16 words of 16 bytes for 128 packed multiply-adds, 64 clocks of either.  A warp
// takes 64 x 32 outputs, a block of two warps 64 x 64, four blocks an SM; the four quarters of K are the blocks of a
// cluster (as many as are not empty), which evens out the last wave, and meet through distributed shared memory.  A
// thread's pairs take 128 registers; the sum over a quarter's spans waits in shared memory, a slot per output and thread.
// Rows lie in a ring of three stages of 16 k, 20 floats apart: the rows that a quarter warp reads are on different banks.
// Measured on a B200 (TFLOP/s): 567 x 16384 x 2048 41, 567 x 2048 x 8192 35, 64 x 16384 x 2048 34; 567 x 8192 x 2048 40,
// 567 x 2048 x 2048 33, 64 x 8192 x 2048 35.  64 x 64 outputs of scalar multiply-adds with a synchronous load of every 16 k
// (before) gave 24, 11 and 10 for the last three.  Blocks of 128 x 64 with four warps and four stages, two an SM, have as
// many warps there and more padding: 36, 34 and 19 for the first three; scalar multiply-adds in this layout 29 where
// packed ones give 38; 8 x 4 outputs per thread with twelve warps an SM and no cluster 36 and 20 for 366 rows.  The order
// of the multiply-adds and the width of the loads from shared memory change less than 2 %.  The fp32 pipes give 74 at most.
// (The figures above are VEC's.)  Rows that are no whole aligned pieces of fp32 (odd sizes, and bfloat16, for which this is
// the stand-in) cannot be copied asynchronously, and a block of two warps waits for the 32 loads a thread that it needs
// every 16 k: four warps of 8 x 4 outputs a thread instead, which fetch their next 16 values into registers while they
// multiply; rows 18 floats apart for their pattern.  Measured, us, bfloat16 / fp32 (K 2050 / 2051): 567 x 8192 766 / 716,
// 200 x 2048 102 / 98, 64 x 1024 48 / 46; two warps of 8 x 8 with loads waited for 1,171 / 1,317 (567 x 8192); one sum per output
// in 64 x 64 blocks of eight warps (before) 785 / 718, 193 / 186 and 152 / 137.  Eight warps of 4 x 4 outputs: 882 / 874,
// 124 / 129, 46 / 50; two of 8 x 8 with the loads a step ahead 964 / 772, 120 / 98, 80 / 63; three blocks an SM 870 / 745.
constexpr int BM = 64, BN = 64, KSTEP = 16;
template <bool VEC> struct TileShape {
  static constexpr int THREADS = VEC ? 64 : 128, BLOCKS = 4;                // (blocks an SM)
  static constexpr int TM = 8, TN = VEC ? 8 : 4;
  static constexpr int ROW = VEC ? KSTEP + 4 : KSTEP + 2;                   // floats from one staged row to the next
  static constexpr int STAGES = VEC ? 3 : 2;
  static constexpr int RING = STAGES * (BM + BN) * ROW;                     // floats
  static constexpr int SMEM = (RING + BM * BN) * 4;
  static constexpr int GROUPS = TM * TN / 4;                                // of four outputs of a thread
  static constexpr int ROWS = THREADS / 16, LOADS = BM / ROWS;              // without VEC: rows at a time, values a thread
};

template <typename T, int EPI, bool VEC>
__global__ void __launch_bounds__(TileShape<VEC>::THREADS, TileShape<VEC>::BLOCKS)
gemm_simt_tile_kernel(const T* A, const T* W, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w) {
  namespace cg = cooperative_groups;
  using S = TileShape<VEC>;
  constexpr int THREADS = S::THREADS, TM = S::TM, TN = S::TN, ROW = S::ROW, STAGES = S::STAGES, GROUPS = S::GROUPS;
  extern __shared__ __align__(16) float ring[];
  float4* sums = reinterpret_cast<float4*>(ring + S::RING);   // [GROUPS][THREADS]: of thread t's output row i, columns 4 h .. 4 h + 3 at i * TN / 4 + h
  pdl_launch_dependents();
  cg::cluster_group cl = cg::this_cluster();
  const int quarters = (int)cl.num_blocks(), quarter = (int)cl.block_rank();
  const int tile = (int)blockIdx.x / quarters;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m_tiles = (M + BM - 1) / BM;                      // blocks of the same weight rows follow one another
  const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * BN;
  // a thread's outputs: rows tm + 8 i, columns tn + col_of(j)
  const int tm = VEC ? lane >> 2 : tid >> 4, tn = VEC ? warp * 32 + (lane & 3) * 2 : tid & 15;
  auto col_of = [](int j) { return VEC ? (j & 1) + 8 * (j >> 1) : 16 * j; };
  const int span = span_length(K);
  const int k_begin = quarter * QUARTER * span, k_end = min(K, k_begin + QUARTER * span);
  const int steps = (k_end - k_begin + KSTEP - 1) / KSTEP;    // (quarters that exist are not empty)
  const int span_steps = span / KSTEP;
  // VEC: four k of rows vrow + 16 i straight into the ring
  const int vrow = tid >> 2, vk = (tid & 3) * 4;
  auto copy_rows = [&](const T* rows, int ld, int first, int count, int step, int at) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = vrow + 16 * i;
      stage_four<T, true>(ring + ((step % STAGES) * (BM + BN) + at + r) * ROW + vk, rows + (size_t)(first + r) * ld,
                          k_begin + step * KSTEP + vk, K, first + r < count);
    }
  };
  // else: one k of rows erow + S::ROWS i, through registers
  const int erow = tid >> 4, ek = tid & 15;
  T next[2][VEC ? 1 : S::LOADS];                              // (A, W)
  auto fetch_rows = [&](const T* rows, int ld, int first, int count, int step, T (&x)[VEC ? 1 : S::LOADS]) {
    const int k = k_begin + step * KSTEP + ek;
#pragma unroll
    for (int i = 0; i < S::LOADS; ++i) {
      const int r = first + erow + S::ROWS * i;
      x[i] = r < count && k < K ? rows[(size_t)r * ld + k] : from_float<T>(0.f);
    }
  };
  auto put_rows = [&](int step) {
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
      for (int i = 0; i < S::LOADS; ++i)
        ring[((step % STAGES) * (BM + BN) + o * BM + erow + S::ROWS * i) * ROW + ek] = to_float(next[o][i]);
  };
  if (!static_w) pdl_wait();    // (W may come from the launch before)
  if constexpr (VEC) {
    for (int s = 0; s < STAGES - 1 && s < steps; ++s) copy_rows(W, ldw, n0, N, s, BM);
    pdl_wait();
    for (int s = 0; s < STAGES - 1; ++s) {
      if (s < steps) copy_rows(A, lda, m0, M, s, 0);
      copies_commit();
    }
  } else {
    fetch_rows(W, ldw, n0, N, 0, next[1]);
    pdl_wait();
    fetch_rows(A, lda, m0, M, 0, next[0]);
    put_rows(0);
  }
  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
  int in_span = 0;
  bool first = true;
  for (int s = 0; s < steps; ++s) {
    if constexpr (VEC) copies_wait<STAGES - 2>();
    __syncthreads();            // stage s is in place, and every warp is past stage s - 1
    if constexpr (VEC) {
      if (s + STAGES - 1 < steps) {
        copy_rows(W, ldw, n0, N, s + STAGES - 1, BM);
        copy_rows(A, lda, m0, M, s + STAGES - 1, 0);
      }
      copies_commit();
    } else if (s + 1 < steps) {
      fetch_rows(W, ldw, n0, N, s + 1, next[1]);
      fetch_rows(A, lda, m0, M, s + 1, next[0]);
    }
    const float* as = ring + ((s % STAGES) * (BM + BN) + tm) * ROW;
    const float* ws = ring + ((s % STAGES) * (BM + BN) + BM + tn) * ROW;
    // two neighbours of k at a time; the next two are on their way from shared memory while these are multiplied
    unsigned long long a[2][TM], b[2][TN];
    auto fetch = [&](int k, unsigned long long (&x)[TM], unsigned long long (&y)[TN]) {
#pragma unroll
      for (int j = 0; j < TN; ++j) y[j] = *reinterpret_cast<const unsigned long long*>(ws + col_of(j) * ROW + k);
#pragma unroll
      for (int i = 0; i < TM; ++i) x[i] = *reinterpret_cast<const unsigned long long*>(as + 8 * i * ROW + k);
    };
    fetch(0, a[0], b[0]);
#pragma unroll
    for (int k = 0; k < KSTEP; k += 2) {
      const int now = (k >> 1) & 1;
      if (k + 2 < KSTEP) fetch(k + 2, a[now ^ 1], b[now ^ 1]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int jj = 0; jj < TN; ++jj) {
          const int j = (i & 1) ? TN - 1 - jj : jj;     // (a row after another shares an operand at the turn)
          fma_two(acc[i][j], a[now][i], b[now][j]);
        }
    }
    if constexpr (!VEC) {
      if (s + 1 < steps) put_rows(s + 1);               // (where stage s - 1 was)
    }
    if (++in_span == span_steps || s == steps - 1) {
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) {
        float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : sums[g * THREADS + tid];
        unsigned long long* q = &acc[g / (TN / 4)][g % (TN / 4) * 4];
        v.x += pair_sum(q[0]); v.y += pair_sum(q[1]); v.z += pair_sum(q[2]); v.w += pair_sum(q[3]);
        sums[g * THREADS + tid] = v;
        q[0] = q[1] = q[2] = q[3] = 0ull;
      }
      in_span = 0;
      first = false;
    }
  }
  // Every block of the cluster finishes a share of the tile; what is added into is fetched while the others arrive.
  auto store = [&](int g, const float4& v, const float* added) {            // group g of this thread's outputs
    const float f[4] = {v.x, v.y, v.z, v.w};
    const int m = m0 + tm + 8 * (g / (TN / 4)), n = n0 + tn + col_of(g % (TN / 4) * 4);
    if (m >= M) return;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int ne = n + col_of(e);
      if (ne >= N) continue;
      if (added != nullptr) ((float*)out)[(size_t)m * ldo + ne] = added[e] + f[e];
      else finish<T, EPI>(out, (size_t)m * ldo + ne, f[e]);
    }
  };
  if (quarters == 1) {
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) store(g, sums[g * THREADS + tid], nullptr);
    return;
  }
  float old[GROUPS / 4][4];
  if (EPI == EPI_ADD_F32 && quarters == 4) {
#pragma unroll
    for (int i = 0; i < GROUPS / 4; ++i) {
      const int g = quarter + 4 * i, m = m0 + tm + 8 * (g / (TN / 4)), n = n0 + tn + col_of(g % (TN / 4) * 4);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        old[i][e] = m < M && n + col_of(e) < N ? ((const float*)out)[(size_t)m * ldo + n + col_of(e)] : 0.f;
    }
  }
  cl.sync();
  auto share = [&](int g, const float* added) {
    float4 v = *cl.map_shared_rank(sums + g * THREADS + tid, 0);
    for (int q = 1; q < quarters; ++q) {
      const float4 u = *cl.map_shared_rank(sums + g * THREADS + tid, q);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    store(g, v, added);
  };
  if (quarters == 4) {
#pragma unroll
    for (int i = 0; i < GROUPS / 4; ++i) share(quarter + 4 * i, EPI == EPI_ADD_F32 ? old[i] : nullptr);
  } else {
    for (int g = quarter; g < GROUPS; g += quarters) share(g, nullptr);
  }
  cl.sync();                    // nobody leaves while its sums may still be read
}

// ------------------------------------------------------------------- few rows
// Bound by the weight, which is read once.  A block of eight warps takes 16 outputs at a time, a lane per output and
// span of K.  A lane's piece of a row is 128 bytes of a stage; the warp copies its 32 pieces (whole lines) and its spans
// of x itself, so that the ring needs no barrier of the block and goes on over the ends of tiles (one block per SM,
// tiles handed out in turn).  The spans meet in shared memory, where a thread per output and row of x adds them up.
// 16-byte words of a piece are permuted by the lane, so that eight lanes read all banks.
// Measured on a B200, two rows: 16384 x 2048 23 us (5.7 TB/s of weight; 64 x 64 tiles 405 us before), 2048 x 8192 13 us
// (555 us), 128256 x 2048 170 us (1.1 ms).  From 8 rows on, fetching x from shared memory counts as much: 32 us and, at
// 16 rows, 52 us for 16384 x 2048.
constexpr int FEW_ROWS = 16, FEW_WARPS = SPANS / 2, KSUB = 32;
template <int MT> struct FewShape {
  static constexpr int XHALF = MT * KSUB + 4;                 // floats of one span's x; the two spans on other banks
  static constexpr int STAGE = 32 * KSUB + 2 * XHALF;         // floats
  static constexpr int STAGES = MT <= 2 ? 5 : (MT <= 8 ? 4 : 3);
  static constexpr int SUMS = SPANS * FEW_ROWS * MT;          // floats, twice
  static constexpr int SMEM = (FEW_WARPS * STAGES * STAGE + 2 * SUMS) * 4;
};

template <typename T, int EPI, int MT, bool VEC>
__global__ void __launch_bounds__(FEW_WARPS * 32, 1)
gemm_simt_few_kernel(const T* A, const T* W, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w) {
  using S = FewShape<MT>;
  extern __shared__ __align__(16) float ring[];
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float* mine = ring + warp * S::STAGES * S::STAGE;
  float* sums = ring + FEW_WARPS * S::STAGES * S::STAGE;
  const int m0 = blockIdx.y * MT;
  const int tiles = (N + FEW_ROWS - 1) / FEW_ROWS;
  const int span = span_length(K), k0 = warp * 2 * span;
  const int subs = k0 < K ? min(span, K - k0 + KSUB - 1) / KSUB : 0;     // stages of a tile: the warp's longer span
  const int my_tiles = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  auto load_w = [&](int tile, int sub, int slot) {
    float* st = mine + slot * S::STAGE;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int seg = i * 4 + (lane >> 3), piece = lane & 7;
      const int n = tile * FEW_ROWS + (seg & 15), k = k0 + (seg >> 4) * span + sub * KSUB + piece * 4;
      stage_four<T, VEC>(st + seg * KSUB + ((piece ^ (seg & 7)) << 2), W + (size_t)n * ldw, k, K, n < N);
    }
  };
  auto load_x = [&](int sub, int slot) {
    float* st = mine + slot * S::STAGE + 32 * KSUB;
#pragma unroll
    for (int i = 0; i < (MT + 1) / 2; ++i) {
      const int seg = i * 4 + (lane >> 3), piece = lane & 7;    // two spans of a row of x, then the next row
      const int m = seg >> 1;
      if (MT == 1 && m >= 1) continue;
      stage_four<T, VEC>(st + (seg & 1) * S::XHALF + m * KSUB + piece * 4, A + (size_t)(m0 + m) * lda,
                         k0 + (seg & 1) * span + sub * KSUB + piece * 4, K, m0 + m < M);
    }
  };
  int left = my_tiles * subs;                 // the loader walks (tile, sub) ahead of the sums
  int l_tile = blockIdx.x, l_sub = 0, l_slot = S::STAGES - 1;
  auto step_on = [&](int& tile, int& sub) {
    if (++sub == subs) {
      sub = 0;
      tile += gridDim.x;
    }
  };
  if (!static_w) pdl_wait();    // (W may come from the launch before)
  {
    int tile = l_tile, sub = 0;
    for (int i = 0; i < S::STAGES - 1 && i < left; ++i) {
      load_w(tile, sub, i);
      step_on(tile, sub);
    }
  }
  pdl_wait();
  for (int i = 0; i < S::STAGES - 1; ++i) {
    if (left > 0) {
      load_x(l_sub, i);
      step_on(l_tile, l_sub);
      --left;
    }
    copies_commit();
  }
  int slot = 0, buf = 0;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    unsigned long long acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = 0ull;
    for (int sub = 0; sub < subs; ++sub) {
      copies_wait<S::STAGES - 2>();
      __syncwarp();             // the stage is in place, and every lane is past the one before
      if (left > 0) {
        load_w(l_tile, l_sub, l_slot);
        load_x(l_sub, l_slot);
        step_on(l_tile, l_sub);
        --left;
      }
      copies_commit();
      l_slot = l_slot + 1 == S::STAGES ? 0 : l_slot + 1;
      const float* st = mine + slot * S::STAGE;
      const float* xs = st + 32 * KSUB + (lane >> 4) * S::XHALF;
#pragma unroll
      for (int j = 0; j < KSUB / 4; ++j) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(st + lane * KSUB + ((j ^ (lane & 7)) << 2));
#pragma unroll
        for (int m = 0; m < MT; ++m) fma_four(acc[m], *reinterpret_cast<const ulonglong2*>(xs + m * KSUB + j * 4), w);
      }
      slot = slot + 1 == S::STAGES ? 0 : slot + 1;
    }
    float* sb = sums + buf * S::SUMS + (warp * 2 + (lane >> 4)) * FEW_ROWS * MT + (lane & 15);
#pragma unroll
    for (int m = 0; m < MT; ++m) sb[m * FEW_ROWS] = pair_sum(acc[m]);
    __syncthreads();            // (the buffer of the tile before is free once all are here: there are two)
    if (tid < FEW_ROWS * MT) {
      const float* sr = sums + buf * S::SUMS + tid;
      float c[SPANS];
#pragma unroll
      for (int i = 0; i < SPANS; ++i) c[i] = sr[i * FEW_ROWS * MT];
      float total = 0.f;
#pragma unroll
      for (int i = 0; i < SPANS; i += QUARTER) total += ((c[i] + c[i + 1]) + c[i + 2]) + c[i + 3];
      const int n = tile * FEW_ROWS + (tid & 15), m = m0 + (tid >> 4);
      if (n < N && m < M) finish<T, EPI>(out, (size_t)m * ldo + n, total);
    }
    buf ^= 1;
  }
  copies_wait<0>();
}

// What a launch asks the runtime once per device (of the first 64; others are asked each time): together half a
// microsecond of host time.
constexpr int DEVICES = 64;
inline int current_device() {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess ? dev : DEVICES;
}
inline int sm_count_of_device() {
  static std::atomic<int> counts[DEVICES];
  const int dev = current_device();
  int n = dev < DEVICES ? counts[dev].load(std::memory_order_relaxed) : 0;
  if (n > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  if (dev < DEVICES) counts[dev].store(n, std::memory_order_relaxed);
  return n;
}
// `allowed`: a bit per device, of this kernel
template <typename F>
inline void allow_smem(std::atomic<unsigned long long>& allowed, F* kernel, int bytes) {
  const int dev = current_device();
  const unsigned long long bit = dev < DEVICES ? 1ull << dev : 0;
  if (allowed.load(std::memory_order_acquire) & bit) return;
  if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
    allowed.fetch_or(bit, std::memory_order_release);
}

template <typename T, int EPI, int MT, bool VEC>
int launch_few(const T* a, const T* w, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w, cudaStream_t stream) {
  static std::atomic<unsigned long long> allowed{0};
  allow_smem(allowed, gemm_simt_few_kernel<T, EPI, MT, VEC>, FewShape<MT>::SMEM);
  const int tiles = (N + FEW_ROWS - 1) / FEW_ROWS, sms = sm_count_of_device();
  launch_kernel(gemm_simt_few_kernel<T, EPI, MT, VEC>, dim3(tiles < sms ? tiles : sms, (M + MT - 1) / MT), dim3(FEW_WARPS * 32),
                FewShape<MT>::SMEM, stream, a, w, out, M, N, K, lda, ldw, ldo, static_w);
  return launch_status();
}

template <typename T, int EPI, bool VEC>
int launch_tile(const T* a, const T* w, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w, cudaStream_t stream) {
  using S = TileShape<VEC>;
  const int quarter = QUARTER * span_length(K), quarters = (K + quarter - 1) / quarter;
  const long long m_tiles = (M + BM - 1) / BM, n_tiles = (N + BN - 1) / BN;
  if (M > 65535 * 64 || m_tiles * n_tiles * quarters > 0x7fffffffLL) return DLGO_ERR_SIZE;
  static std::atomic<unsigned long long> allowed{0};
  allow_smem(allowed, gemm_simt_tile_kernel<T, EPI, VEC>, S::SMEM);
  launch_kernel_cluster(gemm_simt_tile_kernel<T, EPI, VEC>, dim3((unsigned)(m_tiles * n_tiles * quarters)), dim3(S::THREADS), S::SMEM,
                        stream, dim3(quarters, 1, 1), a, w, out, M, N, K, lda, ldw, ldo, static_w);
  return launch_status();
}

// Rows up to which the few-row kernel runs: at 16 rows of 16384 x 2048 it takes 52 us and the tile kernel 125 us, which
// it takes for 17 to 64 rows alike.
constexpr int FEW_MAX = 16;

// Up to 64 k have two spans: one warp of a few-row block works.  Where it can also not copy asynchronously and has more than
// two tiles to take in turn, the tile kernel is the better one: 1 / 16 rows of 8192 x 37 6.7 / 10.1 us, tiles 5.3; of
// 2048 x 37, less than a tile a block, 2.7 / 4.2 and 3.9.
inline bool few_rows(bool vec, int M, int N, int K) {
  return M <= FEW_MAX && (vec || K > 64 || N <= 2 * FEW_ROWS * sm_count_of_device());
}

template <typename T, int EPI, bool VEC>
int launch_gemm_simt(const T* a, const T* w, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w, cudaStream_t stream) {
  if (few_rows(VEC, M, N, K)) {
    if constexpr (VEC) {
      if (M <= 1) return launch_few<T, EPI, 1, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
      if (M <= 2) return launch_few<T, EPI, 2, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
      if (M <= 4) return launch_few<T, EPI, 4, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
    }
    if (M <= 8) return launch_few<T, EPI, 8, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
    return launch_few<T, EPI, 16, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
  }
  return launch_tile<T, EPI, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
}

template <typename T, bool VEC>
int by_epilogue(const void* A, const void* W, void* out, int M, int N, int K, int lda, int ldw, int ldo, int epilogue,
                int static_w, cudaStream_t stream) {
  const T* a = (const T*)A;
  const T* w = (const T*)W;
  switch (epilogue) {
    case EPI_STORE:
      if constexpr (sizeof(T) < 4) return launch_gemm_simt<T, EPI_STORE, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
      else return DLGO_ERR_SIZE;
    case EPI_STORE_F32: return launch_gemm_simt<T, EPI_STORE_F32, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
    case EPI_ADD_F32: return launch_gemm_simt<T, EPI_ADD_F32, VEC>(a, w, out, M, N, K, lda, ldw, ldo, static_w, stream);
    default: return DLGO_ERR_SIZE;
  }
}

}  // namespace dlgo

// A[M, K] (row stride lda), W[N, K] (row stride ldw), both of element type `dtype`;
// out[M, N] (row stride ldo): epilogue 0 stores `dtype`, 1 stores f32, 2 adds into f32.  static_w: nothing launched before
// on the stream writes W (its first pieces are fetched before the launch before has finished).
DLGO_EXPORT int dlgo_gemm_simt(const void* A, const void* W, void* out, int dtype, int M, int N, int K, int lda,
                               int ldw, int ldo, int epilogue, int static_w, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return DLGO_OK;
  if (K <= 0 || lda < K || ldw < K || ldo < N) return DLGO_ERR_SIZE;
  if (dtype == DLGO_F32) {
    // whole aligned pieces of four in every row: asynchronous copies, else element by element
    const bool vec = ((K | lda | ldw) & 3) == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    if (epilogue == dlgo::EPI_STORE) epilogue = dlgo::EPI_STORE_F32;      // the same
    return vec ? dlgo::by_epilogue<float, true>(A, W, out, M, N, K, lda, ldw, ldo, epilogue, static_w, stream)
               : dlgo::by_epilogue<float, false>(A, W, out, M, N, K, lda, ldw, ldo, epilogue, static_w, stream);
  }
  if (dtype == DLGO_BF16) return dlgo::by_epilogue<__nv_bfloat16, false>(A, W, out, M, N, K, lda, ldw, ldo, epilogue, static_w, stream);
  return DLGO_ERR_DTYPE;
}
