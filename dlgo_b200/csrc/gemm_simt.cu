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
// Measured on a B200 (TFLOP/s): 567 x 16384 x 2048 41, 567 x 2048 x 8192 35, 64 x 16384 x 2048 34.  Blocks of 128 x 64 with
// four warps and four stages, two an SM, have as many warps there and more padding: 36, 34 and 19.  64 x 64 outputs of
// scalar multiply-adds with a synchronous load of every 16 k (before) 4; scalar multiply-adds in this layout 29 where
// packed ones give 38; 8 x 4 outputs per thread with twelve warps an SM and no cluster 36 and 20 for 366 rows.  The order
// of the multiply-adds and the width of the loads from shared memory change less than 2 %.  The fp32 pipes give 74 at most.
constexpr int BM = 64, BN = 64, KSTEP = 16, ROW = KSTEP + 4, STAGES = 3, THREADS = 64;
constexpr int TILE_RING = STAGES * (BM + BN) * ROW;      // floats
constexpr int TILE_SMEM = (TILE_RING + BM * BN) * 4;

template <typename T, int EPI, bool VEC>
__global__ void __launch_bounds__(THREADS, 4)
gemm_simt_tile_kernel(const T* A, const T* W, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w) {
  namespace cg = cooperative_groups;
  constexpr int LROWS = THREADS / 4;
  extern __shared__ __align__(16) float ring[];
  float4* sums = reinterpret_cast<float4*>(ring + TILE_RING);   // [16][THREADS]: of thread t's output row i, columns 4 h .. 4 h + 3 at 2 i + h
  pdl_launch_dependents();
  cg::cluster_group cl = cg::this_cluster();
  const int quarters = (int)cl.num_blocks(), quarter = (int)cl.block_rank();
  const int tile = (int)blockIdx.x / quarters;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m_tiles = (M + BM - 1) / BM;                      // blocks of the same weight rows follow one another
  const int m0 = (tile % m_tiles) * BM, n0 = (tile / m_tiles) * BN;
  const int tm = lane >> 2;                                   // rows tm + 8 i
  const int tn = warp * 32 + (lane & 3) * 2;                  // columns tn + (j & 1) + 8 (j >> 1)
  const int lrow = tid >> 2, lk = (tid & 3) * 4;              // loading
  const int span = span_length(K);
  const int k_begin = quarter * QUARTER * span, k_end = min(K, k_begin + QUARTER * span);
  const int steps = (k_end - k_begin + KSTEP - 1) / KSTEP;    // (quarters that exist are not empty)
  const int span_steps = span / KSTEP;
  auto load_w = [&](int step) {
    float* ws = ring + ((step % STAGES) * (BM + BN) + BM) * ROW;
#pragma unroll
    for (int i = 0; i < BN / LROWS; ++i) {
      const int n = n0 + lrow + LROWS * i;
      stage_four<T, VEC>(ws + (lrow + LROWS * i) * ROW + lk, W + (size_t)n * ldw, k_begin + step * KSTEP + lk, K, n < N);
    }
  };
  auto load_a = [&](int step) {
    float* as = ring + (step % STAGES) * (BM + BN) * ROW;
#pragma unroll
    for (int i = 0; i < BM / LROWS; ++i) {
      const int m = m0 + lrow + LROWS * i;
      stage_four<T, VEC>(as + (lrow + LROWS * i) * ROW + lk, A + (size_t)m * lda, k_begin + step * KSTEP + lk, K, m < M);
    }
  };
  if (!static_w) pdl_wait();    // (W may come from the launch before)
  for (int s = 0; s < STAGES - 1 && s < steps; ++s) load_w(s);
  pdl_wait();
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) load_a(s);
    copies_commit();
  }
  unsigned long long acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  int in_span = 0;
  bool first = true;
  for (int s = 0; s < steps; ++s) {
    copies_wait<STAGES - 2>();
    __syncthreads();            // stage s is in place, and every warp is past stage s - 1
    if (s + STAGES - 1 < steps) {
      load_w(s + STAGES - 1);
      load_a(s + STAGES - 1);
    }
    copies_commit();
    const float* as = ring + ((s % STAGES) * (BM + BN) + tm) * ROW;
    const float* ws = ring + ((s % STAGES) * (BM + BN) + BM + tn) * ROW;
    // two neighbours of k at a time; the next two are on their way from shared memory while these are multiplied
    unsigned long long a[2][8], b[2][8];
    auto fetch = [&](int k, unsigned long long (&x)[8], unsigned long long (&y)[8]) {
#pragma unroll
      for (int j = 0; j < 8; ++j) y[j] = *reinterpret_cast<const unsigned long long*>(ws + ((j & 1) + 8 * (j >> 1)) * ROW + k);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const unsigned long long*>(as + 8 * i * ROW + k);
    };
    fetch(0, a[0], b[0]);
#pragma unroll
    for (int k = 0; k < KSTEP; k += 2) {
      const int now = (k >> 1) & 1;
      if (k + 2 < KSTEP) fetch(k + 2, a[now ^ 1], b[now ^ 1]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) {
          const int j = (i & 1) ? 7 - jj : jj;          // (a row after another shares an operand at the turn)
          fma_two(acc[i][j], a[now][i], b[now][j]);
        }
    }
    if (++in_span == span_steps || s == steps - 1) {
#pragma unroll
      for (int g = 0; g < 16; ++g) {
        float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : sums[g * THREADS + tid];
        unsigned long long* q = &acc[g >> 1][(g & 1) * 4];
        v.x += pair_sum(q[0]); v.y += pair_sum(q[1]); v.z += pair_sum(q[2]); v.w += pair_sum(q[3]);
        sums[g * THREADS + tid] = v;
        q[0] = q[1] = q[2] = q[3] = 0ull;
      }
      in_span = 0;
      first = false;
    }
  }
  // Every block of the cluster finishes a share of the tile; what is added into is fetched while the others arrive.
  float old[4][4];
  if (EPI == EPI_ADD_F32 && quarters == 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int g = quarter + 4 * i, m = m0 + tm + 8 * (g >> 1), n = n0 + tn + 16 * (g & 1);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int ne = n + (e & 1) + 8 * (e >> 1);
        old[i][e] = m < M && ne < N ? ((const float*)out)[(size_t)m * ldo + ne] : 0.f;
      }
    }
  }
  if (quarters > 1) cl.sync();
  auto share = [&](int g, const float* added) {
    float4 v = *cl.map_shared_rank(sums + g * THREADS + tid, 0);
    for (int q = 1; q < quarters; ++q) {
      const float4 u = *cl.map_shared_rank(sums + g * THREADS + tid, q);
      v.x += u.x; v.y += u.y; v.z += u.z; v.w += u.w;
    }
    const float f[4] = {v.x, v.y, v.z, v.w};
    const int m = m0 + tm + 8 * (g >> 1), n = n0 + tn + 16 * (g & 1);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int ne = n + (e & 1) + 8 * (e >> 1);
      if (m >= M || ne >= N) continue;
      if (added != nullptr) ((float*)out)[(size_t)m * ldo + ne] = added[e] + f[e];
      else finish<T, EPI>(out, (size_t)m * ldo + ne, f[e]);
    }
  };
  if (quarters == 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) share(quarter + 4 * i, EPI == EPI_ADD_F32 ? old[i] : nullptr);
  } else {
    for (int g = quarter; g < 16; g += quarters) share(g, nullptr);
  }
  if (quarters > 1) cl.sync();  // nobody leaves while its sums may still be read
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

inline int sm_count_of_device() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return n;
}
template <typename F>
inline void allow_smem(F* kernel, int bytes) {
  cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

template <typename T, int EPI, int MT, bool VEC>
int launch_few(const T* a, const T* w, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w, cudaStream_t stream) {
  allow_smem(gemm_simt_few_kernel<T, EPI, MT, VEC>, FewShape<MT>::SMEM);
  const int tiles = (N + FEW_ROWS - 1) / FEW_ROWS, sms = sm_count_of_device();
  launch_kernel(gemm_simt_few_kernel<T, EPI, MT, VEC>, dim3(tiles < sms ? tiles : sms, (M + MT - 1) / MT), dim3(FEW_WARPS * 32),
                FewShape<MT>::SMEM, stream, a, w, out, M, N, K, lda, ldw, ldo, static_w);
  return launch_status();
}

template <typename T, int EPI, bool VEC>
int launch_tile(const T* a, const T* w, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w, cudaStream_t stream) {
  const int quarter = QUARTER * span_length(K), quarters = (K + quarter - 1) / quarter;
  const long long m_tiles = (M + BM - 1) / BM, n_tiles = (N + BN - 1) / BN;
  if (M > 65535 * 64 || m_tiles * n_tiles * quarters > 0x7fffffffLL) return DLGO_ERR_SIZE;
  allow_smem(gemm_simt_tile_kernel<T, EPI, VEC>, TILE_SMEM);
  launch_kernel_cluster(gemm_simt_tile_kernel<T, EPI, VEC>, dim3((unsigned)(m_tiles * n_tiles * quarters)), dim3(THREADS),
                        TILE_SMEM, stream, dim3(quarters, 1, 1), a, w, out, M, N, K, lda, ldw, ldo, static_w);
  return launch_status();
}

// Rows up to which the few-row kernel runs: at 16 rows of 16384 x 2048 it takes 52 us and the tile kernel 125 us, which
// it takes for 17 to 64 rows alike.
constexpr int FEW_MAX = 16;

template <typename T, int EPI, bool VEC>
int launch_gemm_simt(const T* a, const T* w, void* out, int M, int N, int K, int lda, int ldw, int ldo, int static_w, cudaStream_t stream) {
  if (M <= FEW_MAX) {
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
