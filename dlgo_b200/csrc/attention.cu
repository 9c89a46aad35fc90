// Grouped-query attention over the paged cache, for prompts and for decode.
//
// Reference: for query head h, kv head g = h / (Hq / Hkv):
//   s_t = (q_h . k_{t,g}) * scale  for t in [0, pos]   (causal by the loop bound,
//   never a -inf fill), softmax (subtract max, exp, sum, times 1/sum), then
//   o_h = sum_t p_t * v_{t,g}                     models/llm/forward.go:258-278
// Prompts attend the same way, reading keys and values back from the cache
// (models/llm/forward_batch.go:188-207), so this one kernel serves both: a
// block takes a tile of consecutive tokens of ONE sequence, one kv head (a
// chunk of its query heads), and one slice of the sequence's pages, and runs an
// online softmax in fp32 over 64-key pages.  With more than one slice the
// partial (max, sum, unnormalised output) go to scratch and a second kernel
// combines them.  A window w > 0 keeps keys t > pos - w only; w < 0 keeps the keys of the query's own chunk of -w
// positions (first_visible in common.cuh).
//
// Storage type T (float or bfloat16) is what q, the pages and the output hold;
// scores, softmax and the weighted sum are fp32 with expf.
#include <math.h>

#include "common.cuh"
#include "attention_combine.cuh"

namespace dlgo {

constexpr int ATT_THREADS = 128;
constexpr int ATT_MAX_ACC = 32;  // accumulators per thread: rows * hd <= 128 * 32

struct AttnParams {
  const void* q;
  int ldq;
  const void* kpages;
  const void* vpages;
  const int* page_table;
  int max_pages;
  const int* tiles;  // [n_tiles][3]: sequence index in the batch, first packed token, token count
  const int* seq_slot;
  const int* token_pos;
  void* out;
  int ldo;
  float* part_acc;  // [T, Hq, n_splits, hd]
  float* part_ml;   // [T, Hq, n_splits, 2]
  int Hq, Hkv, hd, page_size, n_splits, gchunk, n_gchunks, rows_max, window;
  float scale;
  const float* sink;  // [Hq] fp32 or null: see join_sink
};

template <typename T> struct Vec;
template <> struct Vec<float> {
  static constexpr int N = 4;
  __device__ static void load(const float* p, float* o) {
    float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <> struct Vec<__nv_bfloat16> {
  static constexpr int N = 8;
  __device__ static void load(const __nv_bfloat16* p, float* o) {
    uint4 v = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 f = __bfloat1622float2(h[i]);
      o[2 * i] = f.x;
      o[2 * i + 1] = f.y;
    }
  }
};

template <typename T>
__global__ void __launch_bounds__(ATT_THREADS) attention_kernel(AttnParams p) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int hd = p.hd, PS = p.page_size, kstride = hd + 1;
  const int G = p.Hq / p.Hkv;
  const int tile = blockIdx.x;
  const int kvh = blockIdx.y / p.n_gchunks, gc = blockIdx.y - kvh * p.n_gchunks;
  const int split = blockIdx.z;
  const int g0 = gc * p.gchunk;
  const int GC = min(p.gchunk, G - g0);
  const int seq = p.tiles[3 * tile], tok0 = p.tiles[3 * tile + 1], ntok = p.tiles[3 * tile + 2];
  const int R = ntok * GC;
  const int slot = p.seq_slot[seq];
  const int pos0 = p.token_pos[tok0];
  const int t_end = pos0 + ntok;  // one past the last key any row may see
  const int t_begin = first_visible(pos0, p.window);
  const int pg_first = t_begin / PS, pg_last = (t_end - 1) / PS;
  const int per = (pg_last - pg_first + 1 + p.n_splits - 1) / p.n_splits;
  const int pg_b = pg_first + split * per;
  const int pg_e = min(pg_last + 1, pg_b + per);

  float* q_s = smem;                          // [rows_max][hd]
  float* k_s = q_s + p.rows_max * hd;         // [PS][hd + 1]
  float* v_s = k_s + PS * kstride;            // [PS][hd]
  float* p_s = v_s + PS * hd;                 // [rows_max][PS]
  float* m_s = p_s + p.rows_max * PS;         // [rows_max] running max
  float* l_s = m_s + p.rows_max;              // [rows_max] running sum
  float* c_s = l_s + p.rows_max;              // [rows_max] correction of this page

  const T* q = (const T*)p.q;
  for (int idx = tid; idx < R * hd; idx += ATT_THREADS) {
    const int r = idx / hd, d = idx - r * hd;
    const int tq = r / GC, g = r - tq * GC;
    q_s[idx] = to_float(q[(size_t)(tok0 + tq) * p.ldq + (size_t)(kvh * G + g0 + g) * hd + d]);
  }
  for (int r = tid; r < R; r += ATT_THREADS) {
    m_s[r] = -INFINITY;
    l_s[r] = 0.f;
  }
  float acc[ATT_MAX_ACC];
#pragma unroll
  for (int i = 0; i < ATT_MAX_ACC; ++i) acc[i] = 0.f;
  __syncthreads();

  constexpr int VN = Vec<T>::N;
  const int vec_per_row = hd / VN;
  for (int pg = pg_b; pg < pg_e; ++pg) {
    const int page = readable_page(p.page_table + (size_t)slot * p.max_pages, pg);
    const size_t base = ((size_t)page * p.Hkv + kvh) * PS * hd;
    const T* kp = (const T*)p.kpages + base;
    const T* vp = (const T*)p.vpages + base;
    for (int idx = tid; idx < PS * vec_per_row; idx += ATT_THREADS) {
      const int key = idx / vec_per_row, dv = (idx - key * vec_per_row) * VN;
      const bool live = pg * PS + key < t_end;  // what lies beyond was never written
      float kf[VN], vf[VN];
      if (live) {
        Vec<T>::load(kp + (size_t)key * hd + dv, kf);
        Vec<T>::load(vp + (size_t)key * hd + dv, vf);
      } else {
#pragma unroll
        for (int j = 0; j < VN; ++j) kf[j] = vf[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < VN; ++j) {
        k_s[key * kstride + dv + j] = kf[j];
        v_s[key * hd + dv + j] = vf[j];
      }
    }
    __syncthreads();
    // scores
    for (int idx = tid; idx < R * PS; idx += ATT_THREADS) {
      const int r = idx / PS, key = idx - r * PS;
      const int t = pg * PS + key;
      const int pos_r = pos0 + r / GC;
      const bool valid = t <= pos_r && t >= first_visible(pos_r, p.window);
      float s = -INFINITY;
      if (valid) {
        const float* qr = q_s + r * hd;
        const float* kr = k_s + key * kstride;
        float dot = 0.f;
        for (int d = 0; d < hd; ++d) dot = fmaf(qr[d], kr[d], dot);
        s = dot * p.scale;
      }
      p_s[idx] = s;
    }
    __syncthreads();
    // online softmax: one warp per row
    for (int r = warp; r < R; r += ATT_THREADS / 32) {
      float mx = -INFINITY;
      for (int key = lane; key < PS; key += 32) mx = fmaxf(mx, p_s[r * PS + key]);
      mx = warp_max(mx);
      const float m_old = m_s[r];
      const float m_new = fmaxf(m_old, mx);
      float sum = 0.f;
      for (int key = lane; key < PS; key += 32) {
        const float s = p_s[r * PS + key];
        const float e = (m_new == -INFINITY || s == -INFINITY) ? 0.f : expf(s - m_new);
        p_s[r * PS + key] = e;
        sum += e;
      }
      sum = warp_sum(sum);
      if (lane == 0) {
        const float c = (m_old == -INFINITY) ? 0.f : expf(m_old - m_new);
        c_s[r] = c;
        l_s[r] = l_s[r] * c + sum;
        m_s[r] = m_new;
      }
    }
    __syncthreads();
    // weighted sum of the values
#pragma unroll
    for (int i = 0; i < ATT_MAX_ACC; ++i) {
      const int idx = tid + ATT_THREADS * i;
      if (idx < R * hd) {
        const int r = idx / hd, d = idx - r * hd;
        float a = acc[i] * c_s[r];
        const float* pr = p_s + r * PS;
        for (int key = 0; key < PS; ++key) a = fmaf(pr[key], v_s[key * hd + d], a);
        acc[i] = a;
      }
    }
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < ATT_MAX_ACC; ++i) {
    const int idx = tid + ATT_THREADS * i;
    if (idx < R * hd) {
      const int r = idx / hd, d = idx - r * hd;
      const int tq = r / GC, g = r - tq * GC;
      const int head = kvh * G + g0 + g;
      const size_t token = tok0 + tq;
      if (p.n_splits == 1) {
        float a = acc[i], l = l_s[r];
        join_sink(a, l, m_s[r], p.sink, head);
        ((T*)p.out)[token * p.ldo + (size_t)head * hd + d] = from_float<T>(a / l);
      } else {
        const size_t o = (token * p.Hq + head) * p.n_splits + split;
        p.part_acc[o * hd + d] = acc[i];
        if (d == 0) {
          p.part_ml[o * 2] = m_s[r];
          p.part_ml[o * 2 + 1] = l_s[r];
        }
      }
    }
  }
}

// ------------------------------------------------------------------ prompt tiles
// The same sums for tiles of up to 32 rows (token, query head) of heads of 16, 32, 64 or 128 and pages of 64 keys in one slice,
// in registers: a thread takes rows 16 apart and, of the scores, 4 keys 16 apart, then the same rows x HD / 16 outputs; the
// sixteen lanes that share a row hold its maximum and its sum.  Keys come 16 bytes at a time from shared memory, for
// 16 TR multiply-adds per 4 + TR loads; the kernel above loads two words for each multiply-add.  Scores and outputs are
// summed in the same order as there, a row's weights in another (four of a thread, then sixteen lanes).
// Bound by the fp32 pipes where tiles fill the SMs, by the longest tile's chain of pages where they do not, so the table's
// last tiles begin first: a prompt's longest.  (Of several prompts the last one's; two of 65 and 301 tokens take the same time
// in either order.)  Measured on a B200, fp32, us by the kernel above / here: 32 heads of 64 on 8, prompts of 65 and 301 tokens
// 214 / 47, one of 1,500 1,883 / 478; 24 heads of 128 on 8 284 / 72 and 3,380 / 851; 4 heads of 16 on 2 55 / 11 and 273 / 77.
template <int HD, int TR> struct RowsShape {
  static constexpr int ROWS = 16 * TR, KROW = HD + 4, PROW = 80;      // floats from one key / one row's weights to the next
  static constexpr int SMEM = (ROWS * HD + 64 * KROW + 64 * HD + ROWS * PROW) * 4;
  static constexpr int DV = HD / 16;                                  // outputs of a thread and row
};

template <typename T, int HD, int TR>
__global__ void __launch_bounds__(256) attention_rows_kernel(AttnParams p) {
  using S = RowsShape<HD, TR>;
  constexpr int DV = S::DV, DW = DV < 4 ? DV : 4, VN = Vec<T>::N, LOADS = (64 * HD / VN + 255) / 256;
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;                          // [ROWS][HD]
  float* k_s = q_s + S::ROWS * HD;            // [64][KROW]
  float* v_s = k_s + 64 * S::KROW;            // [64][HD]
  float* p_s = v_s + 64 * HD;                 // [ROWS][PROW]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int G = p.Hq / p.Hkv;
  const int tile = gridDim.x - 1 - blockIdx.x;
  const int kvh = blockIdx.y / p.n_gchunks, g0 = (blockIdx.y - kvh * p.n_gchunks) * p.gchunk;
  const int GC = min(p.gchunk, G - g0);
  const int seq = p.tiles[3 * tile], tok0 = p.tiles[3 * tile + 1], ntok = p.tiles[3 * tile + 2];
  const int R = ntok * GC;
  const int* page_row = p.page_table + (size_t)p.seq_slot[seq] * p.max_pages;
  const int pos0 = p.token_pos[tok0], t_end = pos0 + ntok;
  const T* q = (const T*)p.q;
  for (int idx = tid; idx < S::ROWS * HD; idx += 256) {
    const int r = idx / HD, d = idx % HD, tq = r / GC;
    q_s[idx] = r < R ? to_float(q[(size_t)(tok0 + tq) * p.ldq + (size_t)(kvh * G + g0 + r - tq * GC) * HD + d]) : 0.f;
  }
  float acc[TR][DV], m[TR], l[TR];
  int pos[TR], low[TR];
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    pos[i] = pos0 + (ty + 16 * i) / GC;
    low[i] = first_visible(pos[i], p.window);
    m[i] = -INFINITY;
    l[i] = 0.f;
#pragma unroll
    for (int e = 0; e < DV; ++e) acc[i][e] = 0.f;
  }
  for (int pg = first_visible(pos0, p.window) / 64; pg <= (t_end - 1) / 64; ++pg) {
    const size_t base = ((size_t)readable_page(page_row, pg) * p.Hkv + kvh) * 64 * HD;
    const T* kp = (const T*)p.kpages + base;
    const T* vp = (const T*)p.vpages + base;
    const int keys = min(64, t_end - pg * 64);          // what lies beyond was never written
    float kf[LOADS][VN], vf[LOADS][VN];
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
      const int at = (tid + 256 * i) * VN;
#pragma unroll
      for (int e = 0; e < VN; ++e) kf[i][e] = vf[i][e] = 0.f;
      if (at < keys * HD) {
        Vec<T>::load(kp + at, kf[i]);
        Vec<T>::load(vp + at, vf[i]);
      }
    }
    __syncthreads();                                    // (everyone is done with the page before)
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
      const int at = (tid + 256 * i) * VN;
      if (at < 64 * HD) {
#pragma unroll
        for (int e = 0; e < VN; e += 4) {
          *reinterpret_cast<float4*>(k_s + at / HD * S::KROW + at % HD + e) = make_float4(kf[i][e], kf[i][e + 1], kf[i][e + 2], kf[i][e + 3]);
          *reinterpret_cast<float4*>(v_s + at + e) = make_float4(vf[i][e], vf[i][e + 1], vf[i][e + 2], vf[i][e + 3]);
        }
      }
    }
    __syncthreads();
    float s[TR][4];
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
    for (int d = 0; d < HD; d += 4) {
      float4 a[TR], b[4];
#pragma unroll
      for (int i = 0; i < TR; ++i) a[i] = *reinterpret_cast<const float4*>(q_s + (ty + 16 * i) * HD + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(k_s + (tx + 16 * j) * S::KROW + d);
#pragma unroll
      for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[i][j] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, s[i][j]))));
    }
#pragma unroll
    for (int i = 0; i < TR; ++i) {
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int t = pg * 64 + tx + 16 * j;
        s[i][j] = t <= pos[i] && t >= low[i] ? s[i][j] * p.scale : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m_new = fmaxf(m[i], mx);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = (m_new == -INFINITY || s[i][j] == -INFINITY) ? 0.f : expf(s[i][j] - m_new);
        p_s[(ty + 16 * i) * S::PROW + tx + 16 * j] = e;
        sum += e;
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const float c = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
      l[i] = l[i] * c + sum;
      m[i] = m_new;
#pragma unroll
      for (int e = 0; e < DV; ++e) acc[i][e] *= c;
    }
    __syncwarp();                                       // (a row's weights come from the lanes that use them)
    for (int key = 0; key < keys; key += 4) {
      float4 w[TR];
#pragma unroll
      for (int i = 0; i < TR; ++i) w[i] = *reinterpret_cast<const float4*>(p_s + (ty + 16 * i) * S::PROW + key);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float v[DV];
#pragma unroll
        for (int e = 0; e < DV; e += DW) {
          const float* src = v_s + (key + k) * HD + tx * DW + e * 16;
          if constexpr (DW == 4) {
            const float4 x = *reinterpret_cast<const float4*>(src);
            v[e] = x.x; v[e + 1] = x.y; v[e + 2] = x.z; v[e + 3] = x.w;
          } else {
#pragma unroll
            for (int f = 0; f < DW; ++f) v[e + f] = src[f];
          }
        }
#pragma unroll
        for (int i = 0; i < TR; ++i) {
          const float pk = k == 0 ? w[i].x : (k == 1 ? w[i].y : (k == 2 ? w[i].z : w[i].w));
#pragma unroll
          for (int e = 0; e < DV; ++e) acc[i][e] = fmaf(pk, v[e], acc[i][e]);
        }
      }
    }
    __syncwarp();                                       // (nobody writes the next weights before)
  }
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    const int r = ty + 16 * i, tq = r / GC, head = kvh * G + g0 + r - tq * GC;
    if (r >= R) continue;
    T* o = (T*)p.out + (size_t)(tok0 + tq) * p.ldo + (size_t)head * HD;
#pragma unroll
    for (int e = 0; e < DV; e += DW)
#pragma unroll
      for (int f = 0; f < DW; ++f) {
        float a = acc[i][e + f], sum = l[i];
        join_sink(a, sum, m[i], p.sink, head);
        o[tx * DW + e * 16 + f] = from_float<T>(a / sum);
      }
  }
}

template <typename T, int HD, int TR>
int launch_rows(const AttnParams& p, int n_tiles, cudaStream_t stream) {
  constexpr int SMEM = RowsShape<HD, TR>::SMEM;
  if (SMEM > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<T, HD, TR>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
  }
  launch_kernel(attention_rows_kernel<T, HD, TR>, dim3(n_tiles, p.Hkv * p.n_gchunks), dim3(256), SMEM, stream, p);
  return launch_status();
}
template <typename T, int HD>
int launch_rows(const AttnParams& p, int n_tiles, cudaStream_t stream) {
  return p.rows_max <= 16 ? launch_rows<T, HD, 1>(p, n_tiles, stream) : launch_rows<T, HD, 2>(p, n_tiles, stream);
}

template <typename T>
int launch_attention(const AttnParams& p, int n_tiles, int T_tokens, cudaStream_t stream) {
  const bool aligned = (((uintptr_t)p.kpages | (uintptr_t)p.vpages) & 15) == 0;
  if (p.n_splits == 1 && p.page_size == 64 && p.rows_max <= 32 && aligned) {
    switch (p.hd) {
      case 16: return launch_rows<T, 16>(p, n_tiles, stream);
      case 32: return launch_rows<T, 32>(p, n_tiles, stream);
      case 64: return launch_rows<T, 64>(p, n_tiles, stream);
      case 128: return launch_rows<T, 128>(p, n_tiles, stream);
      default: break;
    }
  }
  const size_t smem = sizeof(float) * ((size_t)p.rows_max * p.hd + (size_t)p.page_size * (p.hd + 1) +
                                       (size_t)p.page_size * p.hd + (size_t)p.rows_max * p.page_size +
                                       3 * (size_t)p.rows_max);
  if (smem > 227 * 1024) return DLGO_ERR_SIZE;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(attention_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid(n_tiles, p.Hkv * p.n_gchunks, p.n_splits);
  launch_kernel(attention_kernel<T>, dim3(grid), dim3(ATT_THREADS), smem, stream, p);
  int st = launch_status();
  if (st != DLGO_OK || p.n_splits == 1) return st;
  dim3 cgrid(T_tokens, p.Hq);
  const int threads = p.hd >= 128 ? 128 : (p.hd >= 64 ? 64 : 32);
  launch_kernel(attention_combine_kernel<T>, dim3(cgrid), dim3(threads), 0, stream, p.part_acc, p.part_ml, (T*)p.out, p.ldo, p.Hq, p.hd,
                                                             p.n_splits, p.sink);
  return launch_status();
}

}  // namespace dlgo

using namespace dlgo;

// Floats of scratch the call needs for `n_splits` > 1 (0 for one slice):
// part_acc [T, Hq, n_splits, hd] followed by part_ml [T, Hq, n_splits, 2].
DLGO_EXPORT long long dlgo_attention_scratch_floats(int T, int Hq, int hd, int n_splits) {
  if (n_splits <= 1) return 0;
  return (long long)T * Hq * n_splits * (hd + 2);
}

// q[T, .] with row stride ldq (head h at column h*hd); pages [n_pages, Hkv, page_size, hd];
// tiles[n_tiles][3]; rows_max = (largest token count of a tile) * gchunk;
// out[T, Hq*hd] with row stride ldo.  `scratch` as sized above.  `sink` [Hq] fp32 or null: joins the denominator.
DLGO_EXPORT int dlgo_attention(const void* q, int dtype, int T, int ldq, const void* kpages, const void* vpages,
                               const int* page_table, int max_pages, const int* tiles, int n_tiles,
                               int tile_tokens_max, const int* seq_slot, const int* token_pos, void* out, int ldo,
                               float* scratch, int Hq, int Hkv, int hd, int page_size, int n_splits, int gchunk,
                               int window, float scale, const float* sink, cudaStream_t stream) {
  if (T <= 0 || n_tiles <= 0) return DLGO_OK;
  if (Hq <= 0 || Hkv <= 0 || Hq % Hkv || hd <= 0 || page_size <= 0 || page_size % 32 || n_splits <= 0 ||
      gchunk <= 0 || tile_tokens_max <= 0)
    return DLGO_ERR_SIZE;
  if (hd % (dtype == DLGO_BF16 ? 8 : 4)) return DLGO_ERR_SIZE;
  const int G = Hq / Hkv;
  if (gchunk > G) gchunk = G;
  AttnParams p;
  p.q = q; p.ldq = ldq; p.kpages = kpages; p.vpages = vpages; p.page_table = page_table; p.max_pages = max_pages;
  p.tiles = tiles; p.seq_slot = seq_slot; p.token_pos = token_pos; p.out = out; p.ldo = ldo;
  p.part_acc = scratch;
  p.part_ml = scratch ? scratch + (size_t)T * Hq * n_splits * hd : nullptr;
  p.Hq = Hq; p.Hkv = Hkv; p.hd = hd; p.page_size = page_size; p.n_splits = n_splits; p.gchunk = gchunk;
  p.n_gchunks = (G + gchunk - 1) / gchunk;
  p.rows_max = tile_tokens_max * gchunk;
  p.window = window; p.scale = scale; p.sink = sink;
  if ((long long)p.rows_max * hd > (long long)ATT_THREADS * ATT_MAX_ACC) return DLGO_ERR_SIZE;
  if (n_splits > 1 && scratch == nullptr) return DLGO_ERR_SIZE;
  if ((long long)Hkv * p.n_gchunks > 65535 || n_splits > 65535) return DLGO_ERR_SIZE;
  if (dtype == DLGO_F32) return launch_attention<float>(p, n_tiles, T, stream);
  if (dtype == DLGO_BF16) return launch_attention<__nv_bfloat16>(p, n_tiles, T, stream);
  return DLGO_ERR_DTYPE;
}

// ---------------------------------------------------------------------------------------------
// The entry point that allocates nothing (see attention_noalloc.h for who needs it and its rules).
#include "attention_noalloc.h"

// The scratch itself.  In host code this name is only a handle for cudaGetSymbolAddress, never a
// device address: a kernel must be given the looked-up pointer.
static __device__ __align__(256) float g_attention_scratch[DLGO_ATTENTION_NOALLOC_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
float* g_scratch_addr[kMaxDevices] = {nullptr};

// Device address of the scratch on the current device; looked up once per device.
int scratch_address(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return DLGO_ERR_SIZE;
  if (g_scratch_addr[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress((void**)&p, g_attention_scratch);
    if (e != cudaSuccess) return (int)e;
    if (p == nullptr) return DLGO_ERR_DRIVER;
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return DLGO_OK;
}
}  // namespace

DLGO_EXPORT long long dlgo_attention_noalloc_needs(int T, int Hq, int hd, int n_splits) {
  return dlgo_attention_scratch_floats(T, Hq, hd, n_splits);
}

DLGO_EXPORT int dlgo_attention_noalloc(const void* q, int dtype, int T, int ldq, const void* kpages,
                                       const void* vpages, const int* page_table, int max_pages, const int* tiles,
                                       int n_tiles, int tile_tokens_max, const int* seq_slot, const int* token_pos,
                                       void* out, int ldo, int Hq, int Hkv, int hd, int page_size, int n_splits,
                                       int gchunk, int window, float scale, cudaStream_t stream) {
  if (T <= 0 || n_tiles <= 0) return DLGO_OK;
  if (Hq <= 0 || hd <= 0 || n_splits <= 0) return DLGO_ERR_SIZE;
  const long long need = dlgo_attention_scratch_floats(T, Hq, hd, n_splits);
  if (need > (long long)DLGO_ATTENTION_NOALLOC_FLOATS) return DLGO_ERR_SIZE;  // beyond the stated maximum
  float* scratch = nullptr;
  if (need > 0) {
    const int st = scratch_address(&scratch);
    if (st != DLGO_OK) return st;
  }
  return dlgo_attention(q, dtype, T, ldq, kpages, vpages, page_table, max_pages, tiles, n_tiles, tile_tokens_max,
                        seq_slot, token_pos, out, ldo, scratch, Hq, Hkv, hd, page_size, n_splits, gchunk, window,
                        scale, nullptr, stream);
}
