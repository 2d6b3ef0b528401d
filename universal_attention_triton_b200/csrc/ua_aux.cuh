// HBM-bound helper kernels: layout conversion between chunk-major storage and
// the reference's key-chunk-innermost tensors, and the merge over key chunks
// (SMVecMatMul, universal_attention_autograd.py:278-297).
#pragma once
#include "ua_common.cuh"

namespace ua {
namespace aux {

// Batched transpose.  For every batch index g (= (bh, r)):
//   to_reference:  dst[(g*X + x)*N + n] = src[((bh*N + n)*R + r)*X + x]
//   else        :  dst[((bh*N + n)*R + r)*X + x] = src[(g*X + x)*N + n]
// with X = L*inner.  32x32 shared-memory tiles keep both sides coalesced.
template <typename E>
__global__ void __launch_bounds__(256) relayout_kernel(const E* __restrict__ src, E* __restrict__ dst, int N, int R,
                                                       long long X, int to_reference) {
  __shared__ E tile[32][33];
  const int g = blockIdx.z;
  const int bh = g / R, r = g - bh * R;
  const long long x0 = (long long)blockIdx.x * 32;
  const int n0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8
  if (to_reference) {
    for (int yy = ty; yy < 32; yy += 8) {
      int n = n0 + yy;
      long long x = x0 + tx;
      if (n < N && x < X) tile[yy][tx] = src[(((long long)bh * N + n) * R + r) * X + x];
    }
    __syncthreads();
    for (int yy = ty; yy < 32; yy += 8) {
      long long x = x0 + yy;
      int n = n0 + tx;
      if (n < N && x < X) dst[((long long)g * X + x) * N + n] = tile[tx][yy];
    }
  } else {
    for (int yy = ty; yy < 32; yy += 8) {
      long long x = x0 + yy;
      int n = n0 + tx;
      if (n < N && x < X) tile[yy][tx] = src[((long long)g * X + x) * N + n];
    }
    __syncthreads();
    for (int yy = ty; yy < 32; yy += 8) {
      int n = n0 + yy;
      long long x = x0 + tx;
      if (n < N && x < X) dst[(((long long)bh * N + n) * R + r) * X + x] = tile[tx][yy];
    }
  }
}

// ---- merge over key chunks (SMVecMatMul) -----------------------------------------
// A block takes 256 / TPR neighbouring rows (b,h,r,l), TPR = D * sizeof(T) / 16 threads each; every thread
// owns one 16-byte slice of the row (8 bf16 or 4 floats), so a block reads a contiguous piece of
// every chunk of out_cm.  Chunks whose softmax weight is exactly zero (rows before a key chunk have
// lse = -1e12) are never read; on B4 H8 L4096 that halves the traffic.
constexpr int kMergeThreads = 256;

template <typename T> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int kN = 4;
  static __device__ __forceinline__ void load(const float* p, float* v) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
  static __device__ __forceinline__ void store(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
  static __device__ __forceinline__ void unpack(const uint4& x, float* v) {
    v[0] = __uint_as_float(x.x); v[1] = __uint_as_float(x.y); v[2] = __uint_as_float(x.z); v[3] = __uint_as_float(x.w);
  }
  static __device__ __forceinline__ uint4 pack(const float* v) {
    return make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  }
};
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int kN = 8;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* v) { unpack(*reinterpret_cast<const uint4*>(p), v); }
  static __device__ __forceinline__ void unpack(const uint4& x, float* v) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
      v[2 * i] = __bfloat162float(h.x);
      v[2 * i + 1] = __bfloat162float(h.y);
    }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float* v) { *reinterpret_cast<uint4*>(p) = pack(v); }
  static __device__ __forceinline__ uint4 pack(const float* v) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};

template <int TPR>
__device__ __forceinline__ float group_max(float v) {
#pragma unroll
  for (int o = TPR / 2; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int TPR>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = TPR / 2; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Weights of a block's kRows rows: W[n][row] = softmax over n of lse[n][row], in shared memory (pitch kRows + 1).  The log-sum-exps
// are read once, coalesced along the rows; the TPR threads of a row share its statistics.  Returns the number of chunks up to the last
// one with a weight that is not zero, for any row of the warp: behind it nothing needs to be read.
template <typename TL, int TPR>
__device__ __forceinline__ int merge_weights(const TL* lse, size_t nstride, int N, int rows_here, float* W, float& m, float& zinv) {
  constexpr int kRows = kMergeThreads / TPR, kPitch = kRows + 1;
  for (int e = threadIdx.x; e < N * kRows; e += kMergeThreads) {
    const int n = e / kRows, q = e % kRows;
    W[n * kPitch + q] = Num<TL>::ld(lse + (size_t)n * nstride + (q < rows_here ? q : rows_here - 1));
  }
  __syncthreads();
  const int sub = threadIdx.x % TPR;
  float* mine = W + threadIdx.x / TPR;
  float mm = -INFINITY;
  for (int n = sub; n < N; n += TPR) mm = fmaxf(mm, mine[n * kPitch]);
  m = group_max<TPR>(mm);
  float z = 0.f;
  for (int n = sub; n < N; n += TPR) z += expf(mine[n * kPitch] - m);
  zinv = 1.0f / group_sum<TPR>(z);
  int last = 0;
  for (int n = sub; n < N; n += TPR) {
    const float w = expf(mine[n * kPitch] - m) * zinv;
    mine[n * kPitch] = w;
    if (w != 0.f) last = n + 1;
  }
  __syncwarp();
  return __reduce_max_sync(0xffffffffu, last);
}
constexpr int kMergeAhead = 8;      // chunks whose loads a thread has in flight
// (in an order the compiler keeps: it would otherwise issue each read beside its use, a few at a time)
__device__ __forceinline__ uint4 load_if(const uint4* p, bool on) {
  uint4 x = make_uint4(0, 0, 0, 0);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.s32 p, %5, 0;\n\t@p ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "+r"(x.x), "+r"(x.y), "+r"(x.z), "+r"(x.w) : "l"(p), "r"((int)on));
  return x;
}

// merged[row][d] = sum_n softmax_n(lse[n][row]) * out_cm[n][row][d]
// Bound by the read of the chunks that count; eight 16-byte loads in flight per thread.  B4 H8 R4 L4096 D64 (1.07 GB read):
// 306 us with one load in flight behind its own exponential -> 205 us (5.2 TB/s).
template <typename T, typename TL, int TPR>
__global__ void __launch_bounds__(kMergeThreads) merge_fwd_kernel(const T* __restrict__ out_cm, const TL* __restrict__ lse_cm,
                                                                  T* __restrict__ merged, float* __restrict__ row_lse, int N, int R, int L) {
  constexpr int kN = Vec16<T>::kN, D = TPR * kN, kRows = kMergeThreads / TPR, kPitch = kRows + 1;
  extern __shared__ float sW[];
  const int tiles = (L + kRows - 1) / kRows, gr = blockIdx.x / tiles, l0 = (blockIdx.x - gr * tiles) * kRows;      // gr = bh * R + r
  const int r = gr % R, row = threadIdx.x / TPR, sub = threadIdx.x % TPR;
  const size_t nstride = (size_t)R * L, base = ((size_t)(gr / R) * N * R + r) * L + l0;
  const int rows_here = L - l0 < kRows ? L - l0 : kRows;
  const bool live = row < rows_here;
  float m, zinv;
  const int last = merge_weights<TL, TPR>(lse_cm + base, nstride, N, rows_here, sW, m, zinv);
  float acc[kN];
#pragma unroll
  for (int i = 0; i < kN; ++i) acc[i] = 0.f;
  const uint4* src = reinterpret_cast<const uint4*>(out_cm + (base + row) * D) + sub;
  const size_t step = nstride * D * sizeof(T) / 16;
  for (int n0 = 0; n0 < last; n0 += kMergeAhead) {
    uint4 raw[kMergeAhead];
    float w[kMergeAhead];
#pragma unroll
    for (int u = 0; u < kMergeAhead; ++u) {
      w[u] = (live && n0 + u < last) ? sW[(n0 + u) * kPitch + row] : 0.f;
      raw[u] = load_if(src + (n0 + u) * step, w[u] != 0.f);
    }
#pragma unroll
    for (int u = 0; u < kMergeAhead; ++u) {
      float v[kN];
      Vec16<T>::unpack(raw[u], v);
#pragma unroll
      for (int i = 0; i < kN; ++i) acc[i] = fmaf(w[u], v[i], acc[i]);
    }
  }
  if (!live) return;
  const size_t orow = (size_t)gr * L + l0 + row;
  Vec16<T>::store(merged + orow * D + sub * kN, acc);
  if (sub == 0 && row_lse) row_lse[orow] = m - logf(zinv);      // log-sum-exp of the row over all key chunks
}

// ... of a few chunks (kFew = 2 .. 4, the sub-chunks of a wide chunk): no tables and no barrier, all of a thread's reads at once.  With
// the kernel above, whose blocks then have next to nothing to do between their barriers, 2 sub-chunks of B1 H8 R4 L2048 D128
// took 179 us.
template <typename T, typename TL, int TPR, int kFew>
__global__ void __launch_bounds__(kMergeThreads) merge_few_kernel(const T* __restrict__ out_cm, const TL* __restrict__ lse_cm,
                                                                  T* __restrict__ merged, float* __restrict__ row_lse, long long rows, int R, int L) {
  constexpr int kN = Vec16<T>::kN, D = TPR * kN;
  const long long row = (long long)blockIdx.x * (kMergeThreads / TPR) + threadIdx.x / TPR;
  if (row >= rows) return;
  const int sub = threadIdx.x % TPR;
  const size_t nstride = (size_t)R * L, base = (size_t)(row / (long long)nstride) * kFew * nstride + (size_t)(row % (long long)nstride);
  uint4 raw[kFew];
  float e[kFew], m = -INFINITY, z = 0.f, acc[kN];
#pragma unroll
  for (int n = 0; n < kFew; ++n) {
    e[n] = Num<TL>::ld(lse_cm + base + n * nstride);
    raw[n] = __ldcs(reinterpret_cast<const uint4*>(out_cm + (base + n * nstride) * D) + sub);
  }
#pragma unroll
  for (int n = 0; n < kFew; ++n) m = fmaxf(m, e[n]);
#pragma unroll
  for (int n = 0; n < kFew; ++n) z += e[n] = expf(e[n] - m);
  const float zinv = 1.0f / z;
#pragma unroll
  for (int i = 0; i < kN; ++i) acc[i] = 0.f;
#pragma unroll
  for (int n = 0; n < kFew; ++n) {
    const float w = e[n] * zinv;
    float v[kN];
    Vec16<T>::unpack(raw[n], v);
#pragma unroll
    for (int i = 0; i < kN; ++i) acc[i] = w != 0.f ? fmaf(w, v[i], acc[i]) : acc[i];
  }
  Vec16<T>::store(merged + (size_t)row * D + sub * kN, acc);
  if (sub == 0 && row_lse) row_lse[row] = m - logf(zinv);
}

// Backward of the merge: g_out_cm[n][row][:] = g[row][:] w_n ; g_lse[n][row] = (s_n - sum_m s_m w_m) w_n,
// s_n = g[row] . out_cm[n][row].  With skip_masked, the (row, chunk) blocks with row < n * chunk (rows before
// the key chunk, whose weight is exactly zero) are not written: the caller promises not to read them.
// Bound by HBM: the chunks that count are read, all are written.  Same shape as the forward; B4 H8 R4 L4096 D64: 952 -> 533 us (6.0 TB/s).
template <typename T, typename TL, int TPR>
__global__ void __launch_bounds__(kMergeThreads) merge_bwd_kernel(const T* __restrict__ out_cm, const TL* __restrict__ lse_cm,
                                                                  const T* __restrict__ g_merged, T* __restrict__ g_out_cm,
                                                                  TL* __restrict__ g_lse_cm, int N, int R, int L, int skip_masked) {
  constexpr int kN = Vec16<T>::kN, D = TPR * kN, kRows = kMergeThreads / TPR, kPitch = kRows + 1;
  extern __shared__ float sW[];
  float *sS = sW + N * kPitch, *sT = sS + N * kPitch;
  const int tiles = (L + kRows - 1) / kRows, gr = blockIdx.x / tiles, l0 = (blockIdx.x - gr * tiles) * kRows;
  const int r = gr % R, row = threadIdx.x / TPR, sub = threadIdx.x % TPR, chunk = L / N;
  const size_t nstride = (size_t)R * L, base = ((size_t)(gr / R) * N * R + r) * L + l0;
  const int rows_here = L - l0 < kRows ? L - l0 : kRows;
  const bool live = row < rows_here;
  float g[kN];
  Vec16<T>::load(g_merged + ((size_t)gr * L + l0 + (live ? row : 0)) * D + sub * kN, g);
  float m, zinv;
  const int last = merge_weights<TL, TPR>(lse_cm + base, nstride, N, rows_here, sW, m, zinv);
  const size_t step = nstride * D * sizeof(T) / 16, first = (base + row) * D * sizeof(T) / 16 + sub;
  const uint4* src = reinterpret_cast<const uint4*>(out_cm) + first;
  uint4* dst = reinterpret_cast<uint4*>(g_out_cm) + first;
  float t = 0.f;
  for (int n0 = 0; n0 < last; n0 += kMergeAhead) {
    uint4 raw[kMergeAhead];
    float w[kMergeAhead];
#pragma unroll
    for (int u = 0; u < kMergeAhead; ++u) {
      w[u] = (live && n0 + u < last) ? sW[(n0 + u) * kPitch + row] : 0.f;
      raw[u] = load_if(src + (n0 + u) * step, w[u] != 0.f);
    }
#pragma unroll
    for (int u = 0; u < kMergeAhead; ++u) {
      if (n0 + u >= last) break;
      float v[kN], o[kN], s = 0.f;
      Vec16<T>::unpack(raw[u], v);
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        s = fmaf(g[i], v[i], s);
        o[i] = g[i] * w[u];
      }
      if (live && (w[u] != 0.f || !(skip_masked && l0 + row < (n0 + u) * chunk))) __stcs(dst + (n0 + u) * step, Vec16<T>::pack(o));
      s = group_sum<TPR>(s);
      t = fmaf(s, w[u], t);
      if (sub == 0) sS[(n0 + u) * kPitch + row] = s;
    }
  }
  for (int n = last; n < N; ++n) {
    if (live && !(skip_masked && l0 + row < n * chunk)) __stcs(dst + n * step, make_uint4(0, 0, 0, 0));
    if (sub == 0) sS[n * kPitch + row] = 0.f;
  }
  if (sub == 0) sT[row] = t;
  __syncthreads();
  for (int e = threadIdx.x; e < N * kRows; e += kMergeThreads) {
    const int n = e / kRows, q = e % kRows;
    if (q < rows_here && !(skip_masked && l0 + q < n * chunk))
      Num<TL>::st(g_lse_cm + base + (size_t)n * nstride + q, (sS[n * kPitch + q] - sT[q]) * sW[n * kPitch + q]);
  }
}
// ... for so many chunks that the tables do not fit shared memory (N above about 860 at head_dim 64): weights from the log-sum-exps on
// the fly, TPR threads per row, and in the backward a first pass over the outputs for sum_m s_m w_m alone.
template <typename T, typename TL, int TPR>
__global__ void __launch_bounds__(kMergeThreads) merge_many_kernel(const T* __restrict__ out_cm, const TL* __restrict__ lse_cm,
                                                                   T* __restrict__ merged, float* __restrict__ row_lse,
                                                                   const T* __restrict__ g_merged, T* __restrict__ g_out_cm, TL* __restrict__ g_lse_cm,
                                                                   long long rows, int N, int R, int L, int skip_masked) {
  constexpr int kN = Vec16<T>::kN, D = TPR * kN;
  const long long first = (long long)blockIdx.x * (kMergeThreads / TPR) + threadIdx.x / TPR, row = first < rows ? first : rows - 1;
  const bool live = first < rows;
  const int sub = threadIdx.x % TPR, l = (int)(row % L), r = (int)(row / L % R), chunk = L / N;
  const size_t nstride = (size_t)R * L, base = ((size_t)(row / L / R) * N * R + r) * L + l;
  auto lse = [&](int n) { return Num<TL>::ld(lse_cm + base + (size_t)n * nstride); };
  float m = -INFINITY, z = 0.f;
  for (int n = sub; n < N; n += TPR) m = fmaxf(m, lse(n));
  m = group_max<TPR>(m);
  for (int n = sub; n < N; n += TPR) z += expf(lse(n) - m);
  const float zinv = 1.0f / group_sum<TPR>(z);
  auto weight = [&](int n) { return expf(lse(n) - m) * zinv; };
  float g[kN], acc[kN], t = 0.f;
#pragma unroll
  for (int i = 0; i < kN; ++i) g[i] = acc[i] = 0.f;
  if (g_merged) Vec16<T>::load(g_merged + (size_t)row * D + sub * kN, g);
  auto product = [&](int n, float w) {      // s_n, and the weighted sum
    float v[kN], s = 0.f;
    if (w != 0.f) {
      Vec16<T>::load(out_cm + (base + (size_t)n * nstride) * D + sub * kN, v);
#pragma unroll
      for (int i = 0; i < kN; ++i) {
        s = fmaf(g[i], v[i], s);
        acc[i] = fmaf(w, v[i], acc[i]);
      }
    }
    return s;
  };
  for (int n = 0; n < N; ++n) {
    const float w = weight(n), s = product(n, w);
    if (g_merged) t = fmaf(group_sum<TPR>(s), w, t);
  }
  if (!g_merged) {
    if (live) Vec16<T>::store(merged + (size_t)row * D + sub * kN, acc);
    if (live && sub == 0 && row_lse) row_lse[row] = m - logf(zinv);
    return;
  }
  for (int n = 0; n < N; ++n) {
    const size_t at = base + (size_t)n * nstride;
    const float w = weight(n), s = group_sum<TPR>(product(n, w));
    if (!live || (skip_masked && w == 0.f && l < n * chunk)) continue;
    float o[kN];
#pragma unroll
    for (int i = 0; i < kN; ++i) o[i] = g[i] * w;
    Vec16<T>::store(g_out_cm + at * D + sub * kN, o);
    if (sub == 0) Num<TL>::st(g_lse_cm + at, (s - t) * w);
  }
}
template <int TPR> inline size_t merge_smem(int N, bool backward) {
  constexpr int kRows = kMergeThreads / TPR;
  return ((size_t)N * (kRows + 1) * (backward ? 2 : 1) + kRows) * sizeof(float);
}

// out[row] = a[row] . b[row] over D = TPR * kN elements (the delta = g . merged of the merged backward)
template <typename T, int TPR>
__global__ void __launch_bounds__(kMergeThreads) row_dot_kernel(const T* __restrict__ a, const T* __restrict__ b,
                                                                float* __restrict__ out, long long rows) {
  constexpr int kN = Vec16<T>::kN;
  constexpr int D = TPR * kN;
  const long long row = (long long)blockIdx.x * (kMergeThreads / TPR) + threadIdx.x / TPR;
  const int sub = threadIdx.x % TPR;
  const bool live = row < rows;
  const long long rr = live ? row : rows - 1;
  float x[kN], y[kN];
  Vec16<T>::load(a + (size_t)rr * D + sub * kN, x);
  Vec16<T>::load(b + (size_t)rr * D + sub * kN, y);
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < kN; ++i) acc = fmaf(x[i], y[i], acc);
  acc = group_sum<TPR>(acc);
  if (live && sub == 0) out[row] = acc;
}

// ---- rows between layouts of heads ----------------------------------------------------------
// Copies (batch, heads, rows) of one width into the rows of another, with the heads in another order: destination head hd takes source
// head (hd % a) * b + hd / a; columns that the source does not have are zero, columns that the destination does not have are
// dropped.  One thread per 16-byte piece of the destination, up to three tensors per launch.
struct HeadCopy {
  const uint4* src;
  uint4* dst;
  unsigned pieces;          // of the destination
  int heads, rows, a, b, src_width, dst_width;      // widths in 16-byte pieces
};
struct HeadCopies {
  HeadCopy t[3];
};
__global__ void __launch_bounds__(kMergeThreads) copy_heads_kernel(HeadCopies all) {
  const HeadCopy& t = all.t[blockIdx.y];
  const unsigned e = blockIdx.x * kMergeThreads + threadIdx.x;
  if (e >= t.pieces) return;
  const unsigned row = e / t.dst_width, c = e - row * t.dst_width, bh = row / t.rows, bb = bh / t.heads, hd = bh - bb * t.heads;
  const size_t from = ((size_t)bb * t.heads + (hd % t.a) * t.b + hd / t.a) * t.rows + (row - bh * t.rows);
  t.dst[e] = (int)c < t.src_width ? __ldg(t.src + from * t.src_width + c) : make_uint4(0, 0, 0, 0);
}

// ---- input prologue -----------------------------------------------------------------
// The model hands over projections in token-major order: query_state (b,s,n,d), key_state / value_state (b,s,n_kv,d)
// and gate logits (b,s,2,n_kv).  The operator wants head-major tensors: xq (b,n_kv,rep,s,d) (query head kv*rep + r),
// kc / vc (b,n_kv,s,d), static_src / static_dest (b,n_kv,s) (the reference's driver does this with transposes and
// views, main.py:24-31).  One pass does the transposes and, on request, the two things a model applies on the way
// (Universal_Attention/triton/_debug.py:470-475): keys divided by (|k| + 1e-6) and gates through a sigmoid.
// One group of TPR threads per row of d elements; rows = b * s * (n + 2 n_kv); the blocks behind the rows' take the gates.
// Bound by HBM in 128-byte pieces on the head-major side: B4 L4096, 32 + 8 heads of 64, 200 MB each way: 45 + 5 us forward and
// 64 + 5 us backward with 64-bit index divisions and the gates in launches of their own -> 44 and 62 us.  (A thread that owns one
// slice of a head for several tokens, or several rows, was slower: 46 - 48 us and 65 - 84 us, and twice as slow at 1024 tokens.)
struct PrepDims {
  int b, s, n, n_kv, normalize_keys, sigmoid_gates;
  unsigned rows, row_blocks;
};

// gates (b, s, 2, n_kv) <-> two (b, n_kv, s): f(token-major index, head-major index, which), consecutive threads along s
template <typename F>
__device__ __forceinline__ void prep_gates(const PrepDims& pd, F f) {
  const unsigned total = (unsigned)pd.b * pd.s * 2 * pd.n_kv, stride = (gridDim.x - pd.row_blocks) * kMergeThreads;
  for (unsigned e = (blockIdx.x - pd.row_blocks) * kMergeThreads + threadIdx.x; e < total; e += stride) {
    const unsigned z = e / pd.s, ss = e - z * pd.s, bb = z / (2 * pd.n_kv), y = z - bb * 2 * pd.n_kv, which = y / pd.n_kv, kv = y - which * pd.n_kv;
    f(((size_t)bb * pd.s + ss) * 2 * pd.n_kv + y, ((size_t)bb * pd.n_kv + kv) * pd.s + ss, (int)which);
  }
}

template <typename T, int TPR>
__global__ void __launch_bounds__(kMergeThreads) prepare_fwd_kernel(PrepDims pd, const T* __restrict__ qs, const T* __restrict__ ks,
                                                                    const T* __restrict__ vs, const T* __restrict__ gs, T* __restrict__ xq,
                                                                    T* __restrict__ kc, T* __restrict__ vc, T* __restrict__ ssrc,
                                                                    T* __restrict__ sdest, float* __restrict__ key_norm) {
  if (blockIdx.x >= pd.row_blocks) {
    prep_gates(pd, [&](size_t tm, size_t hm, int which) {
      float x = Num<T>::ld(gs + tm);
      if (pd.sigmoid_gates) x = 1.0f / (1.0f + __expf(-x));
      Num<T>::st((which ? sdest : ssrc) + hm, x);
    });
    return;
  }
  constexpr int kN = Vec16<T>::kN;
  constexpr int D = TPR * kN;
  const unsigned heads = pd.n + 2 * pd.n_kv;
  const unsigned row = blockIdx.x * (kMergeThreads / TPR) + threadIdx.x / TPR;
  const int sub = threadIdx.x % TPR;
  const bool live = row < pd.rows;
  const unsigned rr = live ? row : pd.rows - 1, tok = rr / heads, bb = tok / pd.s;      // tok = bb * s + ss
  const int hh = (int)(rr - tok * heads), ss = (int)(tok - bb * pd.s);
  const bool is_q = hh < pd.n, is_k = !is_q && hh < pd.n + pd.n_kv;
  const int kv = is_q ? 0 : (is_k ? hh - pd.n : hh - pd.n - pd.n_kv);
  const size_t hm = ((size_t)bb * pd.n_kv + kv) * pd.s + ss;          // head-major row of a key / value
  float v[kN];
  if (is_q) Vec16<T>::load(qs + ((size_t)tok * pd.n + hh) * D + sub * kN, v);
  else Vec16<T>::load((is_k ? ks : vs) + ((size_t)tok * pd.n_kv + kv) * D + sub * kN, v);
  float ssq = 0.f;
#pragma unroll
  for (int i = 0; i < kN; ++i) ssq = fmaf(v[i], v[i], ssq);
  ssq = group_sum<TPR>(ssq);                        // every lane takes part, whatever kind of row its group holds
  const float nrm = sqrtf(ssq);
  if (is_k && pd.normalize_keys) {
    const float inv = 1.0f / (nrm + 1e-6f);
#pragma unroll
    for (int i = 0; i < kN; ++i) v[i] *= inv;
  }
  if (!live) return;
  if (is_q) {
    Vec16<T>::store(xq + (((size_t)bb * pd.n + hh) * pd.s + ss) * D + sub * kN, v);
  } else {
    Vec16<T>::store((is_k ? kc : vc) + hm * D + sub * kN, v);
    if (is_k && sub == 0 && key_norm) key_norm[hm] = nrm;
  }
}

// backward of prepare_fwd_kernel: gradients flow back along the same row mapping; key rows pass through the
// derivative of k / (|k| + eps):  dk = g / (|k| + eps) - khat (g . khat) / |k|
template <typename T, int TPR>
__global__ void __launch_bounds__(kMergeThreads) prepare_bwd_kernel(PrepDims pd, const T* __restrict__ g_xq, const T* __restrict__ g_kc,
                                                                    const T* __restrict__ g_vc, const T* __restrict__ g_src,
                                                                    const T* __restrict__ g_dest, const T* __restrict__ kc,
                                                                    const float* __restrict__ key_norm, const T* __restrict__ ssrc,
                                                                    const T* __restrict__ sdest, T* __restrict__ d_qs, T* __restrict__ d_ks,
                                                                    T* __restrict__ d_vs, T* __restrict__ d_gs) {
  if (blockIdx.x >= pd.row_blocks) {
    prep_gates(pd, [&](size_t tm, size_t hm, int which) {
      // ssrc / sdest hold the forward's outputs (the gate values), g_* their gradients
      const float gate = Num<T>::ld((which ? sdest : ssrc) + hm);
      float g = Num<T>::ld((which ? g_dest : g_src) + hm);
      if (pd.sigmoid_gates) g *= gate * (1.0f - gate);
      Num<T>::st(d_gs + tm, g);
    });
    return;
  }
  constexpr int kN = Vec16<T>::kN;
  constexpr int D = TPR * kN;
  const unsigned heads = pd.n + 2 * pd.n_kv;
  const unsigned row = blockIdx.x * (kMergeThreads / TPR) + threadIdx.x / TPR;
  const int sub = threadIdx.x % TPR;
  const bool live = row < pd.rows;
  const unsigned rr = live ? row : pd.rows - 1, tok = rr / heads, bb = tok / pd.s;      // tok = bb * s + ss
  const int hh = (int)(rr - tok * heads), ss = (int)(tok - bb * pd.s);
  const bool is_q = hh < pd.n, is_k = !is_q && hh < pd.n + pd.n_kv;
  const int kv = is_q ? 0 : (is_k ? hh - pd.n : hh - pd.n - pd.n_kv);
  const size_t hm = ((size_t)bb * pd.n_kv + kv) * pd.s + ss;
  float g[kN], kh[kN];
  if (is_q) Vec16<T>::load(g_xq + (((size_t)bb * pd.n + hh) * pd.s + ss) * D + sub * kN, g);
  else Vec16<T>::load((is_k ? g_kc : g_vc) + hm * D + sub * kN, g);
  float dot = 0.f;
  const bool norm = is_k && pd.normalize_keys;
  if (norm) {
    Vec16<T>::load(kc + hm * D + sub * kN, kh);
#pragma unroll
    for (int i = 0; i < kN; ++i) dot = fmaf(g[i], kh[i], dot);
  }
  dot = group_sum<TPR>(dot);
  if (norm) {
    const float nrm = key_norm[hm];
    const float a = 1.0f / (nrm + 1e-6f), c = nrm > 0.f ? dot / nrm : 0.f;
#pragma unroll
    for (int i = 0; i < kN; ++i) g[i] = g[i] * a - kh[i] * c;
  }
  if (!live) return;
  if (is_q) Vec16<T>::store(d_qs + ((size_t)tok * pd.n + hh) * D + sub * kN, g);
  else Vec16<T>::store((is_k ? d_ks : d_vs) + ((size_t)tok * pd.n_kv + kv) * D + sub * kN, g);
}

}  // namespace aux
}  // namespace ua
