// Tiled fp32 kernels of the Universal Attention operator: fp32 mode, and bf16 shapes that the tensor-core kernels do not take,
// for chunks of 32, 64 or 128 keys and head dims up to 128 (see tiled::fits).
//
// One block per (b, h, chunk i, 32 rows[, query head]): nothing is swept, so the problem is as parallel as it has tiles.  What runs
// along the rows -- the decay prefix upwards, the sum of its gradient downwards -- crosses tiles through per-tile totals:
//   totals_kernel      log-retention sum of every key over every tile
//   forward_kernel     prefix = totals of the tiles before + scan of the tile; scores, softmax, P V
//   backward_kernel    the same up to P, then dP, dS; dV, dK, dQ; dC = dS summed over the heads, and its total per tile
//   decay_kernel       reverse sum = totals of the tiles after + scan of the tile; affinity gradient, dK, d src, d dest
// All products are 32 x C x D on 256 threads, 4 x (C / 32) results per thread from 16-byte shared-memory reads (rows padded by 16
// bytes: conflict free), fp32 throughout; bf16 inputs are widened on load, and P and dS / dG are rounded to the input type before
// their products as the reference does (universal_attention_autograd.py:159, :245, :251).  Bound by the fp32 FMA rate once there
// are tiles for every SM, by the latency of one block (about 5 us) below.
// Against one block per chunk that sweeps all rows (ua_simt.cuh), fp32 B1 H2 R2 L256 c64 D64: forward 588 -> 21 us,
// backward 1221 -> 42 us.
#pragma once
#include "ua_common.cuh"
#include "ua_tiled_host.h"

namespace ua {
namespace tiled {

constexpr int kThreads = 256;

// shared memory in floats; tiles of rows have a pitch of D + 4, planes [32 rows][C keys] one of C + 4
template <int C> struct Lay {
  int DP, oK, oV, oKj, oQ, oG, oS, oD, oVec, total;
  __host__ __device__ Lay(int D, int row_tiles, bool v, bool two_planes) {
    DP = D + 4;
    oK = 0;
    oV = oK + C * DP;
    oKj = oV + (v ? C * DP : 0);
    oQ = oKj + kRows * DP;
    oG = oQ + (row_tiles > 1 ? kRows * DP : 0);
    oS = oG + (row_tiles > 2 ? kRows * DP : 0);
    oD = oS + kRows * (C + 4);
    oVec = oD + (two_planes ? kRows * (C + 4) : 0);
    total = oVec + 2 * C + 4 * kRows;      // s3[C], base[C], t3[32], three row vectors
  }
};

__device__ __forceinline__ float pow23(float g) { return g > 0.f ? powf(g, 2.0f / 3.0f) : 0.f; }
__device__ __forceinline__ float log_retention(float a) { return log1pf(-fminf(fmaxf(a, 0.f), clamp_hi())); }

template <typename T> __device__ __forceinline__ float4 ld4(const T* p);
template <> __device__ __forceinline__ float4 ld4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 ld4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 x = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(x.x << 16), __uint_as_float(x.x & 0xffff0000u), __uint_as_float(x.y << 16), __uint_as_float(x.y & 0xffff0000u));
}
template <typename T> __device__ __forceinline__ void st4(T* p, float4 v) {
  Num<T>::st(p, v.x); Num<T>::st(p + 1, v.y); Num<T>::st(p + 2, v.z); Num<T>::st(p + 3, v.w);
}
template <> __device__ __forceinline__ void st4<float>(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
template <> __device__ __forceinline__ void st4<__nv_bfloat16>(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

template <typename T>
__device__ __forceinline__ void load_rows(float* dst, const T* src, int rows, int D, int DP) {
  const int d4 = D >> 2;
  for (int e = threadIdx.x; e < rows * d4; e += kThreads) {
    const int r = e / d4, c = (e - r * d4) * 4;
    *reinterpret_cast<float4*>(dst + r * DP + c) = ld4<T>(src + (size_t)r * D + c);
  }
}
__device__ __forceinline__ void red4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// (one chain in ascending order: the Gram values come out bit for bit as in the sweeping kernels.  Near zero, where the decay
// gradient goes with g^(-1/3), another order of the same sum moves dK by 1e-4.)
__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) { return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc)))); }
__device__ __forceinline__ void axpy4(float4& acc, float a, float4 b) {
  acc.x = fmaf(a, b.x, acc.x); acc.y = fmaf(a, b.y, acc.y); acc.z = fmaf(a, b.z, acc.z); acc.w = fmaf(a, b.w, acc.w);
}

// A thread's share of a [32 rows][C keys] plane: keys kt + (C / 4) y, rows qt + kQS z.
template <int C> struct Own {
  static constexpr int kKT = C / 4, kQS = kThreads / kKT, kQ = kRows / kQS;      // kQ = 1, 2, 4 for C = 32, 64, 128
};

// acc[y][z] = A[key] . B[row] over D
template <int C>
__device__ __forceinline__ void plane_product(const float* A, const float* B, int D, int DP, float (&acc)[4][Own<C>::kQ]) {
  using O = Own<C>;
  const int kt = threadIdx.x % O::kKT, qt = threadIdx.x / O::kKT;
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < O::kQ; ++z) acc[y][z] = 0.f;
#pragma unroll 4
  for (int d = 0; d < D; d += 4) {
    float4 a[4], b[O::kQ];
#pragma unroll
    for (int y = 0; y < 4; ++y) a[y] = *reinterpret_cast<const float4*>(A + (kt + O::kKT * y) * DP + d);
#pragma unroll
    for (int z = 0; z < O::kQ; ++z) b[z] = *reinterpret_cast<const float4*>(B + (qt + O::kQS * z) * DP + d);
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int z = 0; z < O::kQ; ++z) acc[y][z] = dot4(a[y], b[z], acc[y][z]);
  }
}

// rows of the result: f(row, column of four, sum_k X[row][k] Y[k][..]) for a plane X [32][C + 4] and key rows Y [C][DP]
template <int C, typename F>
__device__ __forceinline__ void rows_product(const float* X, const float* Y, int D, int DP, F f) {
  const int d4 = D >> 2;
  // two rows per thread where there is work for all threads in that form
  for (int e = threadIdx.x; e < 16 * d4; e += kThreads) {
    const int q = e / d4, c = (e - q * d4) * 4;
    float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
    const float *x0 = X + q * (C + 4), *x1 = X + (q + 16) * (C + 4);
#pragma unroll 4
    for (int k = 0; k < C; k += 4) {
      const float4 p = *reinterpret_cast<const float4*>(x0 + k), r = *reinterpret_cast<const float4*>(x1 + k);
      const float4 y0 = *reinterpret_cast<const float4*>(Y + (k + 0) * DP + c), y1 = *reinterpret_cast<const float4*>(Y + (k + 1) * DP + c);
      const float4 y2 = *reinterpret_cast<const float4*>(Y + (k + 2) * DP + c), y3 = *reinterpret_cast<const float4*>(Y + (k + 3) * DP + c);
      axpy4(a0, p.x, y0); axpy4(a0, p.y, y1); axpy4(a0, p.z, y2); axpy4(a0, p.w, y3);
      axpy4(a1, r.x, y0); axpy4(a1, r.y, y1); axpy4(a1, r.z, y2); axpy4(a1, r.w, y3);
    }
    f(q, c, a0);
    f(q + 16, c, a1);
  }
}
// keys of the result: global rows dst[key][..] += sum_q X[q][key] Z[q][..]
template <int C>
__device__ __forceinline__ void keys_product_add(const float* X, const float* Z, int D, int DP, float* dst) {
  const int d4 = D >> 2;
  for (int e = threadIdx.x; e < (C / 4) * d4; e += kThreads) {
    const int k = e / d4 * 4, c = (e % d4) * 4;
    float4 a[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) a[y] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int q = 0; q < kRows; ++q) {
      const float4 x = *reinterpret_cast<const float4*>(X + q * (C + 4) + k), z = *reinterpret_cast<const float4*>(Z + q * DP + c);
      axpy4(a[0], x.x, z); axpy4(a[1], x.y, z); axpy4(a[2], x.z, z); axpy4(a[3], x.w, z);
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) red4(dst + (size_t)(k + y) * D + c, a[y]);
  }
}

struct Where {
  int i, bh, j0, jt;       // chunk, unit, first row of the tile, tile number
};
// Block -> (tile, chunk, unit): valid tiles only (those that reach the chunk's first row), chunk 0 (most tiles) first; or all tiles.
template <int C>
__device__ __forceinline__ Where locate(const Shape& s, int block, bool all) {
  const int BH = s.B * s.H, T = s.L / kRows;
  Where w;
  w.bh = block % BH;
  int x = block / BH;
  if (all) {
    w.i = x / T;
    w.jt = T - 1 - x % T;
  } else {
    for (w.i = 0;; ++w.i) {
      const int nt = T - w.i * (C / kRows);
      if (x < nt) break;
      x -= nt;
    }
    w.jt = T - 1 - x;
  }
  w.j0 = w.jt * kRows;
  return w;
}

// gates: s3[C] of the chunk's keys, t3[32] of the tile's rows
template <int C, typename TG>
__device__ __forceinline__ void load_gates(const Params& p, const Where& w, float* s3, float* t3) {
  const TG* ss = static_cast<const TG*>(p.ssrc) + (size_t)w.bh * p.s.L + (size_t)w.i * C;
  const TG* sd = static_cast<const TG*>(p.sdest) + (size_t)w.bh * p.s.L + w.j0;
  if (threadIdx.x < C) s3[threadIdx.x] = cbrtf(Num<TG>::ld(ss + threadIdx.x));
  else if (threadIdx.x >= 128 && threadIdx.x < 128 + kRows) t3[threadIdx.x - 128] = cbrtf(Num<TG>::ld(sd + threadIdx.x - 128));
}

// log-retention of the thread's pairs -> plane S (zero at and before the key)
template <int C>
__device__ __forceinline__ void retention_plane(const Where& w, const float (&g)[4][Own<C>::kQ], const float* s3, const float* t3, float* S) {
  using O = Own<C>;
  const int kt = threadIdx.x % O::kKT, qt = threadIdx.x / O::kKT;
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < O::kQ; ++z) {
      const int k = kt + O::kKT * y, q = qt + O::kQS * z;
      S[q * (C + 4) + k] = (w.j0 + q <= w.i * C + k) ? 0.f : log_retention(pow23(g[y][z]) * s3[k] * t3[q]);
    }
}

// ---------------------------------------------------------------------------------- totals --
template <int C, typename T, typename TG>
__global__ void __launch_bounds__(kThreads) totals_kernel(Params p) {
  extern __shared__ __align__(16) float sm[];
  const int D = p.s.D;
  const Lay<C> l(D, 1, false, false);
  const Where w = locate<C>(p.s, blockIdx.x, false);
  float *s3 = sm + l.oVec, *t3 = s3 + 2 * C, *S = sm + l.oS;
  const T* kc = static_cast<const T*>(p.kc) + (size_t)w.bh * p.s.L * D;
  load_rows<T>(sm + l.oK, kc + (size_t)w.i * C * D, C, D, l.DP);
  load_rows<T>(sm + l.oKj, kc + (size_t)w.j0 * D, kRows, D, l.DP);
  load_gates<C, TG>(p, w, s3, t3);
  __syncthreads();
  float g[4][Own<C>::kQ];
  plane_product<C>(sm + l.oK, sm + l.oKj, D, l.DP, g);
  retention_plane<C>(w, g, s3, t3, S);
  __syncthreads();
  if (threadIdx.x < C) {
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < kRows; ++q) sum += S[q * (C + 4) + threadIdx.x];
    p.totals[(((size_t)w.bh * p.s.N + w.i) * (p.s.L / kRows) + w.jt) * C + threadIdx.x] = sum;
  }
}

// sum of a table's tiles [lo, hi) for key threadIdx.x, into dst[C]
template <int C>
__device__ __forceinline__ void sum_tiles(const Params& p, const Where& w, const float* table, int lo, int hi, float* dst) {
  if (threadIdx.x < C) {
    const float* t = table + ((size_t)w.bh * p.s.N + w.i) * (p.s.L / kRows) * C + threadIdx.x;
    float sum = 0.f;
#pragma unroll 8
    for (int j = lo; j < hi; ++j) sum += t[(size_t)j * C];
    dst[threadIdx.x] = sum;
  }
}

// Plane S := decay prefix (mask value before the key).  Needs K_i, K_j, gates and base in shared memory; begins and ends with
// all threads past a barrier.
template <int C>
__device__ __forceinline__ void prefix_plane(const Params& p, const Where& w, const Lay<C>& l, float* sm) {
  float *s3 = sm + l.oVec, *base = s3 + C, *t3 = base + C, *S = sm + l.oS;
  float g[4][Own<C>::kQ];
  plane_product<C>(sm + l.oK, sm + l.oKj, p.s.D, l.DP, g);
  retention_plane<C>(w, g, s3, t3, S);
  __syncthreads();
  if (threadIdx.x < C) {
    const float b = base[threadIdx.x];
    float local = 0.f;
#pragma unroll
    for (int q = 0; q < kRows; ++q) {
      float* at = S + q * (C + 4) + threadIdx.x;
      local += *at;
      *at = (w.j0 + q < w.i * C + (int)threadIdx.x) ? mask_value() : local + b;
    }
  }
  __syncthreads();
}

// Plane S += K_i Q^T
template <int C>
__device__ __forceinline__ void add_scores(const Lay<C>& l, float* sm, int D) {
  using O = Own<C>;
  const int kt = threadIdx.x % O::kKT, qt = threadIdx.x / O::kKT;
  float acc[4][O::kQ];
  plane_product<C>(sm + l.oK, sm + l.oQ, D, l.DP, acc);
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < O::kQ; ++z) sm[l.oS + (qt + O::kQS * z) * (C + 4) + kt + O::kKT * y] += acc[y][z];
}

template <typename F> __device__ __forceinline__ float warp_all(float v, F f) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_max(float v) { return warp_all(v, [](float a, float b) { return fmaxf(a, b); }); }
__device__ __forceinline__ float warp_sum(float v) { return warp_all(v, [](float a, float b) { return a + b; }); }

// --------------------------------------------------------------------------------- forward --
template <int C, typename T, typename TG>
__global__ void __launch_bounds__(kThreads) forward_kernel(Params p) {
  extern __shared__ __align__(16) float sm[];
  const int D = p.s.D, L = p.s.L, R = p.s.R, N = p.s.N, r = blockIdx.y;
  const Lay<C> l(D, 2, true, false);
  const Where w = locate<C>(p.s, blockIdx.x, p.fill_masked != 0);
  const T* kc = static_cast<const T*>(p.kc) + (size_t)w.bh * L * D;
  const T* vc = static_cast<const T*>(p.vc) + (size_t)w.bh * L * D;
  const size_t row0 = (((size_t)w.bh * N + w.i) * R + r) * L + w.j0;
  T* out = static_cast<T*>(p.out) + row0 * D;
  float* S = sm + l.oS;
  load_rows<T>(sm + l.oV, vc + (size_t)w.i * C * D, C, D, l.DP);
  if (w.j0 + kRows <= w.i * C) {
    // rows before the chunk: uniform softmax (universal_attention_autograd.py:28, :154)
    __syncthreads();
    const float wgt = Num<T>::rnd(1.0f / (float)C);
    for (int c = threadIdx.x * 4; c < D; c += 4 * kThreads) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = 0; k < C; ++k) axpy4(acc, wgt, *reinterpret_cast<const float4*>(sm + l.oV + k * l.DP + c));
      *reinterpret_cast<float4*>(S + c) = acc;
    }
    __syncthreads();
    for (int e = threadIdx.x * 4; e < kRows * D; e += 4 * kThreads) st4<T>(out + e, *reinterpret_cast<const float4*>(S + e % D));
    if (threadIdx.x < kRows) {
      p.lse[row0 + threadIdx.x] = mask_value();
      if (p.denom) Num<T>::st(static_cast<T*>(p.denom) + row0 + threadIdx.x, mask_value());
    }
    return;
  }
  load_rows<T>(sm + l.oK, kc + (size_t)w.i * C * D, C, D, l.DP);
  load_rows<T>(sm + l.oKj, kc + (size_t)w.j0 * D, kRows, D, l.DP);
  load_rows<T>(sm + l.oQ, static_cast<const T*>(p.xq) + (((size_t)w.bh * R + r) * L + w.j0) * D, kRows, D, l.DP);
  load_gates<C, TG>(p, w, sm + l.oVec, sm + l.oVec + 2 * C);
  sum_tiles<C>(p, w, p.totals, w.i * (C / kRows), w.jt, sm + l.oVec + C);
  __syncthreads();
  prefix_plane<C>(p, w, l, sm);
  add_scores<C>(l, sm, D);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = warp; q < kRows; q += kThreads / 32) {
    float e[C / 32], m = -INFINITY, z = 0.f;
#pragma unroll
    for (int x = 0; x < C / 32; ++x) m = fmaxf(m, e[x] = S[q * (C + 4) + x * 32 + lane]);
    m = warp_max(m);
#pragma unroll
    for (int x = 0; x < C / 32; ++x) z += e[x] = expf(e[x] - m);
    z = warp_sum(z);
#pragma unroll
    for (int x = 0; x < C / 32; ++x) S[q * (C + 4) + x * 32 + lane] = Num<T>::rnd(e[x] / z);
    if (lane == 0) {
      const float v = m + logf(z);
      p.lse[row0 + q] = v;
      if (p.denom) Num<T>::st(static_cast<T*>(p.denom) + row0 + q, v);
    }
  }
  __syncthreads();
  rows_product<C>(S, sm + l.oV, D, l.DP, [&](int q, int c, float4 v) { st4<T>(out + (size_t)q * D + c, v); });
}

// -------------------------------------------------------------------------------- backward --
template <int C, typename T, typename TG>
__global__ void __launch_bounds__(kThreads) backward_kernel(Params p) {
  extern __shared__ __align__(16) float sm[];
  using O = Own<C>;
  const int D = p.s.D, L = p.s.L, R = p.s.R, N = p.s.N, r = blockIdx.y;
  const Lay<C> l(D, 3, true, true);
  const Where w = locate<C>(p.s, blockIdx.x, p.skip_masked == 0);
  const bool masked = w.j0 + kRows <= w.i * C;
  if (p.only_masked && !masked) return;
  const T* kc = static_cast<const T*>(p.kc) + (size_t)w.bh * L * D;
  const T* vc = static_cast<const T*>(p.vc) + (size_t)w.bh * L * D;
  const size_t chunk_id = (size_t)w.bh * N + w.i, row0 = (chunk_id * R + r) * L + w.j0;
  const size_t qrow0 = ((size_t)w.bh * R + r) * L + w.j0;
  float *S = sm + l.oS, *Dp = sm + l.oD, *gd = sm + l.oVec + 2 * C + kRows;
  load_rows<T>(sm + l.oK, kc + (size_t)w.i * C * D, C, D, l.DP);
  load_rows<T>(sm + l.oV, vc + (size_t)w.i * C * D, C, D, l.DP);
  load_rows<T>(sm + l.oQ, static_cast<const T*>(p.xq) + qrow0 * D, kRows, D, l.DP);
  load_rows<T>(sm + l.oG, static_cast<const T*>(p.g_out) + row0 * D, kRows, D, l.DP);
  if (threadIdx.x >= 192 && threadIdx.x < 192 + kRows) {
    const size_t at = row0 + threadIdx.x - 192;
    gd[threadIdx.x - 192] = p.g_denom_is_f32 ? static_cast<const float*>(p.g_denom)[at] : Num<T>::ld(static_cast<const T*>(p.g_denom) + at);
  }
  if (!masked) {
    load_rows<T>(sm + l.oKj, kc + (size_t)w.j0 * D, kRows, D, l.DP);
    load_gates<C, TG>(p, w, sm + l.oVec, sm + l.oVec + 2 * C);
    sum_tiles<C>(p, w, p.totals, w.i * (C / kRows), w.jt, sm + l.oVec + C);
    __syncthreads();
    prefix_plane<C>(p, w, l, sm);
    add_scores<C>(l, sm, D);
  } else {
    for (int e = threadIdx.x; e < kRows * (C + 4); e += kThreads) S[e] = mask_value();
    __syncthreads();
  }
  {
    const int kt = threadIdx.x % O::kKT, qt = threadIdx.x / O::kKT;
    float acc[4][O::kQ];
    plane_product<C>(sm + l.oV, sm + l.oG, D, l.DP, acc);
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int z = 0; z < O::kQ; ++z) Dp[(qt + O::kQS * z) * (C + 4) + kt + O::kKT * y] = acc[y][z];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* dc = p.dc + ((chunk_id * (L / kRows) + w.jt) * kRows) * C;
#pragma unroll
  for (int q = warp; q < kRows; q += kThreads / 32) {
    float e[C / 32], dp[C / 32], m = -INFINITY, z = 0.f, delta = 0.f;
#pragma unroll
    for (int x = 0; x < C / 32; ++x) {
      m = fmaxf(m, e[x] = S[q * (C + 4) + x * 32 + lane]);
      dp[x] = Dp[q * (C + 4) + x * 32 + lane];
    }
    m = warp_max(m);
#pragma unroll
    for (int x = 0; x < C / 32; ++x) z += e[x] = expf(e[x] - m);
    const float zinv = 1.0f / warp_sum(z);
#pragma unroll
    for (int x = 0; x < C / 32; ++x) delta = fmaf(e[x] *= zinv, dp[x], delta);
    delta = warp_sum(delta);
#pragma unroll
    for (int x = 0; x < C / 32; ++x) {
      const int k = x * 32 + lane;
      const float ds = e[x] * (dp[x] - delta) + e[x] * gd[q];
      if (!masked) {
        if (R > 1) atomicAdd(dc + q * C + k, ds);
        else dc[q * C + k] = ds;
      }
      S[q * (C + 4) + k] = Num<T>::rnd(e[x]);
      Dp[q * (C + 4) + k] = Num<T>::rnd(ds);
    }
  }
  __syncthreads();
  keys_product_add<C>(S, sm + l.oG, D, l.DP, p.acc_dv + ((size_t)w.bh * L + (size_t)w.i * C) * D);        // dV_i += P dO
  keys_product_add<C>(Dp, sm + l.oQ, D, l.DP, p.acc_dk + ((size_t)w.bh * L + (size_t)w.i * C) * D);       // dK_i += dS Q
  rows_product<C>(Dp, sm + l.oK, D, l.DP, [&](int q, int c, float4 v) { red4(p.acc_dq + (qrow0 + q) * D + c, v); });      // dQ_j += dS^T K_i
}

// sums of dC over the rows of every tile: block per (tile, chunk, unit), thread = key
template <int C>
__global__ void __launch_bounds__(C) dc_totals_kernel(Params p) {
  const Where w = locate<C>(p.s, blockIdx.x, false);
  const size_t tile = ((size_t)w.bh * p.s.N + w.i) * (p.s.L / kRows) + w.jt;
  float sum = 0.f;
#pragma unroll
  for (int q = 0; q < kRows; ++q) sum += p.dc[(tile * kRows + q) * C + threadIdx.x];
  p.dc_total[tile * C + threadIdx.x] = sum;
}

template <int C, typename T, typename TG>
__global__ void __launch_bounds__(kThreads) decay_kernel(Params p) {
  extern __shared__ __align__(16) float sm[];
  using O = Own<C>;
  const int D = p.s.D, L = p.s.L, N = p.s.N;
  const Lay<C> l(D, 1, false, true);
  const Where w = locate<C>(p.s, blockIdx.x, false);
  const T* kc = static_cast<const T*>(p.kc) + (size_t)w.bh * L * D;
  float *s3 = sm + l.oVec, *suffix = s3 + C, *t3 = suffix + C, *S = sm + l.oS, *Dg = sm + l.oD;
  const size_t tile = ((size_t)w.bh * N + w.i) * (L / kRows) + w.jt;
  load_rows<T>(sm + l.oK, kc + (size_t)w.i * C * D, C, D, l.DP);
  load_rows<T>(sm + l.oKj, kc + (size_t)w.j0 * D, kRows, D, l.DP);
  load_rows<float>(S, p.dc + tile * kRows * C, kRows, C, C + 4);
  load_gates<C, TG>(p, w, s3, t3);
  sum_tiles<C>(p, w, p.dc_total, w.jt + 1, L / kRows, suffix);
  __syncthreads();
  // S := sum of dC over this row and all after it (zero at and before the key)
  if (threadIdx.x < C) {
    const float b = suffix[threadIdx.x];
    float run = 0.f;
#pragma unroll
    for (int q = kRows - 1; q >= 0; --q) {
      float* at = S + q * (C + 4) + threadIdx.x;
      run += *at;
      *at = (w.j0 + q <= w.i * C + (int)threadIdx.x) ? 0.f : run + b;
    }
  }
  float g[4][O::kQ];
  plane_product<C>(sm + l.oK, sm + l.oKj, D, l.DP, g);
  __syncthreads();
  const int kt = threadIdx.x % O::kKT, qt = threadIdx.x / O::kKT;
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < O::kQ; ++z) {
      const int k = kt + O::kKT * y, q = qt + O::kQS * z, at = q * (C + 4) + k;
      const float gv = g[y][z], pw = pow23(gv), a = pw * s3[k] * t3[q];
      float da = S[at] / (fminf(fmaxf(a, clamp_lo_bwd()), clamp_hi()) - 1.0f);
      if (!(a <= clamp_hi())) da = 0.f;
      S[at] = da * pw;                                       // d (s^(1/3) t^(1/3))
      float dg = Num<T>::rnd(da * s3[k] * t3[q]);
      dg = (gv > 0.f) ? dg * (2.0f / 3.0f) * powf(fabsf(gv) + 1e-9f, -1.0f / 3.0f) : 0.f;
      Dg[at] = Num<T>::rnd(dg);
    }
  __syncthreads();
  if (threadIdx.x < C) {
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < kRows; ++q) sum = fmaf(S[q * (C + 4) + threadIdx.x], t3[q], sum);
    const float c = s3[threadIdx.x];
    if (sum != 0.f) atomicAdd(p.acc_ds + (size_t)w.bh * L + (size_t)w.i * C + threadIdx.x, sum / (3.0f * c * c));
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int q = warp; q < kRows; q += kThreads / 32) {
    float sum = 0.f;
#pragma unroll
    for (int x = 0; x < C / 32; ++x) sum = fmaf(S[q * (C + 4) + x * 32 + lane], s3[x * 32 + lane], sum);
    sum = warp_sum(sum);
    if (lane == 0 && sum != 0.f) atomicAdd(p.acc_dt + (size_t)w.bh * L + w.j0 + q, sum / (3.0f * t3[q] * t3[q]));
  }
  rows_product<C>(Dg, sm + l.oK, D, l.DP, [&](int q, int c, float4 v) { red4(p.acc_dk + ((size_t)w.bh * L + w.j0 + q) * D + c, v); });      // dK_j += dG^T K_i
  keys_product_add<C>(Dg, sm + l.oKj, D, l.DP, p.acc_dk + ((size_t)w.bh * L + (size_t)w.i * C) * D);                                        // dK_i += dG K_j
}

template <typename T, typename TG>
__global__ void __launch_bounds__(kThreads) leave_kernel(Leave v) {
  const size_t stride = (size_t)gridDim.x * kThreads;
#pragma unroll
  for (int t = 0; t < 5; ++t)
    for (size_t e = (size_t)blockIdx.x * kThreads + threadIdx.x; e < v.n[t] / 4; e += stride) {
      const float4 x = reinterpret_cast<const float4*>(v.src[t])[e];
      if (v.gate[t]) st4<TG>(static_cast<TG*>(v.dst[t]) + 4 * e, x);
      else st4<T>(static_cast<T*>(v.dst[t]) + 4 * e, x);
    }
}

// ---- host side ---------------------------------------------------------------------------------
template <int C> inline int smem_of(int D, int kernel) {      // 0 totals, 1 forward, 2 backward, 3 decay
  const int rows[4] = {1, 2, 3, 1};
  return 4 * Lay<C>(D, rows[kernel], kernel == 1 || kernel == 2, kernel >= 2).total;
}
inline unsigned valid_tiles(const Shape& s) {
  unsigned n = 0;
  for (int i = 0; i < s.N; ++i) n += s.L / kRows - i * (s.C / kRows);
  return n * (unsigned)(s.B * s.H);
}
template <typename K> inline bool launch(K kern, dim3 grid, int threads, int smem, const Params& p, cudaStream_t st) {
  if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return false;
  kern<<<grid, threads, smem, st>>>(p);
  return true;
}
template <int C, typename T, typename TG> bool forward_c(const Params& p, cudaStream_t st) {
  const unsigned tiles = valid_tiles(p.s), all = (unsigned)(p.s.B * p.s.H * p.s.N * (p.s.L / kRows));
  return launch(totals_kernel<C, T, TG>, dim3(tiles), kThreads, smem_of<C>(p.s.D, 0), p, st) &&
         launch(forward_kernel<C, T, TG>, dim3(p.fill_masked ? all : tiles, p.s.R), kThreads, smem_of<C>(p.s.D, 1), p, st);
}
template <int C, typename T, typename TG> bool backward_c(const Params& p, cudaStream_t st) {
  const unsigned tiles = valid_tiles(p.s), all = (unsigned)(p.s.B * p.s.H * p.s.N * (p.s.L / kRows));
  if (p.only_masked) return launch(backward_kernel<C, T, TG>, dim3(all, p.s.R), kThreads, smem_of<C>(p.s.D, 2), p, st);
  return launch(totals_kernel<C, T, TG>, dim3(tiles), kThreads, smem_of<C>(p.s.D, 0), p, st) &&
         launch(backward_kernel<C, T, TG>, dim3(p.skip_masked ? tiles : all, p.s.R), kThreads, smem_of<C>(p.s.D, 2), p, st) &&
         launch(dc_totals_kernel<C>, dim3(tiles), C, 0, p, st) &&
         launch(decay_kernel<C, T, TG>, dim3(tiles), kThreads, smem_of<C>(p.s.D, 3), p, st);
}
template <typename T, typename TG> bool forward_t(const Params& p, cudaStream_t st) {
  return p.s.C == 32 ? forward_c<32, T, TG>(p, st) : p.s.C == 64 ? forward_c<64, T, TG>(p, st) : forward_c<128, T, TG>(p, st);
}
template <typename T, typename TG> bool backward_t(const Params& p, cudaStream_t st) {
  return p.s.C == 32 ? backward_c<32, T, TG>(p, st) : p.s.C == 64 ? backward_c<64, T, TG>(p, st) : backward_c<128, T, TG>(p, st);
}

}  // namespace tiled
}  // namespace ua
