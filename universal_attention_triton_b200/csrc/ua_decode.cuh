// Incremental (decode) step of the Universal Attention operator: ONE new row against cached keys and values.
//
// The operator's forward (universal_attention_autograd.py:9-38, row-chunked form :104-163) needs, for a new row t and
// every earlier key k, the decay prefix  C[k, t] = sum_{k < q <= t} log1p(-affinity(k, q)).  That prefix is a running
// sum per key, so a serving loop keeps it as state next to the key / value caches:
//     state[k] <- state[k] + log1p(-clamp(relu(k_k . k_t)^(2/3) src_k^(1/3) dest_t^(1/3)))     for k < t
//     state[t]  = 0
// and the new row's outputs are, per key chunk i of `chunk` keys (only the chunks that hold keys <= t exist),
//     lse[r][i] = logsumexp_k (k_k . q_r + state[k]),     out[r][i][:] = sum_k softmax_k(...) v_k
// exactly row t of the full forward.  O(t * d) work and cache reads per step: HBM-bound, one block per (b, h, chunk),
// one thread per key of the chunk, fp32 CUDA-core arithmetic (no tile is large enough for the tensor cores).
#pragma once
#include "ua_aux.cuh"
#include "ua_common.cuh"

namespace ua {
namespace decode {

struct Params {
  int BH, R, D, C;        // (batch * kv heads), query heads per kv head, head_dim, keys per chunk (= threads per block)
  int Lcap;               // rows of the caches per (b, h)
  int t;                  // position of the new row; keys 0..t are in the caches
  const void* kcache;     // (BH, Lcap, D)
  const void* vcache;     // (BH, Lcap, D)
  const void* src;        // (BH, Lcap) gate of the keys
  const void* q;          // (BH, R, D) queries of the new row
  const void* dest;       // (BH) gate of the new row
  float* state;           // (BH, Lcap) decay prefix, updated in place
  void* out;              // (BH, nt, R, D), nt = t / C + 1
  float* lse;             // (BH, nt, R)
};

constexpr int kMaxR = 8;

template <typename T, typename TG>
__global__ void step_kernel(Params p) {
  extern __shared__ float sm[];
  const int D = p.D, R = p.R, C = p.C;
  float* s_kt = sm;                    // [D]   key of the new row
  float* s_q = s_kt + D;               // [R][D]
  float* s_p = s_q + R * D;            // [R][C] probabilities
  float* s_red = s_p + R * C;          // [2][kMaxR][32] warp partials
  const int bh = blockIdx.x, i = blockIdx.y, tid = threadIdx.x;
  const int nt = p.t / C + 1;
  const T* kc = static_cast<const T*>(p.kcache) + (size_t)bh * p.Lcap * D;
  const T* vc = static_cast<const T*>(p.vcache) + (size_t)bh * p.Lcap * D;
  for (int e = tid; e < D; e += C) s_kt[e] = Num<T>::ld(kc + (size_t)p.t * D + e);
  for (int e = tid; e < R * D; e += C) s_q[e] = Num<T>::ld(static_cast<const T*>(p.q) + (size_t)bh * R * D + e);
  __syncthreads();

  const int kk = i * C + tid;          // this thread's key
  const bool live = kk <= p.t;
  float g = 0.f, s[kMaxR];
#pragma unroll
  for (int r = 0; r < kMaxR; ++r) s[r] = 0.f;
  if (live) {
    // the thread's key row, 16 bytes at a time (head_dim is a multiple of 16 bytes: checked by the host)
    constexpr int kN = aux::Vec16<T>::kN;
    const T* krow = kc + (size_t)kk * D;
    for (int e0 = 0; e0 < D; e0 += kN) {
      float kv[kN];
      aux::Vec16<T>::load(krow + e0, kv);
#pragma unroll
      for (int u = 0; u < kN; ++u) {
        g = fmaf(kv[u], s_kt[e0 + u], g);
#pragma unroll
        for (int r = 0; r < kMaxR; ++r)
          if (r < R) s[r] = fmaf(kv[u], s_q[r * D + e0 + u], s[r]);
      }
    }
  }
  // decay state of this key after row t
  float cstate = 0.f;
  if (live && kk < p.t) {
    const float s3 = cbrtf(Num<TG>::ld(static_cast<const TG*>(p.src) + (size_t)bh * p.Lcap + kk));
    const float t3 = cbrtf(Num<TG>::ld(static_cast<const TG*>(p.dest) + bh));
    const float pw = g > 0.f ? powf(g, 2.0f / 3.0f) : 0.f;
    const float a = pw * s3 * t3;
    cstate = p.state[(size_t)bh * p.Lcap + kk] + log1pf(-fminf(fmaxf(a, 0.f), clamp_hi()));
  }
  if (live) p.state[(size_t)bh * p.Lcap + kk] = cstate;

  // softmax over the chunk's keys, per head: block-wide max and sum through warp shuffles and shared memory
  const int warp = tid >> 5, lane = tid & 31, nwarps = (C + 31) >> 5;
  float m[kMaxR];
#pragma unroll
  for (int r = 0; r < kMaxR; ++r) {
    float v = (live && r < R) ? s[r] + cstate : -INFINITY;
    s[r] = v;
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) s_red[r * 32 + warp] = v;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kMaxR; ++r) {
    float v = -INFINITY;
    for (int w = 0; w < nwarps; ++w) v = fmaxf(v, s_red[r * 32 + w]);
    m[r] = v;
  }
#pragma unroll
  for (int r = 0; r < kMaxR; ++r) {
    const float e = (live && r < R) ? __expf(s[r] - m[r]) : 0.f;
    s[r] = e;
    float v = e;
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) s_red[(kMaxR + r) * 32 + warp] = v;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kMaxR; ++r) {
    float v = 0.f;
    for (int w = 0; w < nwarps; ++w) v += s_red[(kMaxR + r) * 32 + w];
    // the reference rounds the normalised probabilities to the input dtype before the product with V (:159)
    if (r < R) {
      s_p[r * C + tid] = Num<T>::rnd(s[r] / v);
      if (tid == 0) p.lse[((size_t)bh * nt + i) * R + r] = m[r] + logf(v);
    }
  }
  __syncthreads();

  // out[r][d] = sum_k P[r][k] v_k[d]: thread = (d, r modulo), keys in the loop; V rows are read coalesced along d
  const int nkeys = min(C, p.t - i * C + 1);
  for (int o = tid; o < R * D; o += C) {
    const int r = o / D, d = o - r * D;
    float acc = 0.f;
    for (int k = 0; k < nkeys; ++k) acc = fmaf(s_p[r * C + k], Num<T>::ld(vc + (size_t)(i * C + k) * D + d), acc);
    Num<T>::st(static_cast<T*>(p.out) + (((size_t)bh * nt + i) * R + r) * D + d, acc);
  }
}

// ---- bf16, head_dim 64 / 128, chunks of 64 / 128 / 256 keys ----------------------------------------------------------
// Bound by the one read of the caches; what it needs is bytes in flight.  One block of 2 C threads per (b, h, chunk): every
// thread issues its 16-byte pieces of K AND of V (128 bytes of each at head_dim 128) before anything else, so that a
// resident block keeps its whole chunk (64 KB at C = 128, D = 128) on the way.  K goes to registers, V through cp.async to the
// thread's own places in shared memory (only the thread that fetched a piece reads it: no barrier), so that four such blocks fit
// an SM; with V in registers as well two did (97 -> 86 us below).
//   scores  mma.sync m16n8k16: the rows are 16 keys of a warp, the columns are the new row's key and its queries (1 + R <= 9:
//           one or two column tiles, the rest zero).  The contraction index is permuted so that a thread's A pieces are 16
//           contiguous bytes of a key row; no shuffles, exact bf16 products, fp32 sums.  (Eight columns are too few for tcgen05:
//           an instruction there is 128 keys x 16 columns at the least and wants its operands in shared memory first.)
//   state   thread = key.   softmax  warp = query head: shuffles only.
//   P V     thread = (8 columns of V, every 2C*8/D-th key), partial sums over the keys through shuffles and shared memory.
// Against the kernel above (one thread per key row, V one 2-byte element at a time): B16 H8 R4 D128 at t = 6150 (418 MB of
// caches) 332 -> 86 us = 4.9 TB/s; B1 H8 R4 D64 at t = 300 13.8 -> 3.7 us.
template <int D, int C, int RT>
struct StepCfg {
  static constexpr int kThreads = 2 * C, kWarps = kThreads / 32;
  static constexpr int kTPR = D / 8;                     // threads per row of V
  static constexpr int kGroups = kThreads / kTPR;        // rows of V per pass
  static constexpr int kVLoads = C / kGroups;
  static constexpr int kKLoads = D / 32;                 // 16-byte pieces of each of the two key rows of a thread
  static constexpr int kNT = RT == 8 ? 2 : 1;            // column tiles of the score product
  static constexpr int kSW = 8 * kNT + 1;                // row stride of the score tile (odd: thread = key reads a column)
  static constexpr int oS = 0, oC = oS + C * kSW, oP = (oC + C + 3) / 4 * 4, oAcc = oP + C * RT;
  // a thread's pieces of V, 16 bytes each and kThreads apart; the partial sums take their place once all have been read (so that
  // chunks of up to 128 keys stay within the 48 KB that need no opt-in)
  static constexpr int oV = oAcc, kAcc = kWarps * RT * D, kV = C * D / 2;
  static constexpr int kSmemFloats = oAcc + (kAcc > kV ? kAcc : kV);
};

template <int D, int C, int RT, typename TG>
__global__ void __launch_bounds__(2 * C) step_mma_kernel(Params p) {
  using Cfg = StepCfg<D, C, RT>;
  extern __shared__ __align__(16) float sm[];
  float *s_s = sm + Cfg::oS, *s_c = sm + Cfg::oC, *s_p = sm + Cfg::oP, *s_acc = sm + Cfg::oAcc;
  const int bh = blockIdx.x, i = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nt = p.t / C + 1, R = p.R;
  const int nkeys = min(C, p.t - i * C + 1);             // live keys of the chunk; what lies behind them in the caches is not read
  const __nv_bfloat16* kc = static_cast<const __nv_bfloat16*>(p.kcache) + (size_t)bh * p.Lcap * D;
  const __nv_bfloat16* vrow = static_cast<const __nv_bfloat16*>(p.vcache) + ((size_t)bh * p.Lcap + (size_t)i * C) * D;
  const uint4 zero = make_uint4(0, 0, 0, 0);

  // all reads of the caches first
  const int kr0 = warp * 16 + (lane >> 2), kr1 = kr0 + 8, c8 = (lane & 3) * 8;
  uint4 a0[Cfg::kKLoads], a1[Cfg::kKLoads], bq[Cfg::kNT][Cfg::kKLoads];
  const __nv_bfloat16* krow = kc + (size_t)i * C * D + c8;
#pragma unroll
  for (int x = 0; x < Cfg::kKLoads; ++x) {
    a0[x] = kr0 < nkeys ? __ldg(reinterpret_cast<const uint4*>(krow + (size_t)kr0 * D + x * 32)) : zero;
    a1[x] = kr1 < nkeys ? __ldg(reinterpret_cast<const uint4*>(krow + (size_t)kr1 * D + x * 32)) : zero;
  }
#pragma unroll
  for (int n = 0; n < Cfg::kNT; ++n) {
    const int col = n * 8 + (lane >> 2);                 // 0: the new key, 1 + r: query head r
    const __nv_bfloat16* row = col == 0 ? kc + (size_t)p.t * D : static_cast<const __nv_bfloat16*>(p.q) + ((size_t)bh * R + col - 1) * D;
#pragma unroll
    for (int x = 0; x < Cfg::kKLoads; ++x) bq[n][x] = col <= R ? __ldg(reinterpret_cast<const uint4*>(row + c8 + x * 32)) : zero;
  }
  const uint32_t my_v = (uint32_t)__cvta_generic_to_shared(sm + Cfg::oV) + tid * 16;
  const int vg = tid / Cfg::kTPR, vc8 = (tid % Cfg::kTPR) * 8;
#pragma unroll
  for (int x = 0; x < Cfg::kVLoads; ++x) {
    const int k = vg + x * Cfg::kGroups;
    // (a piece beyond the live keys is filled with zeros and not read)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(my_v + x * Cfg::kThreads * 16),
                 "l"(vrow + (size_t)(k < nkeys ? k : 0) * D + vc8), "r"(k < nkeys ? 16 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // (per-key values of the state update; a thread beyond the live keys reads nothing)
  const size_t key_at = (size_t)bh * p.Lcap + (size_t)i * C + tid;
  const bool updates = tid < nkeys && i * C + tid < p.t;
  float src = 0.f, dst = 0.f, old = 0.f;
  if (updates) {
    src = Num<TG>::ld(static_cast<const TG*>(p.src) + key_at);
    dst = Num<TG>::ld(static_cast<const TG*>(p.dest) + bh);
    old = p.state[key_at];
  }

#pragma unroll
  for (int n = 0; n < Cfg::kNT; ++n) {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    auto mma = [&](uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t y0, uint32_t y1) {
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(y0), "r"(y1));
    };
#pragma unroll
    for (int x = 0; x < Cfg::kKLoads; ++x) {
      mma(a0[x].x, a1[x].x, a0[x].y, a1[x].y, bq[n][x].x, bq[n][x].y);
      mma(a0[x].z, a1[x].z, a0[x].w, a1[x].w, bq[n][x].z, bq[n][x].w);
    }
    const int cc = n * 8 + (lane & 3) * 2;
    s_s[kr0 * Cfg::kSW + cc] = d[0]; s_s[kr0 * Cfg::kSW + cc + 1] = d[1];
    s_s[kr1 * Cfg::kSW + cc] = d[2]; s_s[kr1 * Cfg::kSW + cc + 1] = d[3];
  }
  __syncthreads();
  if (tid < C) {
    float cstate = 0.f;
    if (updates) {
      const float g = s_s[tid * Cfg::kSW];
      const float pw = g > 0.f ? powf(g, 2.0f / 3.0f) : 0.f;
      cstate = old + log1pf(-fminf(fmaxf(pw * cbrtf(src) * cbrtf(dst), 0.f), clamp_hi()));
    }
    if (tid < nkeys) p.state[key_at] = cstate;
    s_c[tid] = cstate;
  }
  __syncthreads();
  if (warp < RT) {
    // (a chunk of 64 keys has four warps: with eight heads a warp takes two)
    for (int r = warp; r < RT; r += Cfg::kWarps) {
      float e[C / 32], m = -INFINITY, z = 0.f;
#pragma unroll
      for (int x = 0; x < C / 32; ++x) {
        const int k = x * 32 + lane;
        e[x] = k < nkeys ? s_s[k * Cfg::kSW + 1 + r] + s_c[k] : -INFINITY;
        m = fmaxf(m, e[x]);
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
#pragma unroll
      for (int x = 0; x < C / 32; ++x) {
        e[x] = x * 32 + lane < nkeys ? __expf(e[x] - m) : 0.f;
        z += e[x];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
      // the reference rounds the normalised probabilities to the input dtype before the product with V (:159)
#pragma unroll
      for (int x = 0; x < C / 32; ++x) s_p[(x * 32 + lane) * RT + r] = Num<__nv_bfloat16>::rnd(e[x] / z);
      if (lane == 0 && r < R) p.lse[((size_t)bh * nt + i) * R + r] = m + logf(z);
    }
  }
  __syncthreads();

  float acc[RT][8];
#pragma unroll
  for (int r = 0; r < RT; ++r)
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[r][u] = 0.f;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int x = 0; x < Cfg::kVLoads; ++x) {
    const float* pk = s_p + (vg + x * Cfg::kGroups) * RT;
    const uint4 v = reinterpret_cast<const uint4*>(sm + Cfg::oV)[x * Cfg::kThreads + tid];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float pr[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) pr[r] = pk[r];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float lo = __uint_as_float(w[u] << 16), hi = __uint_as_float(w[u] & 0xffff0000u);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        acc[r][2 * u] = fmaf(pr[r], lo, acc[r][2 * u]);
        acc[r][2 * u + 1] = fmaf(pr[r], hi, acc[r][2 * u + 1]);
      }
    }
  }
  __syncthreads();      // (every thread has read its pieces of V)
#pragma unroll
  for (int r = 0; r < RT; ++r) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int o = Cfg::kTPR; o < 32; o <<= 1) acc[r][u] += __shfl_xor_sync(0xffffffffu, acc[r][u], o);
    if (lane < Cfg::kTPR) {
      float4* dst4 = reinterpret_cast<float4*>(s_acc + ((size_t)warp * RT + r) * D + vc8);
      dst4[0] = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      dst4[1] = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
    }
  }
  __syncthreads();
  for (int o = tid; o < R * D; o += Cfg::kThreads) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < Cfg::kWarps; ++w) sum += s_acc[w * RT * D + o];
    Num<__nv_bfloat16>::st(static_cast<__nv_bfloat16*>(p.out) + ((size_t)bh * nt + i) * R * D + o, sum);
  }
}

template <int D, int C, int RT, typename TG>
inline bool launch_step_mma(const Params& p, int nt, cudaStream_t st) {
  using Cfg = StepCfg<D, C, RT>;
  constexpr int smem = Cfg::kSmemFloats * 4;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(step_mma_kernel<D, C, RT, TG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return false;
  step_mma_kernel<D, C, RT, TG><<<dim3((unsigned)p.BH, (unsigned)nt), Cfg::kThreads, smem, st>>>(p);
  return true;
}
template <int D, int C, typename TG>
inline bool launch_step_mma_r(const Params& p, int nt, cudaStream_t st) {
  if (p.R == 1) return launch_step_mma<D, C, 1, TG>(p, nt, st);
  if (p.R == 2) return launch_step_mma<D, C, 2, TG>(p, nt, st);
  return p.R <= 4 ? launch_step_mma<D, C, 4, TG>(p, nt, st) : launch_step_mma<D, C, 8, TG>(p, nt, st);
}
template <int D, typename TG>
inline bool launch_step_mma_c(const Params& p, int nt, cudaStream_t st) {
  if (p.C == 64) return launch_step_mma_r<D, 64, TG>(p, nt, st);
  return p.C == 128 ? launch_step_mma_r<D, 128, TG>(p, nt, st) : launch_step_mma_r<D, 256, TG>(p, nt, st);
}
// What the kernel above takes: its tiles are whole 16-byte pieces of 64- or 128-wide bf16 rows, and chunks whose threads
// (two per key) make whole warps and at most 512 of them.  Everything else (fp32, other widths) runs on step_kernel.
inline bool step_mma_takes(const Params& p, bool bf16_in) {
  return bf16_in && (p.D == 64 || p.D == 128) && (p.C == 64 || p.C == 128 || p.C == 256) &&
         (reinterpret_cast<uintptr_t>(p.q) & 15u) == 0;
}

inline size_t smem_bytes(const Params& p) {
  return sizeof(float) * ((size_t)p.D + (size_t)p.R * p.D + (size_t)p.R * p.C + 2 * kMaxR * 32);
}

}  // namespace decode
}  // namespace ua
