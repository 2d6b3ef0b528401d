// Incremental (decode) step of the Universal Attention operator: ONE new row against cached keys and values.
//
// The operator's forward (universal_attention_autograd.py:9-38, row-chunked form :104-163) needs, for a new row t and
// every earlier key k, the decay prefix  C[k, t] = sum_{k < q <= t} log1p(-affinity(k, q)).  That prefix is a running
// sum per key, so a serving loop keeps it as state next to the key / value caches:
//     state[k] <- state[k] + log1p(-clamp(relu(k_k . k_t)^(2/3) src_k^(1/3) dest_t^(1/3)))     for k < t
//     state[t]  = 0
// and the new row's outputs are, per key chunk i of `chunk` keys (only the chunks that hold keys <= t exist),
//     lse[r][i] = logsumexp_k (k_k . q_r + state[k]),     out[r][i][:] = sum_k softmax_k(...) v_k
// exactly row t of the full forward.  O(t * d) work and cache reads per step: HBM-bound.  Three kernels:
//   step_mma_kernel   bf16, head_dim 128, chunks of 64 / 128 keys: blocks that stay and take one (b, h, chunk) after another
//   step_once_kernel  bf16, head_dim 64, and chunks of 256 keys: a block per (b, h, chunk), the whole chunk in flight at once
//   step_kernel       fp32, other head_dims and chunks, unaligned queries: a block per (b, h, chunk), thread = key, CUDA cores
// The first two form scores (the first P V as well) with mma.sync; eight columns are too few for tcgen05.
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

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

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

// ---- bf16, head_dim 128, chunks of 64 / 128 keys ---------------------------------------------------------------------
// Bound by the one read of the caches; what it needs is bytes in flight at all times.  Blocks of 2 C threads stay on their SM and take one
// (b, h, chunk) after another; K and V of a chunk are on their way through cp.async while the chunk before is worked on: the next K is asked for
// as soon as the scores of this one are formed, the next V as soon as P V is.
//   scores  mma.sync m16n8k16: the rows are 16 keys of a warp, the columns are the new row's key and its queries (1 + R <= 9:
//           one or two column tiles, the rest zero).  The contraction index is permuted so that a thread's A pieces are 16
//           contiguous bytes of a key row, which it fetches itself to places of its own: no shuffles, no barrier, exact bf16 products, fp32
//           sums.  (Eight columns are too few for tcgen05: an instruction there is 128 keys x 16 columns at the least.)
//   state   thread = key.   softmax  warp = query head: shuffles only.
//   P V     mma.sync as well: the rows are the query heads, a warp takes columns of V (ldmatrix from swizzled rows), all keys of the
//           chunk: no sums across warps.
// Against one block per chunk that issues its reads and then waits for them (P V on the CUDA cores, partial sums through shared memory):
// B16 H8 R4 D128 at t = 6150 (418 MB of caches) 86 -> 76 us = 5.5 TB/s, R1 81 -> 73, R8 142 -> 104, chunks of 64 keys 78 -> 70; with items in the
// order of the memory (chunks of a (b, h) one after the other) instead of 2 MB apart 82 -> 78 of it, with one cube root instead of a power and two 78 -> 76.
template <int D, int C, int RT>
struct StepCfg {
  static constexpr int kThreads = 2 * C, kWarps = kThreads / 32;
  static constexpr int kTPR = D / 8;                     // 16-byte pieces per row
  static constexpr int kGroups = kThreads / kTPR;        // rows of V per pass of the fetch
  static constexpr int kVLoads = C / kGroups;
  static constexpr int kKLoads = D / 32;                 // 16-byte pieces of each of the two key rows of a thread
  static constexpr int kNT = RT == 8 ? 2 : 1;            // column tiles of the score product
  static constexpr int kSW = 8 * kNT + 1;                // row stride of the score tile (odd: thread = key reads a column)
  static constexpr int kVT = D / 8 / kWarps;             // column tiles of P V per warp
  static_assert(kVT >= 1, "a column tile for every warp");
  static constexpr int kPW = C + 8;                      // row stride of P, in elements (conflict-free fragments)
  static constexpr int oK = 0, oV = oK + C * D * 2, oS = oV + C * D * 2, oC = oS + C * kSW * 4, oP = (oC + C * 4 + 15) / 16 * 16;
  static constexpr int kSmemBytes = oP + RT * kPW * 2;
  // blocks per SM: what shared memory holds (1 KB per block is the system's), within the threads of an SM at 80 registers each
  static constexpr int kBySmem = 233472 / (kSmemBytes + 1024), kByRegs = 65536 / (80 * kThreads);
  static constexpr int kBlocks = kBySmem < kByRegs ? kBySmem : kByRegs;
};

template <int D, int C, int RT, typename TG>
__global__ void __launch_bounds__(2 * C, StepCfg<D, C, RT>::kBlocks) step_mma_kernel(Params p, int items) {
  using Cfg = StepCfg<D, C, RT>;
  extern __shared__ __align__(16) uint8_t sm_step[];
  float *s_s = reinterpret_cast<float*>(sm_step + Cfg::oS), *s_c = reinterpret_cast<float*>(sm_step + Cfg::oC);
  __nv_bfloat16* s_p = reinterpret_cast<__nv_bfloat16*>(sm_step + Cfg::oP);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nt = p.t / C + 1, R = p.R;
  const __nv_bfloat16 *kcache = static_cast<const __nv_bfloat16*>(p.kcache), *vcache = static_cast<const __nv_bfloat16*>(p.vcache);
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const int kr0 = warp * 16 + (lane >> 2), kr1 = kr0 + 8, c8 = (lane & 3) * 8;
  const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(sm_step), my_k = s0 + Cfg::oK + tid * 16;
  const int vg = tid / Cfg::kTPR, vc = tid % Cfg::kTPR;
  auto live_keys = [&](int i) { return min(C, p.t - i * C + 1); };      // what lies behind them in the caches is not read
  auto cp16 = [&](uint32_t dst, const void* src, bool live) {           // (a piece beyond the live keys is filled with zeros)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
  };
  auto fetch_k = [&](int item) {
    if (item < items) {
      const int bh = item / nt, i = item % nt, nkeys = live_keys(i);
      const __nv_bfloat16* row = kcache + ((size_t)bh * p.Lcap + (size_t)i * C) * D + c8;
#pragma unroll
      for (int x = 0; x < Cfg::kKLoads; ++x) {
        cp16(my_k + 2 * x * Cfg::kThreads * 16, row + (size_t)(kr0 < nkeys ? kr0 : 0) * D + x * 32, kr0 < nkeys);
        cp16(my_k + (2 * x + 1) * Cfg::kThreads * 16, row + (size_t)(kr1 < nkeys ? kr1 : 0) * D + x * 32, kr1 < nkeys);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto fetch_v = [&](int item) {
    if (item < items) {
      const int bh = item / nt, i = item % nt, nkeys = live_keys(i);
      const __nv_bfloat16* row = vcache + ((size_t)bh * p.Lcap + (size_t)i * C) * D + vc * 8;
#pragma unroll
      for (int x = 0; x < Cfg::kVLoads; ++x) {
        const int k = vg + x * Cfg::kGroups;
        cp16(s0 + Cfg::oV + k * D * 2 + (vc ^ (k & 7)) * 16, row + (size_t)(k < nkeys ? k : 0) * D, k < nkeys);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint4 bq[Cfg::kNT][Cfg::kKLoads];      // the new key and the queries, as columns of the score product
  auto fetch_q = [&](int bh) {
#pragma unroll
    for (int n = 0; n < Cfg::kNT; ++n) {
      const int col = n * 8 + (lane >> 2);                 // 0: the new key, 1 + r: query head r
      const __nv_bfloat16* row = col == 0 ? kcache + ((size_t)bh * p.Lcap + p.t) * D : static_cast<const __nv_bfloat16*>(p.q) + ((size_t)bh * R + col - 1) * D;
#pragma unroll
      for (int x = 0; x < Cfg::kKLoads; ++x) bq[n][x] = col <= R ? __ldg(reinterpret_cast<const uint4*>(row + c8 + x * 32)) : zero;
    }
  };
  // (per-key values of the state update; a thread beyond the live keys reads nothing)
  float src = 0.f, dst = 0.f, old = 0.f;
  auto fetch_state = [&](int bh, int i) {
    if (tid < live_keys(i) && i * C + tid < p.t) {
      const size_t at = (size_t)bh * p.Lcap + (size_t)i * C + tid;
      src = Num<TG>::ld(static_cast<const TG*>(p.src) + at);
      dst = Num<TG>::ld(static_cast<const TG*>(p.dest) + bh);
      old = p.state[at];
    }
  };

  int item = blockIdx.x;
  fetch_k(item);
  fetch_v(item);
  fetch_q(item / nt);
  fetch_state(item / nt, item % nt);
  for (; item < items; item += gridDim.x) {
    const int bh = item / nt, i = item % nt, nkeys = live_keys(i), next = item + gridDim.x;
    asm volatile("cp.async.wait_group 1;" ::: "memory");      // K (V of the chunk may be on its way)
    uint4 a0[Cfg::kKLoads], a1[Cfg::kKLoads];
#pragma unroll
    for (int x = 0; x < Cfg::kKLoads; ++x) {
      a0[x] = *reinterpret_cast<const uint4*>(sm_step + Cfg::oK + (2 * x * Cfg::kThreads + tid) * 16);
      a1[x] = *reinterpret_cast<const uint4*>(sm_step + Cfg::oK + ((2 * x + 1) * Cfg::kThreads + tid) * 16);
    }
#pragma unroll
    for (int n = 0; n < Cfg::kNT; ++n) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int x = 0; x < Cfg::kKLoads; ++x) {
        mma_16816(d, a0[x].x, a1[x].x, a0[x].y, a1[x].y, bq[n][x].x, bq[n][x].y);
        mma_16816(d, a0[x].z, a1[x].z, a0[x].w, a1[x].w, bq[n][x].z, bq[n][x].w);
      }
      const int cc = n * 8 + (lane & 3) * 2;
      s_s[kr0 * Cfg::kSW + cc] = d[0]; s_s[kr0 * Cfg::kSW + cc + 1] = d[1];
      s_s[kr1 * Cfg::kSW + cc] = d[2]; s_s[kr1 * Cfg::kSW + cc + 1] = d[3];
    }
    fetch_k(next);                       // (over pieces that only this thread reads, and has read)
    if (next < items && next / nt != bh) fetch_q(next / nt);
    __syncthreads();
    if (tid < C) {
      float cstate = 0.f;
      if (tid < nkeys && i * C + tid < p.t) {
        const float g = s_s[tid * Cfg::kSW];
        // relu(g)^(2/3) src^(1/3) dest^(1/3) as one cube root.  Each gate (at most 1) brings its own factor g down before the two meet: g * g
        // of long keys leaves fp32, src * dst of closed gates falls below it, and infinity times zero is no affinity
        const float a = g > 0.f ? cbrtf((g * src) * (g * dst)) : 0.f;
        cstate = old + log1pf(-fminf(fmaxf(a, 0.f), clamp_hi()));
      }
      if (tid < nkeys) p.state[(size_t)bh * p.Lcap + (size_t)i * C + tid] = cstate;
      s_c[tid] = cstate;
    }
    if (next < items) fetch_state(next / nt, next % nt);
    __syncthreads();
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
      for (int x = 0; x < C / 32; ++x) s_p[r * Cfg::kPW + x * 32 + lane] = __float2bfloat16_rn(e[x] / z);
      if (lane == 0 && r < R) p.lse[((size_t)bh * nt + i) * R + r] = m + logf(z);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");      // V (the next K may be on its way)
    __syncthreads();
    {
      float acc[Cfg::kVT][4];
#pragma unroll
      for (int n = 0; n < Cfg::kVT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
      const int head = lane >> 2;
      const uint32_t* prow = reinterpret_cast<const uint32_t*>(s_p + head * Cfg::kPW) + (lane & 3);
#pragma unroll 4
      for (int k = 0; k < C; k += 16) {
        const uint32_t x0 = head < RT ? prow[k / 2] : 0u, x2 = head < RT ? prow[k / 2 + 4] : 0u;      // (rows 8..15 of the tile: none)
        const int krow = k + (lane & 15);
#pragma unroll
        for (int n = 0; n < Cfg::kVT; ++n) {
          uint32_t y0, y1;
          asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(y0), "=r"(y1)
                       : "r"(s0 + Cfg::oV + krow * D * 2 + ((warp * Cfg::kVT + n) ^ (krow & 7)) * 16));
          mma_16816(acc[n], x0, 0u, x2, 0u, y0, y1);
        }
      }
      if (head < R) {
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + (((size_t)bh * nt + i) * R + head) * D + warp * Cfg::kVT * 8 + (lane & 3) * 2;
#pragma unroll
        for (int n = 0; n < Cfg::kVT; ++n) {
          Num<__nv_bfloat16>::st(out + n * 8, acc[n][0]);
          Num<__nv_bfloat16>::st(out + n * 8 + 1, acc[n][1]);
        }
      }
    }
    if (next < items) __syncthreads();      // V, the scores and P have been read
    fetch_v(next);
  }
}

// ---- the same with one block per (b, h, chunk) ---------------------------------------------------------------------
// For head_dim 64 and for chunks of 256 keys (see launch_step_mma): every thread issues its 16-byte pieces of K AND of V before anything else, so
// that a resident block keeps its whole chunk on the way; K goes to registers, V through cp.async to the thread's own places in shared
// memory (only the thread that fetched a piece reads it: no barrier).  Scores and state as above; P V on the CUDA cores: thread = (8 columns
// of V, every 2C*8/D-th key), partial sums over the keys through shuffles and shared memory.
// At head_dim 128 the blocks follow the memory (chunks of a (b, h) one after the other: C256 R4 109 -> 104 us, R2 93 -> 88); at 64 the (b, h)s of a
// chunk do (the other way 59.7 -> 61.6 at B8 H16 R2 t8000, 30.8 -> 28.7 at B16 H4 R1 t7000).
template <int D, int C, int RT>
struct OnceCfg {
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
__global__ void __launch_bounds__(2 * C) step_once_kernel(Params p) {
  using Cfg = OnceCfg<D, C, RT>;
  extern __shared__ __align__(16) float sm[];
  float *s_s = sm + Cfg::oS, *s_c = sm + Cfg::oC, *s_p = sm + Cfg::oP, *s_acc = sm + Cfg::oAcc;
  const int nt = p.t / C + 1, R = p.R;
  const int bh = D == 64 ? blockIdx.x % p.BH : blockIdx.x / nt, i = D == 64 ? blockIdx.x / p.BH : blockIdx.x % nt;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
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
#pragma unroll
    for (int x = 0; x < Cfg::kKLoads; ++x) {
      mma_16816(d, a0[x].x, a1[x].x, a0[x].y, a1[x].y, bq[n][x].x, bq[n][x].y);
      mma_16816(d, a0[x].z, a1[x].z, a0[x].w, a1[x].w, bq[n][x].z, bq[n][x].w);
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
inline bool launch_step_once(const Params& p, int nt, cudaStream_t st) {
  using Cfg = OnceCfg<D, C, RT>;
  constexpr int smem = Cfg::kSmemFloats * 4;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(step_once_kernel<D, C, RT, TG>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return false;
  step_once_kernel<D, C, RT, TG><<<(unsigned)(p.BH * nt), Cfg::kThreads, smem, st>>>(p);
  return true;
}
template <int D, int C, int RT, typename TG>
inline bool launch_step_mma(const Params& p, int nt, cudaStream_t st) {
  // Blocks that stay pay where a chunk is long enough to hide their work and several of them fit an SM.  At t = 6150, B16 H8, staying / one
  // chunk per block in us: D128 C128 R1 73 / 80, R4 76 / 86, R8 104 / 142, C64 R4 70 / 78; but C256 R2 117 / 93, R4 118 / 109 (one block of
  // 150 KB per SM), and D64 R2 58 / 47 (half the bytes for the same chain of scores, softmax and P V).
  // With fewer chunks than resident blocks no block takes a second one, and the form is still the shorter chain (P V without sums across
  // warps).  B1 H8, GPU time per step at t = 300 / 1000 / 3000, staying / one chunk per block: C128 R1 4.0 / 4.4 / 6.1, 5.0 / 5.2 / 6.3; R4 4.4 / 4.5 / 6.3,
  // 5.0 / 5.0 / 6.7; R8 4.8 / 4.8 / 6.9, 6.1 / 6.2 / 9.1; C64 R1 3.7 / 4.0 / 5.5, 4.9 / 5.1 / 6.0; R4 3.7 / 4.1 / 5.6, 4.4 / 4.6 / 6.3.  Chunks of 128 keys then
  // need the opt-in to more than 48 KB, a driver call of 0.08 us per step (remembering it per context saves half of that).
  if constexpr (D == 64 || C == 256) {
    return launch_step_once<D, C, RT, TG>(p, nt, st);
  } else {
    using Cfg = StepCfg<D, C, RT>;
    if (Cfg::kSmemBytes > 48 * 1024 &&
        cudaFuncSetAttribute(step_mma_kernel<D, C, RT, TG>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess)
      return false;
    const int items = p.BH * nt, grid = items < kSms * Cfg::kBlocks ? items : kSms * Cfg::kBlocks;
    step_mma_kernel<D, C, RT, TG><<<(unsigned)grid, Cfg::kThreads, Cfg::kSmemBytes, st>>>(p, items);
    return true;
  }
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
// What the two mma.sync kernels take between them: tiles of whole 16-byte pieces of 64- or 128-wide bf16 rows, chunks whose threads
// (two per key) are 512 at the most.  Everything else (fp32, other widths) runs on step_kernel.
inline bool step_mma_takes(const Params& p, bool bf16_in) {
  return bf16_in && (p.D == 64 || p.D == 128) && (p.C == 64 || p.C == 128 || p.C == 256) &&
         (reinterpret_cast<uintptr_t>(p.q) & 15u) == 0;
}

inline size_t smem_bytes(const Params& p) {
  return sizeof(float) * ((size_t)p.D + (size_t)p.R * p.D + (size_t)p.R * p.C + 2 * kMaxR * 32);
}

}  // namespace decode
}  // namespace ua
