// Tensor-core forward of the Universal Attention operator for sm_100a.
//
// bf16 inputs, key chunk kC = 128 or 64, head_dim D in {64, 128}.  One thread block owns
// one key chunk (b, h, i) and sweeps the 128-row tiles from the chunk's first row to the
// end of the sequence upwards, so the per-key decay prefix is carried in registers.  Where
// that leaves the chip idle (fewer blocks than SMs, or one long sweep among short ones) the
// sweep of a chunk is cut into segments of p.seg tiles, one block each: tile_totals_kernel
// first sums the log-retention of every (chunk, tile), and a segment starts from the sum of
// the tiles before it (see ua_split.h for when).
//
// kC = 64: tiles start at the chunk's own first row (so only the first one has masked
// pairs; the last may be half a tile); the 64 keys are TMEM lanes 0..63 of G and columns
// 0..63 of S, lanes 64..127 of G hold the next chunk's keys and are not looked at.
//
//   G    = K_i  K_j^T    tcgen05.mma  M = keys, N = rows   (keys on TMEM lanes)
//   S_r  = Q_rj K_i^T    tcgen05.mma  M = rows, N = keys   (rows on TMEM lanes)
//   O_r  = P_r  V_i      tcgen05.mma  A = P (bf16, TMEM), B = V_i (MN-major smem)
//
// Warp roles (512 threads):
//   warp 0      TMA producer: K_i, V_i once; K_j and Q_rj tiles through mbarrier rings
//   warp 1      MMA issuer (one elected thread issues every tcgen05.mma / commit)
//   warps 4-7   decay group: thread = key.  Reads G from TMEM, computes the
//               log-retention, scans it along the rows in registers (carry kept
//               across tiles), writes the prefix C^T[row][key] to shared memory.
//   warps 8-15  two softmax groups alternating over (tile, r): thread = row.
//               S + C, row max / sum in registers (no shuffles), P -> TMEM as
//               bf16, then the epilogue O / l -> out and m + log l -> lse.
//
// The two reductions of the operator run along perpendicular axes of the tile
// (scan along rows per key, softmax along keys per row); putting keys on lanes
// for G and rows on lanes for S makes both of them thread-local, at the price
// of one 64 KB shared-memory transpose of C per tile, shared by the R heads.
//
// Every mbarrier wait is bounded; on a timeout the block raises a shared abort
// flag, every role leaves its loop, TMEM is freed and status[0] is set.
#pragma once
#include <type_traits>
#include "ua_common.cuh"
#include "ua_ptx.cuh"

namespace ua {
namespace sm100 {

using namespace ua::ptx;

struct FwdParams {
  Shape s;
  const void* ssrc;
  const void* sdest;
  const void* vc;        // values, for the masked-row fill
  __nv_bfloat16* out;    // chunk-major (b,h,n,r,L,d); null: only lse / denom are produced
  float* lse;            // (b,h,n,r,L)
  __nv_bfloat16* denom;  // (b,h,n,r,L) or null
  int* status;           // device word: 0 = ok, otherwise a role-specific timeout code
  int fill_masked;       // write the rows before the key chunk (uniform softmax) from the two otherwise idle warps
  // Row range (sequence sharding): this call computes row tiles [j_begin, j_end) only.  xq, static_dest, out,
  // lse and denom then hold just those Lr = (j_end - j_begin) * 128 rows; keys, values and static_src are whole.
  int j_begin, j_end, Lr;  // Lr: rows per (chunk, head) slab of the row-indexed tensors
  int r0;                  // row of the slab where the range starts (several ranges can share one slab)
  const float* carry_in;   // optional (b*h*n, 128): decay prefix of key k at its first row tile of the range
  float* total_out;        // optional (b*h*n, 128): decay prefix after the last row tile of the range
  float* carry;          // optional: (b*h*n, L / 64, 128) decay prefix of key k at the start of every 64 rows
  // segments (whole sequence only): row tiles per block, 0 = a block sweeps its whole chunk; with segments, tile_totals
  // (b*h*n, tiles, 128) holds every key's log-retention sum over every row tile of its chunk's sweep
  int seg, tiles;
  const float* tile_totals;
  // merged-output mode (fwd_kernel<..., kMerge = true>): instead of writing `out`, every (chunk, row tile, head) adds its
  // share of the row's softmax over ALL keys, exp(m - row_lse) * (P~ V) with P~ = exp(s - m) unnormalised, to merged_acc
  float* merged_acc;     // (b,h,r,L,d) fp32, zeroed by the caller
  const float* row_lse;  // (b,h,r,L) fp32: log-sum-exp of every row over all key chunks (from a statistics-only run)
};

// Gated affinity and log-retention of one (key, row) pair from the Gram value
// (universal_attention_autograd.py:148-150), with hardware ex2/lg2.  Shared by
// the forward, the carry pre-pass and the backward so that recomputation is
// bit-identical.
__device__ __forceinline__ float gram_pow23(float gv) { return gv > 0.f ? ex2(lg2(gv) * (2.0f / 3.0f)) : 0.f; }
__device__ __forceinline__ float gated_affinity(float pw, float s3, float t3) { return pw * s3 * t3; }
__device__ __forceinline__ float log_retention(float a) {
  return lg2(1.0f - fminf(a, clamp_hi())) * 0.6931471805599453f;
}

// packed fp32 pairs (one instruction for two lanes of work: the element-wise phases are bound by instruction issue)
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return d;
}

// What the softmax groups produce: the per-chunk output tiles (and log-sum-exp), the merged-output contribution, or the
// log-sum-exp alone (then no probabilities are written, no PV product is issued, nothing is drained).
enum FwdOut { kOutTiles = 0, kOutMerged = 1, kOutStats = 2 };

// three-input maximum (one instruction on sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int D>
struct FwdCfg {
  static constexpr int kTileBytes = 128 * D * 2;   // one [128][D] bf16 tile
  static constexpr int kBoxBytes = 128 * 128;      // one TMA box: 128 rows x 64 elements
  static constexpr int kBoxes = D / 64;
  static constexpr bool kOneSlot = (D == 128);      // K_j and Q tiles share one slot
  static constexpr int kKjStages = kOneSlot ? 0 : 2;
  static constexpr int kQStages = kOneSlot ? 1 : 2;
  static constexpr int kOBufs = (D == 64) ? 2 : 1;
  static constexpr int oKi = 0;
  static constexpr int oVi = oKi + kTileBytes;
  static constexpr int oKj = oVi + kTileBytes;
  static constexpr int oQ = oKj + kKjStages * kTileBytes;
  // The decay prefix crosses from keys-on-lanes to rows-on-lanes through 64 KB fp32 tiles C^T[row][key]; with two of them the decay
  // group is a tile ahead of the softmax groups.  At head_dim 128 that leaves shared memory for ONE 32 KB slot, which K_j and Q
  // tiles pass through in the order of their products (each is read for 0.3 us, and the next one is needed 2 us later); with two
  // slots for Q, one for K_j and a single C^T tile the groups took turns: B1 H8 R4 L8192 D128 1523 -> 1312 us.
  static constexpr int kCBufs = 2;
  static constexpr int oCs = oQ + kQStages * kTileBytes;
  static constexpr int oT3 = oCs + kCBufs * 65536;
  static constexpr int oBar = oT3 + 1024;
  static constexpr int oMisc = oBar + 256;
  static constexpr int oFill = oMisc + 64;                // bf16[D]: value of a fully masked output row
  static constexpr int kSmemBytes = oFill + 256 + 1024;  // + slack to align the base to 1024 B
  static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");
  static constexpr uint32_t tG = 0, tS0 = 128, tS1 = 256, tO0 = 384, tO1 = 384 + D;
};

enum FwdBar {
  // (kCReady / kCFree: one barrier per C^T buffer, so that no waiter can fall two phases behind on a shared one)
  kKvFull = 0, kKjFull = 1, kKjEmpty = 3, kQFull = 5, kQEmpty = 7, kGFull = 9, kGFree = 10, kCReady = 11, kCFree = 13,
  kSFull = 15, kPReady = 17, kOFull = 19, kOFree = 21, kT3Ready = 23, kNumBars = 24
};

template <int D>
struct FwdCtx {
  uint8_t* smem;
  uint32_t bars;      // shared address of barrier 0
  uint32_t tmem;
  volatile int* abort_flag;
  int i, bh, ntiles;
  int row0, srow0;    // first row of the block's first tile: in the sequence, and inside the slabs of row-indexed tensors
  int t0;             // number of that tile in the chunk's sweep (0 unless the sweep is cut into segments)
  __device__ __forceinline__ uint32_t bar(int idx) const { return bars + 8u * idx; }
  __device__ __forceinline__ bool wait(int idx, uint32_t parity) const { return mbar_wait(bar(idx), parity & 1u, abort_flag); }
  // warp-collective forms for the decay and softmax groups
  __device__ __forceinline__ bool wait_w(int idx, uint32_t parity) const { return mbar_wait_warp(bar(idx), parity & 1u, abort_flag); }
  __device__ __forceinline__ void arrive_w(int idx) const { mbar_arrive_warp(bar(idx)); }
};

// ------------------------------------------------------------------ producer --
template <int D, int kC, bool kCarryOnly>
__device__ __forceinline__ void fwd_producer(const FwdCtx<D>& c, const FwdParams& p, const CUtensorMap* tmK,
                                             const CUtensorMap* tmV, const CUtensorMap* tmQ) {
  using Cfg = FwdCfg<D>;
  const int L = p.s.L, R = p.s.R;
  const uint32_t sbase = smem_u32(c.smem);
  const int krow = c.bh * L + c.i * kC;
  mbar_expect_tx(c.bar(kKvFull), (kCarryOnly ? 1 : 2) * Cfg::kTileBytes);
  for (int b = 0; b < Cfg::kBoxes; ++b) {
    tma_load_2d(sbase + Cfg::oKi + b * Cfg::kBoxBytes, tmK, b * 64, krow, c.bar(kKvFull));
    if (!kCarryOnly) tma_load_2d(sbase + Cfg::oVi + b * Cfg::kBoxBytes, tmV, b * 64, krow, c.bar(kKvFull));
  }
  int use = 0;                          // of the one slot (head_dim 128)
  auto load_slot = [&](const CUtensorMap* tm, int y) -> bool {
    if (use >= 1 && !c.wait(kQEmpty, use - 1)) return false;
    mbar_expect_tx(c.bar(kQFull), Cfg::kTileBytes);
    for (int b = 0; b < Cfg::kBoxes; ++b) tma_load_2d(sbase + Cfg::oQ + b * Cfg::kBoxBytes, tm, b * 64, y, c.bar(kQFull));
    ++use;
    return true;
  };
  auto load_kj = [&](int T) -> bool {
    if constexpr (Cfg::kOneSlot) return load_slot(tmK, c.bh * L + c.row0 + T * 128);
    const int ks = T & 1, u = T >> 1;
    if (u >= 1 && !c.wait(kKjEmpty + ks, u - 1)) return false;
    mbar_expect_tx(c.bar(kKjFull + ks), Cfg::kTileBytes);
    for (int b = 0; b < Cfg::kBoxes; ++b)
      tma_load_2d(sbase + Cfg::oKj + ks * Cfg::kTileBytes + b * Cfg::kBoxBytes, tmK, b * 64, c.bh * L + c.row0 + T * 128,
                  c.bar(kKjFull + ks));
    return true;
  };
  if (!load_kj(0)) return;
  if (kCarryOnly) {
    for (int T = 1; T < c.ntiles; ++T)
      if (!load_kj(T)) return;
    return;
  }
  int t = 0;
  for (int T = 0; T < c.ntiles; ++T) {
    for (int r = 0; r < R; ++r, ++t) {
      if constexpr (Cfg::kOneSlot) {
        if (!load_slot(tmQ, (c.bh * R + r) * p.Lr + c.srow0 + T * 128)) return;
        if (r == 0 && T + 1 < c.ntiles && !load_kj(T + 1)) return;
        continue;
      }
      const int qs = t & 1, u = t >> 1;
      if (u >= 1 && !c.wait(kQEmpty + qs, u - 1)) return;
      mbar_expect_tx(c.bar(kQFull + qs), Cfg::kTileBytes);
      for (int b = 0; b < Cfg::kBoxes; ++b)
        tma_load_2d(sbase + Cfg::oQ + qs * Cfg::kTileBytes + b * Cfg::kBoxBytes, tmQ, b * 64,
                    (c.bh * R + r) * p.Lr + c.srow0 + T * 128, c.bar(kQFull + qs));
      if (r == 0 && T + 1 < c.ntiles && !load_kj(T + 1)) return;
    }
  }
}

// ---------------------------------------------------------------- MMA issuer --
template <int D, int kC, bool kCarryOnly, int kOut>
__device__ __forceinline__ void fwd_mma(const FwdCtx<D>& c, const FwdParams& p) {
  using Cfg = FwdCfg<D>;
  const int R = p.s.R;
  const uint32_t sbase = smem_u32(c.smem);
  constexpr uint32_t idesc_g = idesc_bf16(128, 128, 0, 0), idesc_s = idesc_bf16(128, kC, 0, 0);
  constexpr uint32_t idesc_pv = idesc_bf16(128, D, 0, 1);
  const uint32_t tS[2] = {c.tmem + Cfg::tS0, c.tmem + Cfg::tS1};
  const uint32_t tO[2] = {c.tmem + Cfg::tO0, c.tmem + (Cfg::kOBufs == 2 ? Cfg::tO1 : Cfg::tO0)};

  // D[128 x 128] = A[128][D] * B[128][D]^T, both K-major.  Operands are passed as descriptor low words
  // (built once: shared-memory addresses never change); a k-step of 16 elements is +32 B (>>4 = 2), the
  // second 64-element box of a tile +16384 B (>>4 = 1024).
  auto issue_kmajor = [&](uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
    mma_ss_c<false>(d_tmem, desc_from_lo(a_lo), desc_from_lo(b_lo), idesc);
#pragma unroll
    for (int ks = 1; ks < D / 16; ++ks) {
      const uint32_t off = (ks >> 2) * 1024 + (ks & 3) * 2;
      mma_ss_c<true>(d_tmem, desc_from_lo(a_lo + off), desc_from_lo(b_lo + off), idesc);
    }
  };
  const uint32_t kKi = desc_lo(sbase + Cfg::oKi, 16);
  const uint32_t mVi = desc_lo(sbase + Cfg::oVi, Cfg::kBoxBytes);
  int use = 0;                          // of the one slot (head_dim 128)
  auto issue_g = [&](int T) -> bool {
    const int ks = T & 1, u = T >> 1;
    if (Cfg::kOneSlot ? !c.wait(kQFull, use++) : !c.wait(kKjFull + ks, u)) return false;
    if (T >= 1 && !c.wait(kGFree, T - 1)) return false;
    tc_fence_after();
    issue_kmajor(c.tmem + Cfg::tG, kKi, desc_lo(sbase + (Cfg::kOneSlot ? Cfg::oQ : Cfg::oKj + ks * Cfg::kTileBytes), 16), idesc_g);
    tc_commit(c.bar(kGFull));
    tc_commit(c.bar(Cfg::kOneSlot ? kQEmpty : kKjEmpty + ks));
    return true;
  };
  auto issue_pv = [&](int tt) -> bool {
    const int sb = tt & 1, ob = tt % Cfg::kOBufs;
    if (!c.wait(kPReady + sb, tt >> 1)) return false;       // (statistics only: the group is done with the S buffer)
    if (kOut == kOutStats) return true;
    // the O buffer must have been drained by the epilogue that used it last
    // (barriers are per softmax group so that each waiter sees consecutive phases)
    if (Cfg::kOBufs == 2) {
      if (tt >= 2 && !c.wait(kOFree + sb, (tt >> 1) - 1)) return false;
    } else {
      if (tt >= 1 && !c.wait(kOFree + ((tt - 1) & 1), (tt - 1) >> 1)) return false;
    }
    tc_fence_after();
    mma_ts_c<false>(tO[ob], tS[sb], desc_from_lo(mVi), idesc_pv);
#pragma unroll
    for (int ks = 1; ks < kC / 16; ++ks) mma_ts_c<true>(tO[ob], tS[sb] + ks * 8, desc_from_lo(mVi + ks * 128), idesc_pv);
    tc_commit(c.bar(kOFull + sb));
    return true;
  };

  if (!c.wait(kKvFull, 0)) return;
  if (!issue_g(0)) return;
  if (kCarryOnly) {
    for (int T = 1; T < c.ntiles; ++T)
      if (!issue_g(T)) return;
    return;
  }
  int t = 0;
  for (int T = 0; T < c.ntiles; ++T) {
    for (int r = 0; r < R; ++r, ++t) {
      const int qs = Cfg::kOneSlot ? 0 : t & 1;
      if (!c.wait(kQFull + qs, Cfg::kOneSlot ? use++ : t >> 1)) return;
      tc_fence_after();
      issue_kmajor(tS[t & 1], desc_lo(sbase + Cfg::oQ + qs * Cfg::kTileBytes, 16), kKi, idesc_s);
      tc_commit(c.bar(kSFull + (t & 1)));
      tc_commit(c.bar(kQEmpty + qs));
      if (t >= 1 && !issue_pv(t - 1)) return;
      if (r == 0 && T + 1 < c.ntiles && !issue_g(T + 1)) return;
    }
  }
  if (t >= 1) issue_pv(t - 1);
}

// --------------------------------------------------------------- decay group --
template <int D, int kC, typename TG, bool kCarryOnly>
__device__ __forceinline__ void fwd_decay(const FwdCtx<D>& c, const FwdParams& p) {
  using Cfg = FwdCfg<D>;
  const int L = p.s.L;
  const int k = threadIdx.x & 127;
  const uint32_t lane_base = (uint32_t)((threadIdx.x >> 5) & 3) * 32u << 16;
  const TG* ss = static_cast<const TG*>(p.ssrc) + (size_t)c.bh * L;
  const TG* sd = static_cast<const TG*>(p.sdest) + (size_t)c.bh * p.Lr + c.srow0 + k;
  // (gate of row k of tile T; with chunks of 64 keys the last tile may reach beyond the sequence)
  auto gate_at = [&](int T) -> float { return (kC == 128 || c.row0 + T * 128 + k < L) ? Num<TG>::ld(sd + T * 128) : 0.f; };
  const bool live = k < kC;              // kC = 64: warps 6-7 hold no key and only fetch gates
  const float s3 = live ? cbrtf(Num<TG>::ld(ss + c.i * kC + k)) : 0.f;
  float raw_next = gate_at(0);           // the gate value of the next tile is fetched one pass ahead: its latency hides behind the pass
  float* sT3 = reinterpret_cast<float*>(c.smem + Cfg::oT3);
  uint8_t* sCs = c.smem + Cfg::oCs;
  const size_t chunk_id = (size_t)c.bh * p.s.N + c.i, key_id = chunk_id * 128 + k;
  // The prefix carried from tile to tile reaches -2e4 at L = 4096, where fp32 spacing is 2e-3: it is kept as an
  // unevaluated sum carry + carry_lo (the rounding error of every tile's addition is carried along), so that what a
  // row sees is one rounding away from the exact sum however many tiles came before it.
  float carry = p.carry_in ? p.carry_in[key_id] : 0.f, carry_lo = 0.f;
  auto add_to_carry = [&](float tile) {      // carry + (carry_lo + tile) as an exact two-term sum
    const float sum = carry + tile, bb = sum - carry;
    carry_lo = (carry - (sum - bb)) + (tile - bb);
    carry = sum;
  };
  if (live)
    for (int T = 0; T < c.t0; ++T) add_to_carry(carry_lo + p.tile_totals[(chunk_id * p.tiles + T) * 128 + k]);
  for (int T = 0; T < c.ntiles; ++T) {
    float* t3buf = sT3 + (T & 1) * 128;
    t3buf[k] = cbrtf(raw_next);
    if (T + 1 < c.ntiles) raw_next = gate_at(T + 1);
    c.arrive_w(kT3Ready);
    if (!c.wait_w(kT3Ready, T)) return;
    if (!live) continue;
    if (!c.wait_w(kGFull, T)) return;
    tc_fence_after();
    const bool diag = (c.row0 + T * 128 == c.i * kC);
    float* carry_row = p.carry ? p.carry + (chunk_id * (L / 64) + (c.row0 + T * 128) / 64) * 128 + k : nullptr;
    if (carry_row) carry_row[0] = carry;
    // The prefix inside a tile is  carry + (carry_lo + sum of the totals of earlier 32-row blocks + scan inside the block).
    float tprev = carry_lo, cval = carry;
#pragma unroll 1
    for (int cb = 0; cb < 4; ++cb) {
      uint32_t g[32];
      tmem_ld32(c.tmem + Cfg::tG + lane_base + cb * 32, g);
      tc_wait_ld();
      if (cb == 3) {
        tc_fence_before();
        c.arrive_w(kGFree);
      }
      if (cb == 2 && carry_row && (kC == 128 || c.row0 + T * 128 + 64 < L)) carry_row[128] = cval;      // prefix after the first 64 rows of the tile
      float v[32], t3r[32];
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const float4 t4 = reinterpret_cast<const float4*>(t3buf + cb * 32)[x];
        t3r[4 * x] = t4.x; t3r[4 * x + 1] = t4.y; t3r[4 * x + 2] = t4.z; t3r[4 * x + 3] = t4.w;
      }
      float local = 0.f;
      // (the diagonal tile is the only one with masked pairs: its tests are compiled into a path of its own)
      auto scan32 = [&](auto on_diag) {
        constexpr bool kDiag = decltype(on_diag)::value;
        const float2 k23 = make_float2(2.0f / 3.0f, 2.0f / 3.0f), s32 = make_float2(s3, s3), one2 = make_float2(1.0f, 1.0f),
                     mone2 = make_float2(-1.0f, -1.0f), ln2 = make_float2(0.6931471805599453f, 0.6931471805599453f);
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
          // two rows at a time with packed fp32 arithmetic: relu(g)^(2/3) through lg2(max(g, 0)) = -inf for g <= 0
          const float2 lg = make_float2(lg2(fmaxf(__uint_as_float(g[x]), 0.f)), lg2(fmaxf(__uint_as_float(g[x + 1]), 0.f)));
          const float2 e23 = fmul2(lg, k23);
          const float2 pw = make_float2(ex2(e23.x), ex2(e23.y));
          const float2 a = fmul2(fmul2(pw, s32), make_float2(t3r[x], t3r[x + 1]));
          const float2 om = ffma2(make_float2(fminf(a.x, clamp_hi()), fminf(a.y, clamp_hi())), mone2, one2);
          const float2 el = fmul2(make_float2(lg2(om.x), lg2(om.y)), ln2);
          const int q = cb * 32 + x;
          float2 run;
          run.x = local + (kDiag && q <= k ? 0.f : el.x);
          run.y = local = run.x + (kDiag && q + 1 <= k ? 0.f : el.y);
          const float2 cv = fadd2(make_float2(carry, carry), fadd2(make_float2(tprev, tprev), run));
          cval = cv.y;
          v[x] = (kDiag && q < k) ? mask_value() : cv.x;
          v[x + 1] = (kDiag && q + 1 < k) ? mask_value() : cv.y;
        }
      };
      if (diag) scan32(std::true_type{});
      else scan32(std::false_type{});
      tprev += local;
      if (!kCarryOnly) {
        if (cb == 0 && T >= Cfg::kCBufs && !c.wait_w(kCFree + T % Cfg::kCBufs, T / Cfg::kCBufs - 1)) return;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
          const int q = cb * 32 + x;
          *reinterpret_cast<float*>(sCs + (T % Cfg::kCBufs) * 65536 + q * 512 + ((((k >> 2) ^ (q & 7)) & 31) << 4) + (k & 3) * 4) = v[x];
        }
      }
    }
    add_to_carry(tprev);      // (tprev = carry_lo + the tile's total)
    if (!kCarryOnly) c.arrive_w(kCReady + T % Cfg::kCBufs);
  }
  if (p.total_out) p.total_out[key_id] = carry;
}

// ------------------------------------------------------------ softmax groups --
template <int D, int kC, int kOut>
__device__ __forceinline__ void fwd_softmax(const FwdCtx<D>& c, const FwdParams& p, int me) {
  constexpr bool kMerge = (kOut == kOutMerged);
  using Cfg = FwdCfg<D>;
  const int R = p.s.R, N = p.s.N;
  const int row = threadIdx.x & 127;
  const uint32_t lane_base = (uint32_t)((threadIdx.x >> 5) & 3) * 32u << 16;
  const uint8_t* sCrow0 = c.smem + Cfg::oCs + row * 512;
  const size_t chunk_id = (size_t)c.bh * N + c.i;
  const float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
  int t = 0;
  for (int T = 0; T < c.ntiles; ++T) {
    // Every softmax thread observes every phase of c_ready and arrives on c_free exactly
    // once per tile (after its last read of C in that tile), whether or not its group has
    // a head to process in this tile; parity waits stay within one phase of the barrier.
    const int cbuf = T % Cfg::kCBufs;
    const uint8_t* sCrow = sCrow0 + cbuf * 65536;
    if (!c.wait_w(kCReady + cbuf, T / Cfg::kCBufs)) return;
    int last_r = -1;
    for (int r = R - 1; r >= 0; --r)
      if (((T * R + r) & 1) == me) { last_r = r; break; }
    if (last_r < 0) c.arrive_w(kCFree + cbuf);
    for (int r = 0; r < R; ++r, ++t) {
      if ((t & 1) != me) continue;
      const int sb = t & 1, ob = t % Cfg::kOBufs;
      const uint32_t tS = c.tmem + (sb ? Cfg::tS1 : Cfg::tS0) + lane_base;
      const uint32_t tO = c.tmem + ((Cfg::kOBufs == 2 && ob) ? Cfg::tO1 : Cfg::tO0) + lane_base;
      if (!c.wait_w(kSFull + sb, t >> 1)) return;
      tc_fence_after();
      // pass 1: s = S + C (written back to TMEM), row max.  64 columns per round trip: the two loads are in flight together.
      float m = -INFINITY;
#pragma unroll 1
      for (int cb = 0; cb < kC / 64; ++cb) {
        uint32_t s[64];
        tmem_ld32(tS + cb * 64, s);
        tmem_ld32(tS + cb * 64 + 32, s + 32);
        tc_wait_ld();
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          const int chunk = cb * 16 + u;
          const float4 cv = *reinterpret_cast<const float4*>(sCrow + (((chunk ^ (row & 7)) & 31) << 4));
          const float2 a01 = fadd2(make_float2(__uint_as_float(s[u * 4 + 0]), __uint_as_float(s[u * 4 + 1])), make_float2(cv.x, cv.y));
          const float2 a23 = fadd2(make_float2(__uint_as_float(s[u * 4 + 2]), __uint_as_float(s[u * 4 + 3])), make_float2(cv.z, cv.w));
          m = fmax3(m, fmax3(a01.x, a01.y, a23.x), a23.y);
          s[u * 4 + 0] = __float_as_uint(a01.x); s[u * 4 + 1] = __float_as_uint(a01.y);
          s[u * 4 + 2] = __float_as_uint(a23.x); s[u * 4 + 3] = __float_as_uint(a23.y);
        }
        tmem_st32(tS + cb * 64, s);
        tmem_st32(tS + cb * 64 + 32, s + 32);
      }
      tc_wait_st();
      if (r == last_r) c.arrive_w(kCFree + cbuf);
      // pass 2: P = exp(s - m) as bf16 into the first 64 columns of the S buffer
      const float mb = m * kLog2e;
      const float2 kL2 = make_float2(kLog2e, kLog2e), nmb2 = make_float2(-mb, -mb);
      float2 l2 = make_float2(0.f, 0.f);
#pragma unroll 1
      for (int cb = 0; cb < kC / 64; ++cb) {
        uint32_t s[64];
        tmem_ld32(tS + cb * 64, s);
        tmem_ld32(tS + cb * 64 + 32, s + 32);
        tc_wait_ld();
        uint32_t pk[32];
#pragma unroll
        for (int u = 0; u < 32; ++u) {
          const float2 arg = ffma2(make_float2(__uint_as_float(s[2 * u]), __uint_as_float(s[2 * u + 1])), kL2, nmb2);
          const float2 pe = make_float2(ex2(arg.x), ex2(arg.y));
          __nv_bfloat162 h = __floats2bfloat162_rn(pe.x, pe.y);
          // the row sum uses the unrounded probabilities: the reference normalises in fp32 and rounds P afterwards
          // (universal_attention_autograd.py:158-159)
          l2 = fadd2(l2, pe);
          pk[u] = *reinterpret_cast<uint32_t*>(&h);
        }
        if (kOut != kOutStats) tmem_st32(tS + cb * 32, pk);
      }
      if (kOut != kOutStats) tc_wait_st();
      tc_fence_before();
      c.arrive_w(kPReady + sb);
      const int qg = c.srow0 + T * 128 + row;                       // row index inside the slab
      const bool in_range = kC == 128 || qg < p.Lr;                 // (kC = 64: the last tile may be half a tile)
      const float l = l2.x + l2.y;
      const float lse = m + lg2(l) * kLn2;
      const size_t orow = (chunk_id * R + r) * p.Lr + qg;
      const size_t mrow = ((size_t)c.bh * R + r) * p.Lr + qg;       // the row in (b,h,r,L) order (merged-output mode)
      float linv;
      if (kMerge) {
        // exp(lse - row_lse) / l = exp(m - row_lse): weight of this chunk in the row's softmax over all keys, applied
        // to the unnormalised P~ V (the load's latency runs under the wait for the PV product)
        linv = ex2((m - p.row_lse[mrow]) * kLog2e);
      } else {
        if (in_range) p.lse[orow] = lse;
        if (p.denom && in_range) p.denom[orow] = __float2bfloat16_rn(lse);
        linv = 1.0f / l;
      }
      if (kOut == kOutStats) continue;
      if (!c.wait_w(kOFull + sb, t >> 1)) return;
      tc_fence_after();
      if (kMerge) {
#pragma unroll 1
        for (int cb = 0; cb < D / 32; ++cb) {
          uint32_t o[32];
          tmem_ld32(tO + cb * 32, o);
          tc_wait_ld();
          if (cb == D / 32 - 1) {
            tc_fence_before();
            c.arrive_w(kOFree + sb);
          }
          float* dst = p.merged_acc + mrow * D + cb * 32;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            red_add_v4(dst + 4 * u, __uint_as_float(o[4 * u]) * linv, __uint_as_float(o[4 * u + 1]) * linv,
                       __uint_as_float(o[4 * u + 2]) * linv, __uint_as_float(o[4 * u + 3]) * linv);
        }
      } else if constexpr (D == 128) {
        // head_dim 128: rows leave as whole 128-byte lines, eight rows per store instruction: O is loaded in the fragment order, in
        // which a quad of threads holds a row, and regrouped to 32 contiguous bytes per thread.  Against the form below: B1 H16 R1 L4096
        // 331 -> 314 us, 2 x (8 x 2) heads of L1536 87 -> 76 us, B1 H8 R4 L8192 1312 -> 1301 us (at head_dim 64, with half as
        // much to store per score, the shuffles cost 1 % more than they give).
        const int lane = threadIdx.x & 31;
        __nv_bfloat16* out0 = p.out + (orow - lane) * D;      // the warp's first row
#pragma unroll 1
        for (int piece = 0; piece < 2 * D / 64; ++piece) {
          const int hh = piece & 1, cb = piece >> 1;          // 16 of the warp's 32 rows, 64 of the columns
          uint32_t o[32];
          tmem_ld_16x64(tO + ((uint32_t)(hh * 16) << 16) + cb * 64, o);
          const int ra = hh * 16 + (lane >> 2);
          const float la = __shfl_sync(0xffffffffu, linv, ra), lb = __shfl_sync(0xffffffffu, linv, ra + 8);
          tc_wait_ld();
          if (piece == 2 * D / 64 - 1) {
            tc_fence_before();
            c.arrive_w(kOFree + sb);
          }
          if (!in_range) continue;
          uint32_t wa[8], wb[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float2 va = fmul2(make_float2(__uint_as_float(o[4 * j]), __uint_as_float(o[4 * j + 1])), make_float2(la, la));
            const float2 vb = fmul2(make_float2(__uint_as_float(o[4 * j + 2]), __uint_as_float(o[4 * j + 3])), make_float2(lb, lb));
            const __nv_bfloat162 ha = __floats2bfloat162_rn(va.x, va.y), hb = __floats2bfloat162_rn(vb.x, vb.y);
            wa[j] = *reinterpret_cast<const uint32_t*>(&ha);
            wb[j] = *reinterpret_cast<const uint32_t*>(&hb);
          }
          quad_gather(wa, lane);
          quad_gather(wb, lane);
          __nv_bfloat16* dst = out0 + (size_t)ra * D + cb * 64 + (lane & 3) * 16;
          st_global_v8(dst, wa);
          st_global_v8(dst + 8 * D, wb);
        }
      } else {
        // 32 bytes per thread and row: with 16-byte stores every one of a warp's 32 rows got half a sector at a time, and the way from
        // L1 to L2 was busy half of the time with them (B4 H8 R4 L4096 970 -> 935 us)
        __nv_bfloat16* orow_ptr = p.out + orow * D;
#pragma unroll 1
        for (int cb = 0; cb < D / 32; ++cb) {
          uint32_t o[32];
          tmem_ld32(tO + cb * 32, o);
          tc_wait_ld();
          if (cb == D / 32 - 1) {
            tc_fence_before();
            c.arrive_w(kOFree + sb);
          }
          if (!in_range) continue;
          uint32_t pk[16];
          const float2 linv2 = make_float2(linv, linv);
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            const float2 ov = fmul2(make_float2(__uint_as_float(o[2 * u]), __uint_as_float(o[2 * u + 1])), linv2);
            __nv_bfloat162 h = __floats2bfloat162_rn(ov.x, ov.y);
            pk[u] = *reinterpret_cast<uint32_t*>(&h);
          }
          st_global_v8(orow_ptr + cb * 32, pk);
          st_global_v8(orow_ptr + cb * 32 + 16, pk + 8);
        }
      }
    }
  }
}

// Rows before key chunk `chunk`: every score is -1e12 (fp32 absorbs k.q), the softmax is
// uniform, so out = sum_k bf16(1/kC) V_k and lse = -1e12 (universal_attention_autograd.py:28,
// :154).  Pure HBM writes of the slab rows [row_lo, row_hi), done by warps 2-3 while the others
// compute.  A block of a whole sweep writes its own chunk's rows (chunks with many of them have
// few tiles to compute); a block of a segment of chunk i writes the same tiles' share of the
// rows before chunk n-1-i, which has as many tiles to write as chunk i has to compute.
template <int D, int kC>
__device__ __forceinline__ void fwd_fill_rows(const FwdCtx<D>& c, const FwdParams& p, __nv_bfloat16* vmean, int chunk, int row_lo, int row_hi) {
  if (row_lo >= row_hi) return;
  const int t = threadIdx.x - 64;                      // 0..63
  const int L = p.s.L, R = p.s.R, N = p.s.N;
  const __nv_bfloat16* v = static_cast<const __nv_bfloat16*>(p.vc) + ((size_t)c.bh * L + (size_t)chunk * kC) * D;
  const float w = 1.0f / kC;
  for (int d = t; d < D; d += 64) {
    float acc = 0.f;
#pragma unroll 16
    for (int k = 0; k < kC; ++k) acc = fmaf(w, __bfloat162float(v[(size_t)k * D + d]), acc);
    vmean[d] = __float2bfloat16_rn(acc);
  }
  named_bar_sync(2, 64);
  const size_t chunk_id = (size_t)c.bh * N + chunk;
  const int rows = row_hi - row_lo;
  constexpr int kVecPerRow = D / 8;                    // 16-byte vectors
  const uint4 mine = reinterpret_cast<const uint4*>(vmean)[t % kVecPerRow];   // 64 % kVecPerRow == 0: fixed per thread
  for (int r = 0; r < R; ++r) {
    const size_t first = (chunk_id * R + r) * p.Lr + row_lo;
    uint4* o = reinterpret_cast<uint4*>(p.out + first * D);
    const size_t nvec = (size_t)rows * kVecPerRow;
    for (size_t e = t; e < nvec; e += 64) o[e] = mine;
    for (int q = t; q < rows; q += 64) {
      p.lse[first + q] = mask_value();
      if (p.denom) p.denom[first + q] = __float2bfloat16_rn(mask_value());
    }
  }
}

// ------------------------------------------------------- log-retention of a tile --
// total[chunk][T][key] = sum of the log-retention of the key over the rows of tile T of its chunk's sweep: what the segments
// of a cut sweep start from.  One block per (b, h, chunk, tile), 16 warps: warp % 4 = TMEM lane quadrant (keys), warp / 4 = 32 of
// the 128 columns (rows).  Short by construction (one product of 128 x 128 x D and 32 elements per thread), so latency is all
// that counts: B1 H8 L640 D64, 120 blocks: 4.9 us.
template <int D, int kC, typename TG>
__global__ void __launch_bounds__(512)
tile_totals_kernel(const __grid_constant__ CUtensorMap tmK, Shape shp, int tiles, const void* ssrc, const void* sdest, float* total, int* status) {
  constexpr int kTile = 128 * D * 2, kBoxes = D / 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* t3 = reinterpret_cast<float*>(smem + 2 * kTile);
  float* part = t3 + 128;                                // [3][128]
  uint32_t* misc = reinterpret_cast<uint32_t*>(part + 384);      // [0] tmem base, [1] abort flag, [2..5] two barriers
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, BH = shp.B * shp.H, L = shp.L;
  const int bh = blockIdx.x % BH;
  int x = blockIdx.x / BH, i = 0;
  for (;; ++i) {
    const int nt = (L - i * kC + 127) / 128;
    if (x < nt) break;
    x -= nt;
  }
  const int row0 = i * kC + x * 128;
  const uint32_t bar = smem_u32(misc + 2), sb = smem_u32(smem);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 1);
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) status[0] = status[1] = 0;      // (spares the call a memset; a wait gives up two seconds later at the earliest)
    misc[1] = 0;
    mbar_init(bar, 1); mbar_init(bar + 8, 1);
    mbar_init_fence();
    mbar_expect_tx(bar, 2 * kTile);
    for (int b = 0; b < kBoxes; ++b) {
      tma_load_2d(sb + b * 16384, &tmK, b * 64, bh * L + i * kC, bar);
      tma_load_2d(sb + kTile + b * 16384, &tmK, b * 64, bh * L + row0, bar);
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(misc), 128);
    tmem_relinquish();
  }
  if (threadIdx.x >= 128 && threadIdx.x < 256) {
    const int q = threadIdx.x - 128;
    t3[q] = row0 + q < L ? cbrtf(Num<TG>::ld(static_cast<const TG*>(sdest) + (size_t)bh * L + row0 + q)) : 0.f;
  }
  const int quad = warp & 3, grp = warp >> 2, k = quad * 32 + lane;
  const float s3 = k < kC ? cbrtf(Num<TG>::ld(static_cast<const TG*>(ssrc) + (size_t)bh * L + i * kC + k)) : 0.f;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = misc[0];
  if (threadIdx.x == 0 && mbar_wait(bar, 0, abort_flag)) {
    constexpr uint32_t idesc = idesc_bf16(128, 128, 0, 0);
    const uint32_t a = desc_lo(sb, 16), b = desc_lo(sb + kTile, 16);
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const uint32_t off = (ks >> 2) * 1024 + (ks & 3) * 2;
      mma_ss(tmem, desc_from_lo(a + off), desc_from_lo(b + off), idesc, ks > 0);
    }
    tc_commit(bar + 8);
  }
  __syncwarp();
  float local = 0.f;
  if (mbar_wait_warp(bar + 8, 0, abort_flag)) {
    tc_fence_after();
    uint32_t g[32];
    tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + grp * 32, g);
    tc_wait_ld();
#pragma unroll
    for (int q = 0; q < 32; ++q) {
      float ell = log_retention(gated_affinity(gram_pow23(__uint_as_float(g[q])), s3, t3[grp * 32 + q]));
      if (x == 0 && grp * 32 + q <= k) ell = 0.f;      // (only the first tile of a sweep has rows at or before the key)
      local += ell;
    }
  }
  if (grp) part[(grp - 1) * 128 + k] = local;
  tc_fence_before();
  __syncthreads();
  if (grp == 0 && k < kC) total[(((size_t)bh * shp.N + i) * tiles + x) * 128 + k] = ((local + part[k]) + part[128 + k]) + part[256 + k];
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    for (int it = 0; it < 64; ++it) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, 128);
}

template <int D, int kC, typename TG, bool kCarryOnly, int kOut = kOutTiles>
__global__ void __launch_bounds__(512, 1)
fwd_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
           const __grid_constant__ CUtensorMap tmQ, FwdParams p) {
  using Cfg = FwdCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint32_t* misc = reinterpret_cast<uint32_t*>(smem + Cfg::oMisc);   // [0] tmem base, [1] abort flag
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int BH = p.s.B * p.s.H;

  FwdCtx<D> c;
  c.smem = smem;
  c.bars = smem_u32(smem + Cfg::oBar);
  c.abort_flag = reinterpret_cast<volatile int*>(misc + 1);
  // heavy chunks (small i: most row tiles) first
  int x = blockIdx.x / BH;
  c.bh = blockIdx.x - x * BH;
  int fill_chunk, fill_lo = 0, fill_hi;      // rows before which chunk this block writes, in slab rows
  if (p.seg == 0) {
    c.i = x;
    c.t0 = 0;
    if (kC == 128) {
      const int j0 = c.i > p.j_begin ? c.i : p.j_begin;
      c.row0 = j0 * 128;
      c.ntiles = p.j_end - j0;              // <= 0: nothing to compute for this chunk in the row range (only the fill)
    } else {
      c.row0 = c.i * kC;
      c.ntiles = (p.s.L - c.row0 + 127) / 128;
    }
    fill_chunk = c.i;
    fill_lo = p.r0;
    fill_hi = p.r0 + (kC == 128 ? ((c.i < p.j_end ? c.i : p.j_end) - p.j_begin) * 128 : c.i * kC);
  } else {
    int nt;
    for (c.i = 0;; ++c.i) {
      nt = (p.s.L - c.i * kC + 127) / 128;
      const int ns = (nt + p.seg - 1) / p.seg;
      if (x < ns) break;
      x -= ns;
    }
    c.t0 = x * p.seg;
    c.row0 = c.i * kC + c.t0 * 128;
    c.ntiles = nt - c.t0 < p.seg ? nt - c.t0 : p.seg;
    fill_chunk = p.s.N - 1 - c.i;
    fill_lo = c.t0 * 128;
    fill_hi = min(fill_lo + c.ntiles * 128, fill_chunk * kC);
  }
  c.srow0 = p.r0 + c.row0 - p.j_begin * 128;

  if (threadIdx.x == 0) {
    misc[1] = 0;
    for (int b = 0; b < kNumBars; ++b) {
      uint32_t count = 1;
      // one arrival per warp of the group that signals
      if (b == kGFree || b == kCReady || b == kCReady + 1) count = kC / 32;
      if (b == kT3Ready) count = 4;
      if (b == kCFree || b == kCFree + 1) count = 8;
      if (b == kPReady || b == kPReady + 1 || b == kOFree || b == kOFree + 1) count = 4;
      mbar_init(c.bar(b), count);
    }
    mbar_init_fence();
    prefetch_tmap(&tmK);
    prefetch_tmap(&tmV);
    prefetch_tmap(&tmQ);
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(misc), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = misc[0];

  if (warp == 0) {
    if (lane == 0 && c.ntiles > 0) fwd_producer<D, kC, kCarryOnly>(c, p, &tmK, &tmV, &tmQ);
  } else if (warp == 1) {
    if (lane == 0 && c.ntiles > 0) fwd_mma<D, kC, kCarryOnly, kOut>(c, p);
  } else if (warp >= 4 && warp < 8) {
    if (c.ntiles > 0) fwd_decay<D, kC, TG, kCarryOnly>(c, p);
    else if (p.total_out)      // no row of the range sees this chunk: its prefix does not move
      p.total_out[((size_t)c.bh * p.s.N + c.i) * 128 + (threadIdx.x & 127)] =
          p.carry_in ? p.carry_in[((size_t)c.bh * p.s.N + c.i) * 128 + (threadIdx.x & 127)] : 0.f;
  } else if (warp >= 8 && !kCarryOnly) {
    if (c.ntiles > 0) fwd_softmax<D, kC, kOut>(c, p, (warp - 8) >> 2);
  } else if ((warp == 2 || warp == 3) && !kCarryOnly && p.fill_masked) {
    fwd_fill_rows<D, kC>(c, p, reinterpret_cast<__nv_bfloat16*>(smem + Cfg::oFill), fill_chunk, fill_lo, fill_hi);
  }

  tc_fence_before();
  __syncthreads();
  if (*c.abort_flag) {
    if (threadIdx.x == 0) atomicExch(p.status, 1);
    // let copies and MMAs that are still in flight drain before shared memory and TMEM are released
    for (int it = 0; it < 64; ++it) __nanosleep(2000);
    __syncthreads();
  }
  if (warp == 0) tmem_dealloc(c.tmem, 512);
}

}  // namespace sm100
}  // namespace ua
