// Launchers of the tensor-core backward.
#include "ua_sm100_host.cuh"

namespace ua {
namespace sm100 {
namespace {

template <int D, int kC, typename TG>
int launch_bwd2_t(const Shape& s, int mode, const void* kc, const void* vc, const void* xq, const void* g_out, const Bwd2Params& p,
                  cudaStream_t st) {
  CUtensorMap tmK, tmV, tmQ, tmG, tmDQ, tmDK;
  const uint64_t BH = (uint64_t)s.B * s.H;
  if (!make_rows_map(&tmK, kc, BH * s.L, D, 64) || !make_rows_map(&tmV, vc, BH * s.L, D, 64) ||
      !make_f32_rows_map(&tmDK, p.acc_dkr, BH * s.L, D, 64))
    return UA_ERR_CUDA;
  if (p.heads == 0) {
    tmQ = tmK; tmG = tmK; tmDQ = tmDK;       // never used
  } else if (!make_rows_map(&tmQ, xq, BH * s.R * p.Lr, D, 64) ||
             !make_rows_map(&tmG, g_out, (mode == 2 ? BH : BH * (s.N / p.m)) * s.R * p.Lr, D, 64) ||
             !make_f32_rows_map(&tmDQ, p.acc_dq, BH * s.R * p.Lr, D, 64)) {
    return UA_ERR_CUDA;
  }
  const int threads = 32 * (8 + 4 * NG);
  CUtensorMap tmO = tmG;
  auto kern = bwd2_kernel<D, kC, TG, 1, false>;
  size_t smem = Bwd2Cfg<D>::kSmemBytes;
  if (p.heads > 0) {
    kern = bwd2_kernel<D, kC, TG, 1, true>;
    if constexpr (kC == 128) {
      if (mode == 2) kern = bwd2_kernel<D, kC, TG, 2, true>;
      if (mode == 3) kern = bwd2_kernel<D, kC, TG, 3, true>;
      if (mode == 4) kern = bwd2_kernel<D, kC, TG, 4, true>;
    }
    // the forward's output tiles at hand (chunks of 128 keys, per-chunk form, head_dim 64): the row term comes from them
    if constexpr (D == 64 && kC == 128) {
      if (mode == 1 && p.out_tiles != nullptr) {
        if (!make_rows_map(&tmO, p.out_tiles, BH * s.N * s.R * p.Lr, D, 64)) return UA_ERR_CUDA;
        kern = s.R == 1 ? bwd2_kernel<D, kC, TG, 1, true, 2> : bwd2_kernel<D, kC, TG, 1, true, 1>;
        smem = s.R == 1 ? Bwd2Cfg<D, 2>::kSmemBytes : Bwd2Cfg<D, 1>::kSmemBytes;
      }
    }
  }
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return UA_ERR_CUDA;
  unsigned per = (unsigned)s.N;
  if (p.seg) {
    per = 0;
    for (int i = 0; i < s.N; ++i) per += ((s.L - i * kC) / 64 + p.seg - 1) / p.seg;
  }
  // (the correction pass of cut sweeps overlaps the end of the pass with heads, launched just before)
  if (p.heads == 0 && p.seg) {
    if (int e = launch_dependent(kern, (unsigned)BH * per, threads, smem, st, tmK, tmV, tmQ, tmG, tmDQ, tmDK, tmO, p)) return e;
  } else {
    kern<<<(unsigned)BH * per, threads, smem, st>>>(tmK, tmV, tmQ, tmG, tmDQ, tmDK, tmO, p);
  }
  if (p.acc_dt && mode != 4) {
    // row ranges: the row-side dK joins the accumulator; d static_dest of the range's rows comes out of it
    const int row_begin = p.j_begin * 128, row_end = p.j_end * 128;
    const long long warps = (long long)BH * (row_end - row_begin);
    if (warps > 0)
      row_side_finish_kernel<D, TG><<<(unsigned)((warps + 7) / 8), 256, 0, st>>>(
          static_cast<const __nv_bfloat16*>(kc), static_cast<const TG*>(p.sdest), p.acc_dkr, p.acc_dk, p.acc_dt, (int)BH, s.L, p.Lr,
          p.r0, row_begin, row_end);
  }
  return cudaGetLastError() == cudaSuccess ? UA_OK : UA_ERR_CUDA;
}

template <int D, typename TG>
int launch_finish_t(const Shape& s, const void* kc, const Bwd2Params& p, void* dkc, void* dxq, void* dvc, void* dss, void* ddest, cudaStream_t st) {
  const int rows = s.B * s.H * s.L, row_blocks = (rows + 8 * 128 / D - 1) / (8 * 128 / D);
  const size_t dq_vec = (size_t)rows * s.R * D / 8;
  using bf16 = __nv_bfloat16;
  return launch_dependent(bwd_finish_kernel<D, TG>, (unsigned)(row_blocks + (dq_vec + 255) / 256), 256, 0, st,
                          static_cast<const bf16*>(kc), static_cast<const TG*>(p.sdest), p.acc_dkr, p.acc_dk, p.acc_dq, p.acc_dv, p.acc_ds, p.dt_cols,
                          static_cast<bf16*>(dkc), static_cast<bf16*>(dxq), static_cast<bf16*>(dvc), static_cast<TG*>(dss), static_cast<TG*>(ddest),
                          rows, row_blocks, dq_vec);
}

}  // namespace

int launch_bwd2(const Shape& s, int gate_dtype, int mode, const void* kc, const void* vc, const void* xq, const void* g_out,
                const Bwd2Params& p, cudaStream_t st) {
#define UA_BWD2(D_, C_) (gate_dtype == UA_F32 ? launch_bwd2_t<D_, C_, float>(s, mode, kc, vc, xq, g_out, p, st) \
                                              : launch_bwd2_t<D_, C_, __nv_bfloat16>(s, mode, kc, vc, xq, g_out, p, st))
  if (s.C == 64) return s.D == 64 ? UA_BWD2(64, 64) : UA_BWD2(128, 64);
  return s.D == 64 ? UA_BWD2(64, 128) : UA_BWD2(128, 128);
#undef UA_BWD2
}

int launch_bwd_finish(const Shape& s, int gate_dtype, const void* kc, const Bwd2Params& p, void* dkc, void* dxq, void* dvc, void* dss,
                      void* ddest, cudaStream_t st) {
#define UA_FINISH(D_) (gate_dtype == UA_F32 ? launch_finish_t<D_, float>(s, kc, p, dkc, dxq, dvc, dss, ddest, st) \
                                            : launch_finish_t<D_, __nv_bfloat16>(s, kc, p, dkc, dxq, dvc, dss, ddest, st))
  return s.D == 64 ? UA_FINISH(64) : UA_FINISH(128);
#undef UA_FINISH
}

namespace {
// Rows before a chunk over the row tiles [p.j_begin, p.j_end): prep (per-chunk constants), sweep (one pass over the upstream
// gradient), finish (dK_i, and dV_i for a row range).  The caller has zeroed (or shares) acc_dq / acc_dk / acc_dv.
template <int D>
int launch_masked_t(const Shape& s, const void* kc, const void* vc, const void* xq, const void* g_out, float* acc_dq, MaskedParams p,
                    cudaStream_t st) {
  using Cfg = MkCfg<D>;
  const uint64_t BH = (uint64_t)s.B * s.H;
  CUtensorMap tmQ, tmG, tmDQ;
  if (!make_rows_map(&tmQ, xq, BH * s.R * p.Lr, D) || !make_rows_map(&tmG, g_out, BH * (s.N / p.m) * s.R * p.Lr, D) ||
      !make_f32_rows_map(&tmDQ, acc_dq, BH * s.R * p.Lr, D))
    return UA_ERR_CUDA;
  // Row tiles per work item.  An item pays for its start-up and for each chunk's N / w / u once, and adds to dQ where the groups at work share
  // L2, so it should be neither short nor long: 16 tiles with one to three query heads, 8 with four or more, and fewer where that would
  // leave SMs without an item.  Sweep times in us for 2 / 4 / 8 / 16 / 32 tiles, L4096:
  //   head_dim 64   B4 H8 R1 259 / 170 / 141 / 136 / 154    R2 340 / 250 / 221 / 224 / 273    R4 493 / 398 / 375 / 405 / 505
  //                 B4 H4 R8 405 / 362 / 371 / 444 / 613    B1 H4 R16 188 / 178 / 323 / 632 / 1199 (the grid's limit leaves 2: 189)
  //   head_dim 128  B1 H16 R1 502 / 301 / 224 / 198 / 199   H8 R4 451 / 350 / 319 / 345 / 420   H8 R8 705 / 599 / 589 / 654 / 808
  //                 H4 R16 627 / 607 / 587 / 703 / 1085
  // (4 tiles would win 3 to 10 % with eight or more heads of head_dim 64 and lose 2 to 3 % at 128.)
  const int last = (s.N - 1) / p.m * p.m, jcap = (last < p.j_end) ? last : p.j_end;      // no row tile at or after the last chunk is before any chunk
  for (p.jp = s.R >= 4 ? 8 : 16;; p.jp /= 2) {
    p.items_per_bh = 0;
    for (int g = 0; g * Cfg::kG < s.N; ++g) {
      int jmax = ((((g + 1) * Cfg::kG < s.N) ? (g + 1) * Cfg::kG : s.N) - 1) / p.m * p.m;
      if (jmax > jcap) jmax = jcap;
      if (jmax > p.j_begin) p.items_per_bh += (jmax - p.j_begin + p.jp - 1) / p.jp;
    }
    if (p.jp <= 2 || BH * p.items_per_bh * Cfg::kKB >= kSms) break;
  }
  if (p.items_per_bh == 0) return UA_OK;
  const auto* k16 = static_cast<const __nv_bfloat16*>(kc);
  const auto* v16 = static_cast<const __nv_bfloat16*>(vc);
  const int prep_smem = 2 * MkDense<D>::kTile + 2 * D * 4, finish_smem = MkDense<D>::kTile + D * 4;
  auto prep = masked_prep_kernel<D>;
  if (cudaFuncSetAttribute(prep, cudaFuncAttributeMaxDynamicSharedMemorySize, prep_smem) != cudaSuccess) return UA_ERR_CUDA;
  prep<<<(unsigned)(BH * s.N), 256, prep_smem, st>>>(k16, v16, p);
  auto sweep = p.m > 1 ? masked_sweep_kernel<D, true> : masked_sweep_kernel<D, false>;
  if (cudaFuncSetAttribute(sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) return UA_ERR_CUDA;
  sweep<<<(unsigned)(BH * p.items_per_bh * Cfg::kKB), 384, Cfg::kSmemBytes, st>>>(tmQ, tmG, tmDQ, p);
  masked_finish_kernel<D><<<(unsigned)(BH * s.N), 256, finish_smem, st>>>(v16, p);      // (at most 35 KB: no opt-in needed)
  return cudaGetLastError() == cudaSuccess ? UA_OK : UA_ERR_CUDA;
}

}  // namespace

int launch_masked(const Shape& s, const void* kc, const void* vc, const void* xq, const void* g_out, float* acc_dq,
                         const MaskedParams& p, cudaStream_t st) {
  return s.D == 64 ? launch_masked_t<64>(s, kc, vc, xq, g_out, acc_dq, p, st) : launch_masked_t<128>(s, kc, vc, xq, g_out, acc_dq, p, st);
}

}  // namespace sm100
}  // namespace ua
