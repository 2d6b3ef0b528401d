// Launchers of the tensor-core forward.
#include "ua_sm100_host.cuh"

namespace ua {
namespace sm100 {
namespace {

template <int D, int kC, typename TG, bool kCarryOnly, int kOut>
int launch_t(const Shape& s, const void* kc, const void* vc, const void* xq, FwdParams p, bool fill_masked, float* totals, cudaStream_t st) {
  using Cfg = FwdCfg<D>;
  CUtensorMap tmK, tmV, tmQ, tmO;
  const uint64_t BH = (uint64_t)s.B * s.H;
  if (!make_rows_map(&tmK, kc, BH * s.L, D)) return UA_ERR_CUDA;
  if (kCarryOnly) {
    tmV = tmK; tmQ = tmK;          // not used by the decay-only pass
  } else if (!make_rows_map(&tmV, vc, BH * s.L, D) || !make_rows_map(&tmQ, xq, BH * s.R * p.Lr, D)) {
    return UA_ERR_CUDA;
  }
  tmO = tmK;                       // (only read where output tiles are written)
  if (!kCarryOnly && kOut == kOutTiles && !make_rows_map(&tmO, p.out, BH * s.N * s.R * p.Lr, D, 32)) return UA_ERR_CUDA;
  p.vc = vc;
  p.fill_masked = (fill_masked && !kCarryOnly) ? 1 : 0;
  p.seg = totals ? fwd_split(s) : 0;
  unsigned blocks = (unsigned)(BH * s.N);
  if (p.seg) {
    p.tiles = sweep_tiles(s, 0);
    p.tile_totals = totals;
    unsigned nt = 0;
    blocks = 0;
    for (int i = 0; i < s.N; ++i) {
      nt += sweep_tiles(s, i);
      blocks += (sweep_tiles(s, i) + p.seg - 1) / p.seg;
    }
    blocks *= (unsigned)BH;
    constexpr int smem = 2 * 128 * D * 2 + 2048 + 64;
    auto tk = tile_totals_kernel<D, kC, TG>;
    if (cudaFuncSetAttribute(tk, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return UA_ERR_CUDA;
    tk<<<nt * (unsigned)BH, 512, smem, st>>>(tmK, s, p.tiles, p.ssrc, p.sdest, totals, p.status);
  }
  auto kern = fwd_kernel<D, kC, TG, kCarryOnly, kOut>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes) != cudaSuccess) return UA_ERR_CUDA;
  if (p.seg) return launch_dependent(kern, blocks, 512, Cfg::kSmemBytes, st, tmK, tmV, tmQ, tmO, p);
  kern<<<blocks, 512, Cfg::kSmemBytes, st>>>(tmK, tmV, tmQ, tmO, p);
  return cudaGetLastError() == cudaSuccess ? UA_OK : UA_ERR_CUDA;
}

template <int kC, bool kCarryOnly, int kOut>
int launch_c(const Shape& s, int gate_dtype, const void* kc, const void* vc, const void* xq, const FwdParams& p, bool fill_masked,
             float* totals, cudaStream_t st) {
  if (s.D == 64)
    return gate_dtype == UA_F32 ? launch_t<64, kC, float, kCarryOnly, kOut>(s, kc, vc, xq, p, fill_masked, totals, st)
                                : launch_t<64, kC, __nv_bfloat16, kCarryOnly, kOut>(s, kc, vc, xq, p, fill_masked, totals, st);
  return gate_dtype == UA_F32 ? launch_t<128, kC, float, kCarryOnly, kOut>(s, kc, vc, xq, p, fill_masked, totals, st)
                              : launch_t<128, kC, __nv_bfloat16, kCarryOnly, kOut>(s, kc, vc, xq, p, fill_masked, totals, st);
}

}  // namespace

int launch_fwd(const Shape& s, int gate_dtype, const void* kc, const void* vc, const void* xq, const FwdParams& p, bool fill_masked,
               float* totals, cudaStream_t st) {
  // without an output tensor only the log-sum-exp (and the decay-prefix table) is wanted: the statistics-only kernel
  if (s.C == 64)
    return p.out ? launch_c<64, false, kOutTiles>(s, gate_dtype, kc, vc, xq, p, fill_masked, totals, st)
                 : launch_c<64, false, kOutStats>(s, gate_dtype, kc, vc, xq, p, false, totals, st);
  return p.out ? launch_c<128, false, kOutTiles>(s, gate_dtype, kc, vc, xq, p, fill_masked, totals, st)
               : launch_c<128, false, kOutStats>(s, gate_dtype, kc, vc, xq, p, false, totals, st);
}

int launch_fwd_carry(const Shape& s, int gate_dtype, const void* kc, const FwdParams& p, cudaStream_t st) {
  return s.C == 64 ? launch_c<64, true, kOutTiles>(s, gate_dtype, kc, nullptr, nullptr, p, false, nullptr, st)
                   : launch_c<128, true, kOutTiles>(s, gate_dtype, kc, nullptr, nullptr, p, false, nullptr, st);
}

int launch_fwd_merge(const Shape& s, int gate_dtype, const void* kc, const void* vc, const void* xq, const FwdParams& p, cudaStream_t st) {
  return launch_c<128, false, kOutMerged>(s, gate_dtype, kc, vc, xq, p, false, nullptr, st);
}

}  // namespace sm100
}  // namespace ua
