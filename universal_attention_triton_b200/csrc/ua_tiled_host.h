// Interface of the tiled fp32 kernels (ua_tiled.cuh, ua_tiled.cu).
#pragma once
#include "ua_common.cuh"

namespace ua {
namespace tiled {

constexpr int kRows = 32;      // rows per tile

struct Params {
  Shape s;
  const void *kc, *vc, *xq, *ssrc, *sdest;
  // forward
  void* out;               // chunk-major (b,h,n,r,L,d)
  float* lse;              // (b,h,n,r,L)
  void* denom;             // (b,h,n,r,L) in T, may be null
  int fill_masked;
  // backward
  const void *g_out, *g_denom;
  int g_denom_is_f32, skip_masked, only_masked;      // only_masked: the rows before each chunk alone (the others are another kernel's)
  float *acc_dk, *acc_dv, *acc_dq, *acc_ds, *acc_dt;     // fp32, zeroed
  float* dc;               // (b*h*n, L / 32, 32, C): dS summed over the heads
  float* dc_total;         // (b*h*n, L / 32, C): its sum over the rows of a tile
  float* totals;           // (b*h*n, L / 32, C): log-retention sums
};

// fp32 accumulators -> results, all of them in one launch
struct Leave {
  const float* src[5];
  void* dst[5];
  size_t n[5];             // elements
  int gate[5];             // in the gates' type
};

// The shapes of these kernels: chunks whose keys make whole quarter-warps of 4-key columns, rows that fit shared memory, and a
// dC table of at most 2 GB (it grows with L^2; beyond that the sweeping kernels of ua_simt.cuh, which keep nothing per pair).
inline bool fits(const Shape& s) {
  if ((s.C != 32 && s.C != 64 && s.C != 128) || s.D > 128) return false;
  if ((double)s.B * s.H * s.L * s.L * 4.0 > 2147483648.0) return false;
  return s.R <= 65535;
}
inline size_t table_bytes(const Shape& s) { return (size_t)s.B * s.H * s.N * (s.L / kRows) * s.C * sizeof(float); }

// Launches; f32: inputs and outputs fp32 (then the gates are too), else bf16.  False: a CUDA error.
bool forward(const Params& p, bool f32, bool gates_f32, cudaStream_t st);
bool backward(const Params& p, bool f32, bool gates_f32, cudaStream_t st);
void leave(const Leave& v, bool f32, bool gates_f32, cudaStream_t st);

}  // namespace tiled
}  // namespace ua
