// Launchers of the tiled fp32 kernels.
#include "ua_tiled.cuh"
#include "ua_tiled_host.h"

namespace ua {
namespace tiled {

bool forward(const Params& p, bool f32, bool gates_f32, cudaStream_t st) {
  if (f32) return forward_t<float, float>(p, st);
  return gates_f32 ? forward_t<__nv_bfloat16, float>(p, st) : forward_t<__nv_bfloat16, __nv_bfloat16>(p, st);
}
bool backward(const Params& p, bool f32, bool gates_f32, cudaStream_t st) {
  if (f32) return backward_t<float, float>(p, st);
  return gates_f32 ? backward_t<__nv_bfloat16, float>(p, st) : backward_t<__nv_bfloat16, __nv_bfloat16>(p, st);
}
void leave(const Leave& v, bool f32, bool gates_f32, cudaStream_t st) {
  size_t most = 0;
  for (size_t n : v.n) most = n > most ? n : most;
  unsigned blocks = (unsigned)((most / 4 + kThreads - 1) / kThreads);
  if (blocks > kSms * 8) blocks = kSms * 8;
  if (f32) leave_kernel<float, float><<<blocks, kThreads, 0, st>>>(v);
  else if (gates_f32) leave_kernel<__nv_bfloat16, float><<<blocks, kThreads, 0, st>>>(v);
  else leave_kernel<__nv_bfloat16, __nv_bfloat16><<<blocks, kThreads, 0, st>>>(v);
}

}  // namespace tiled
}  // namespace ua
