// flow_fp32.cu -- the one-launch sweeps with FP32 storage.
#include "flow_kernel.cuh"
#include "sweep_kernel.cuh"

namespace mlx {
const void* flow_kernel_fp32(int mat_kind, bool damp, bool ct, bool small) {
  if (ct && !small && mat_kind == MAT_NH) return (const void*)k_flow<float, MAT_NH, false, true, 512>;
  if (ct) return flow_kernel_of<float, true, 256>(mat_kind, damp);
  return small ? flow_kernel_of<float, false, 256>(mat_kind, damp) : flow_kernel_of<float, false, 512>(mat_kind, damp);
}
const void* flow_pack_kernel_fp32(int mat_kind) { return flow_pack_kernel_of<float>(mat_kind); }
const void* sweep_kernel_fp32(int mat_kind, bool damp) { return sweep_kernel_of<float>(mat_kind, damp); }
}  // namespace mlx
