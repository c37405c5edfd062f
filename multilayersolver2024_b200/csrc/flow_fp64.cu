// flow_fp64.cu -- the one-launch sweeps with FP64 storage.
#include "flow_kernel.cuh"
#include "sweep_kernel.cuh"

namespace mlx {
const void* flow_kernel_fp64(int mat_kind, bool damp, bool ct) {
  return ct ? flow_kernel_of<double, true, 256>(mat_kind, damp) : flow_kernel_of<double, false, 256>(mat_kind, damp);
}
const void* flow_pack_kernel_fp64(int mat_kind) { return flow_pack_kernel_of<double>(mat_kind); }
const void* sweep_kernel_fp64(int mat_kind, bool damp) { return sweep_kernel_of<double>(mat_kind, damp); }
}  // namespace mlx
