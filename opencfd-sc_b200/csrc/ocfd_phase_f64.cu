// Instantiations of the merged stage launch (ocfd_phase.cuh), double arithmetic.
#include "ocfd_phase.cuh"

namespace ocfd {
template cudaError_t launch_phase<double>(bool, int, const FaceArgs<double>[3], const ViscArgs<double, double>&, cudaStream_t);
cudaError_t setup_phase_kernels_f32();
cudaError_t setup_phase_kernels() {
  cudaError_t e = setup_phase<double>();
  return e == cudaSuccess ? setup_phase_kernels_f32() : e;
}
}  // namespace ocfd
