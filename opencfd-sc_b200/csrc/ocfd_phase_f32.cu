// Instantiations of the merged stage launch (ocfd_phase.cuh), float arithmetic.
#include "ocfd_phase.cuh"

namespace ocfd {
template cudaError_t launch_phase<float>(bool, int, const FaceArgs<float>[3], const ViscArgs<float, float>&, cudaStream_t);
cudaError_t setup_phase_kernels_f32() { return setup_phase<float>(); }
}  // namespace ocfd
