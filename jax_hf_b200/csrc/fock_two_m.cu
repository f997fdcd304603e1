#include "fock_two_launch.cuh"

namespace hf {
// complex128 storage, FP32 transform
template int two_fock<double, float>(FockParams&, cudaStream_t, bool*);
}  // namespace hf
