#include "fock_two_launch.cuh"

namespace hf {
// complex64 storage, FP32 transform
template int two_fock<float, float>(FockParams&, cudaStream_t, bool*);
}  // namespace hf
