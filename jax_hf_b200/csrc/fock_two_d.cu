#include "fock_two_launch.cuh"

namespace hf {
// complex128 storage, FP64 transform
template int two_fock<double, double>(FockParams&, cudaStream_t, bool*);
}  // namespace hf
