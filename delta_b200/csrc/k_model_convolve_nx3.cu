// The model convolve for n_max = 2 (model_convolve_fast.cuh).
#include "model_convolve_fast.cuh"

namespace dgpu {
template bool launch_model_convolve_nx<3>(cudaStream_t, const SubtractArgs&, const int2*, int, size_t);
}  // namespace dgpu
