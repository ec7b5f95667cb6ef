// The any-size position pass with the prime radices 17 to 31 (float).
#include "anypass.cuh"

namespace cubo {

AnyKernelF any_wide_f32() { return any_pass_kernel<float, true>; }

}  // namespace cubo
