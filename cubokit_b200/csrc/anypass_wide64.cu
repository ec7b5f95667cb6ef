// The any-size position pass with the prime radices 17 to 31 (double).
#include "anypass.cuh"

namespace cubo {

AnyKernelD any_wide_f64() { return any_pass_kernel<double, true>; }

}  // namespace cubo
