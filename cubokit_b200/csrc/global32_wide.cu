// The FP32 pass through global memory with the prime radices 17 to 31.
#include "global32.cuh"

namespace cubo {

G32Kernel g32_wide_rows_forward() { return g32_rows_forward<true>; }
G32Kernel g32_wide_rows_inverse() { return g32_rows_inverse<true>; }
G32Kernel g32_wide_columns() { return g32_columns<true>; }

}  // namespace cubo
