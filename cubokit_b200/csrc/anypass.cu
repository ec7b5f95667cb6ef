// Host side of the any-size position pass (anypass.cuh): the radix plans, the launch, and the instances without the primes
// above 13.
#include <algorithm>
#include <type_traits>

#include "anypass.cuh"

namespace cubo {

namespace {

constexpr size_t kAnySmem = 226 * 1024;  // dynamic shared memory of one CTA: 227 KB less the kernel's static part

template <typename T>
size_t any_smem(int rows, int columns) {
    const size_t pitch = (size_t)(columns | 1);
    return (rows * pitch + rows + columns) * sizeof(C2<T>) + (size_t)(rows + columns) * sizeof(unsigned short);
}

bool wide(const AnyLine &l) {
    for (int i = 0; i < l.stages; i++)
        if (l.r[i] > 16) return true;
    return false;
}

template <typename T>
void (*any_kernel(bool wide_radices))(AnyPassArgs<T>) {
    if constexpr (std::is_same<T, float>::value) return wide_radices ? any_wide_f32() : any_pass_kernel<T, false>;
    else return wide_radices ? any_wide_f64() : any_pass_kernel<T, false>;
}

// Threads per CTA by how many CTAs' planes fit one SM (the registers allow 1024 FP32 and 512 FP64 threads there): the SM
// full, but no more than 128 threads for planes of a few thousand pixels, whose stages hold only n / 8 butterflies.
// Measured at a 60^2 scan, before the projection's present form, ms per pass: FP32 80 x 80 (4 fit) 0.246 at 256 threads, 0.294 at 512, 0.284 at 128; 48 x 48
// (11 fit) 0.097 at 128, 0.116 at 256; 120 x 112 (2 fit) 0.538 at 512, 0.596 at 256; 128 x 128 at a 64^2 scan (1 fits)
// 0.794 at 1024, 0.866 at 512.  FP64 96 x 100 (1 fits) 1.00 at 512, 1.17 at 256; 60 x 60 (3 fit) 0.311 at 256, 0.342 at
// 512; 40 x 40 (8 fit) 0.130 at 128, 0.141 at 256.
template <typename T>
int any_threads(int rows, int columns) {
    const int fit = (int)(kAnySmem / any_smem<T>(rows, columns));
    if (std::is_same<T, float>::value) return fit <= 1 ? 1024 : fit == 2 ? 512 : fit <= 4 ? 1024 / fit / 32 * 32 : fit <= 7 ? 192 : 128;
    return fit <= 2 ? 512 : fit == 3 ? 256 : 128;
}

}  // namespace

bool any_pass_applicable(int rows, int columns, bool fp64) {
    AnyLine r{}, c{};
    if (rows < 2 || columns < 2 || (long long)rows * columns >= 65536 || !plan_line(rows, 31, false, &r) || !plan_line(columns, 31, true, &c)) return false;
    return (fp64 ? any_smem<double>(rows, columns) : any_smem<float>(rows, columns)) <= kAnySmem;
}

cudaError_t configure_any_pass() {
    for (bool w : {false, true}) {
        cudaError_t e = cudaFuncSetAttribute(any_kernel<float>(w), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kAnySmem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(any_kernel<double>(w), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kAnySmem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename T>
cudaError_t launch_any_pass(const PositionPassArgs<T> &a, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    AnyPassArgs<T> g{};
    g.p = a;
    if (!plan_line(a.rows, 31, false, &g.rows) || !plan_line(a.columns, 31, true, &g.columns)) return cudaErrorInvalidValue;
    g.by_rows = divisor(a.rows);
    g.by_columns = divisor(a.columns);
    g.pitch = a.columns | 1;
    const int threads = any_threads<T>(a.rows, a.columns);
    any_kernel<T>(wide(g.rows) || wide(g.columns))<<<a.count, threads, any_smem<T>(a.rows, a.columns), s>>>(g);
    return cudaGetLastError();
}
template cudaError_t launch_any_pass<float>(const PositionPassArgs<float> &, cudaStream_t);
template cudaError_t launch_any_pass<double>(const PositionPassArgs<double> &, cudaStream_t);

}  // namespace cubo
