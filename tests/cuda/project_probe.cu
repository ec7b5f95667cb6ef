// Test harness of project.cuh: the modulus and ratio of arrays of powers and measured amplitudes, and whole groups of values
// through the projection.
#include "project.cuh"

namespace {

template <typename T>
__global__ void ratio_kernel(const T *power, const T *measured, int n, T *modulus, T *ratio) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < n) cubo::modulus_and_ratio(power[i], measured[i], modulus[i], ratio[i]);
}

template <typename T>
__global__ void project_kernel(const cubo::C2<T> *in, const float *measured, int groups, T inv_n, cubo::C2<T> *out,
                               double *err) {
    const int g = blockIdx.x * 64 + threadIdx.x;
    if (g >= groups) return;
    cubo::C2<T> x[4];
    float m[4];
    for (int i = 0; i < 4; i++) { x[i] = in[4 * g + i]; m[i] = measured[4 * g + i]; }
    double e = 0;
    cubo::project_values<T, 4>(x, m, inv_n, e);
    for (int i = 0; i < 4; i++) out[4 * g + i] = x[i];
    err[g] = e;
}

template <typename T>
int run_ratio(const T *power, const T *measured, int n, T *modulus, T *ratio) {
    T *d = nullptr;
    if (cudaMalloc(&d, 4 * (size_t)n * sizeof(T)) != cudaSuccess) return 1;
    cudaMemcpy(d, power, n * sizeof(T), cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, measured, n * sizeof(T), cudaMemcpyHostToDevice);
    ratio_kernel<T><<<(n + 255) / 256, 256>>>(d, d + n, n, d + 2 * (size_t)n, d + 3 * (size_t)n);
    cudaMemcpy(modulus, d + 2 * (size_t)n, n * sizeof(T), cudaMemcpyDeviceToHost);
    cudaMemcpy(ratio, d + 3 * (size_t)n, n * sizeof(T), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return cudaGetLastError() != cudaSuccess;
}

template <typename T>
int run_project(const cubo::C2<T> *in, const float *measured, int groups, T inv_n, cubo::C2<T> *out, double *err) {
    using V = cubo::C2<T>;
    const size_t n = 4 * (size_t)groups;
    V *x = nullptr, *y = nullptr;
    float *m = nullptr;
    double *e = nullptr;
    if (cudaMalloc(&x, n * sizeof(V)) || cudaMalloc(&y, n * sizeof(V)) || cudaMalloc(&m, n * sizeof(float)) ||
        cudaMalloc(&e, groups * sizeof(double)))
        return 1;
    cudaMemcpy(x, in, n * sizeof(V), cudaMemcpyHostToDevice);
    cudaMemcpy(m, measured, n * sizeof(float), cudaMemcpyHostToDevice);
    project_kernel<T><<<(groups + 63) / 64, 64>>>(x, m, groups, inv_n, y, e);
    cudaMemcpy(out, y, n * sizeof(V), cudaMemcpyDeviceToHost);
    cudaMemcpy(err, e, groups * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(x);
    cudaFree(y);
    cudaFree(m);
    cudaFree(e);
    return cudaGetLastError() != cudaSuccess;
}

}  // namespace

extern "C" {
int ratio_f32(const float *p, const float *a, int n, float *m, float *r) { return run_ratio<float>(p, a, n, m, r); }
int ratio_f64(const double *p, const double *a, int n, double *m, double *r) { return run_ratio<double>(p, a, n, m, r); }
int project_f32(const float2 *x, const float *a, int g, float s, float2 *y, double *e) {
    return run_project<float>(x, a, g, s, y, e);
}
int project_f64(const double2 *x, const float *a, int g, double s, double2 *y, double *e) {
    return run_project<double>(x, a, g, s, y, e);
}
}
