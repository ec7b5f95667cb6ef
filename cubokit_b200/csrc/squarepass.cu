// The FP32 position pass for 64 x 64 and 96 x 96 detectors (sm_100a): the any-size pass (anypass.cuh) with its geometry
// fixed at compile time.
//
// Same arithmetic as the other passes (exit wave, forward 2-D FFT, Fourier-modulus projection with the 1/n of ifft2
// folded in, inverse 2-D FFT; Ptychography.swift:321-350), one CTA per position, the plane in shared memory, two in-place
// stages a line (N = RA RB): decimation in frequency forward, digit-reversed spectrum, decimation in time back.  Seven
// steps: exit wave and first row stage from global memory; second row stage; first column stage; second column stage,
// projection and its inverse; then the mirrored three, the last writing dpsi.  No division is left, every loop's trip count
// is known and a thread keeps its column (or row, or sample of a row) through a step.  The position's amplitudes are
// prefetched into L2 when the CTA starts.
//
// Bound by shared-memory wavefronts (64 x 64 82 % of the pipe, 96 x 96 83 %; issue 62 and 51 %, HBM a quarter and a fifth).
// Below that the CTAs per SM decide (before the projection's present form: 96 x 96 three of 384 threads at 56 registers 0.26
// ms per pass of 3,600 positions, two at 80 registers 0.29, three of 192 threads 0.30; 64 x 64 four of 256 threads 0.109 ms,
// eight of 128 0.121).  They replace register-resident line transforms, two CTAs per SM: 96 x 96 0.558 -> 0.240 ms (59 -> 138
// Gpixel/s), 64 x 64 0.197 -> 0.087 (75 -> 170).
#include "engine.h"
#include "project.cuh"
#include "regdft.cuh"

namespace cubo {

namespace {

__device__ __forceinline__ int swrap(int v, int size) { return v < 0 ? v + size : (v >= size ? v - size : v); }

// x[q] *= W_N^{jq} (conjugate when INV)
template <bool INV, int R>
__device__ __forceinline__ void stwiddle(float2 (&x)[R], int j, const float2 *tw) {
#pragma unroll
    for (int q = 1; q < R; q++) x[q] = regdft::turn<float2, INV>(x[q], tw[q * j]);
}

// One position.  Row slots: q RB + s holds the column frequency q + RA s; column slots: q RA + s the row frequency q + RB s.
template <int N, int RA, int RB, int NT>
__device__ __forceinline__ void square_pass_body(const PositionPassArgs<float> &a, int p) {
    static_assert(RA * RB == N && NT % RB == 0 && NT % N == 0 && N % 32 == 0, "shape");
    constexpr int P = N + 1, kRows = NT / RB, kGroups = NT / N;
    static_assert(N % kRows == 0 && RA % kGroups == 0 && RB % kGroups == 0, "shape");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double scratch[NT / 32];
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = D + N * P;
    const int tid = threadIdx.x;
    const float *A = a.amplitudes + (size_t)p * (N * N);
    if (tid == 0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A), "r"((unsigned)(N * N * sizeof(float)))
                     : "memory");
    for (int i = tid; i < N; i += NT) tw[i] = a.tw_rows[i];
    const int rr = a.scan.rr[p], cc = a.scan.cc[p], cls = a.scan.cls[p];
    __syncthreads();
    const int j1 = tid % RB, r1 = tid / RB;     // the ends: samples j1 + RB r of rows r1 + kRows k
    const int line = tid % N, group = tid / N;  // the inner steps: a row or a column, blocks group + kGroups k
    {  // exit wave (Ptychography.swift:321-336) and first row stage
        const float2 *S = a.shifted + (size_t)cls * (N * N) + j1;
        const bool interior = cc >= N / 2 && cc + N / 2 <= a.object_columns;
#pragma unroll
        for (int k = 0; k < N / kRows; k++) {
            const int row = r1 + k * kRows;
            const float2 *orow =
                a.object + (size_t)swrap(rr + (row < N / 2 ? row : row - N), a.object_rows) * a.object_columns;
            const float2 *s = S + row * N;
            float2 x[RA], o[RA];
#pragma unroll
            for (int r = 0; r < RA; r++) {
                const int c = j1 + r * RB;
                const int off = c < N / 2 ? c : c - N;
                x[r] = s[r * RB];
                o[r] = orow[interior ? cc + off : swrap(cc + off, a.object_columns)];
            }
#pragma unroll
            for (int r = 0; r < RA; r++) x[r] = regdft::turn<float2, false>(x[r], o[r]);
            regdft::dft<float, false, RA>(x);
            stwiddle<false, RA>(x, j1, tw);
            float2 *y = D + row * P + j1;
#pragma unroll
            for (int q = 0; q < RA; q++) y[q * RB] = x[q];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RA / kGroups; k++) {  // rows, second stage: adjacent slots
        float2 *x0 = D + line * P + (group + k * kGroups) * RB;
        float2 x[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) x[r] = x0[r];
        regdft::dft<float, false, RB>(x);
#pragma unroll
        for (int r = 0; r < RB; r++) x0[r] = x[r];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RA / kGroups; k++) {  // columns, first stage
        const int j = group + k * kGroups;
        float2 *x0 = D + j * P + line;
        float2 x[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) x[r] = x0[r * RA * P];
        regdft::dft<float, false, RB>(x);
        stwiddle<false, RB>(x, j, tw);
#pragma unroll
        for (int r = 0; r < RB; r++) x0[r * RA * P] = x[r];
    }
    __syncthreads();
    double err = 0;
    {
        const float *am = A + (line / RB + RA * (line % RB));  // this column slot's frequency
#pragma unroll
        for (int k = 0; k < RB / kGroups; k++) {  // columns, second stage, projection (Ptychography.swift:338-349) and back
            const int b = group + k * kGroups;
            float2 *x0 = D + b * RA * P + line;
            float measured[RA];
#pragma unroll
            for (int q = 0; q < RA; q++) measured[q] = am[(b + RB * q) * N];
            float2 x[RA];
#pragma unroll
            for (int r = 0; r < RA; r++) x[r] = x0[r * P];
            regdft::dft<float, false, RA>(x);
            project_values<float, RA>(x, measured, a.inv_n, err);
            regdft::dft<float, true, RA>(x);
#pragma unroll
            for (int r = 0; r < RA; r++) x0[r * P] = x[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RA / kGroups; k++) {  // columns, first stage, inverse
        const int j = group + k * kGroups;
        float2 *x0 = D + j * P + line;
        float2 x[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) x[r] = x0[r * RA * P];
        stwiddle<true, RB>(x, j, tw);
        regdft::dft<float, true, RB>(x);
#pragma unroll
        for (int r = 0; r < RB; r++) x0[r * RA * P] = x[r];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < RA / kGroups; k++) {  // rows, second stage, inverse
        float2 *x0 = D + line * P + (group + k * kGroups) * RB;
        float2 x[RB];
#pragma unroll
        for (int r = 0; r < RB; r++) x[r] = x0[r];
        regdft::dft<float, true, RB>(x);
#pragma unroll
        for (int r = 0; r < RB; r++) x0[r] = x[r];
    }
    __syncthreads();
    {  // rows, first stage, inverse, into dpsi
        float2 *out = a.dpsi + (size_t)p * (N * N) + j1;
#pragma unroll
        for (int k = 0; k < N / kRows; k++) {
            const int row = r1 + k * kRows;
            const float2 *y = D + row * P + j1;
            float2 x[RA];
#pragma unroll
            for (int q = 0; q < RA; q++) x[q] = y[q * RB];
            stwiddle<true, RA>(x, j1, tw);
            regdft::dft<float, true, RA>(x);
#pragma unroll
            for (int r = 0; r < RA; r++) out[row * N + r * RB] = x[r];
        }
    }
    // the position's squared residual, summed over the CTA in a fixed order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) err += __shfl_down_sync(0xffffffffu, err, o);
    if ((tid & 31) == 0) scratch[tid >> 5] = err;
    __syncthreads();
    if (tid == 0) {
        double total = 0;
        for (int w = 0; w < NT / 32; w++) total += scratch[w];
        a.error[p] = total;
    }
}

template <int N, int RA, int RB, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) square_pass_kernel(const __grid_constant__ PositionPassArgs<float> a) {
    square_pass_body<N, RA, RB, NT>(a, a.first + blockIdx.x);
}

// Grouped form (batches): one CTA per (item, position) unit; prefix[i] .. prefix[i + 1] - 1 are item i's units.
template <int N, int RA, int RB, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) square_pass_grouped_kernel(const PositionPassArgs<float> *args,
                                                                       const int *prefix, int items, int total) {
    const int u = blockIdx.x;
    int lo = 0, hi = items - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= u) lo = mid; else hi = mid - 1;
    }
    const PositionPassArgs<float> a = args[lo];
    square_pass_body<N, RA, RB, NT>(a, a.first + (u - prefix[lo]));
}

template <int N>
constexpr size_t square_smem() { return (size_t)(N * (N + 1) + N) * sizeof(float2); }

constexpr auto square64 = square_pass_kernel<64, 4, 16, 256, 4>;
constexpr auto square96 = square_pass_kernel<96, 12, 8, 384, 3>;
constexpr auto square64_grouped = square_pass_grouped_kernel<64, 4, 16, 256, 4>;
constexpr auto square96_grouped = square_pass_grouped_kernel<96, 12, 8, 384, 3>;

}  // namespace

bool square_pass_applicable(int rows, int columns) { return rows == columns && (rows == 64 || rows == 96); }

cudaError_t configure_square_pass() {
    cudaError_t e = cudaFuncSetAttribute(square64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)square_smem<64>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(square96, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)square_smem<96>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(square64_grouped, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)square_smem<64>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(square96_grouped, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)square_smem<96>());
    return e;
}

cudaError_t launch_square_pass(const PositionPassArgs<float> &a, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    if (a.rows == 64 && a.columns == 64) square64<<<a.count, 256, square_smem<64>(), s>>>(a);
    else if (a.rows == 96 && a.columns == 96) square96<<<a.count, 384, square_smem<96>(), s>>>(a);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_square_pass_grouped(const PositionPassArgs<float> *args, const int *prefix, int items, int total,
                                       int N, cudaStream_t s) {
    if (total <= 0) return cudaSuccess;
    if (N == 64) square64_grouped<<<total, 256, square_smem<64>(), s>>>(args, prefix, items, total);
    else if (N == 96) square96_grouped<<<total, 384, square_smem<96>(), s>>>(args, prefix, items, total);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

}  // namespace cubo
