// The FP32 position pass for a 128 x 128 detector (sm_100a).
//
// Same arithmetic as the other passes (exit wave, forward 2-D FFT, Fourier-modulus projection with the 1/n of ifft2
// folded in, inverse 2-D FFT; Ptychography.swift:321-350), with the in-place transforms of the any-size pass (anypass.cuh:
// decimation in frequency forward, digit-reversed spectrum, decimation in time back), laid out for one plane per SM:
//
//  * Persistent CTAs of 1024 threads (one per SM, 64 registers) walk the positions in a fixed stride; the 128 KB plane
//    stays in shared memory.  A row line is 8 x 16 (slot 16 q + s holds the frequency q + 8 s), a column line 16 x 8 (slot
//    8 q + s: q + 16 s).
//  * Warp w does all row steps of rows 4w .. 4w + 3 and all column steps of column slots 4w .. 4w + 3, so the two stages
//    of a line, and the column transform, projection and inverse column transform, follow one another behind __syncwarp;
//    the CTA meets only where rows become columns and back, twice a position.  Across a position's end there is no barrier
//    at all: a thread's last inverse row stage reads exactly the slots that its first stage of the next position writes,
//    so while some warps wait for the next exit wave's loads others still transform.
//  * Slot s of row r lies at column s ^ ((s >> 4) & 7) ^ 4 ((r ^ (r >> 3)) & 3): the 16 lanes of a half-warp then fall on
//    16 different 8-byte banks in every step (16 adjacent slots of a row; 2 rows x 8 blocks; 4 columns x 4 rows; 4 columns
//    x 4 row blocks), without padding, and a thread's address differs between its samples by an exclusive or with a
//    constant.
//  * The amplitudes are stored once per plan in the order the threads take them (four 16-byte loads each, consecutive
//    threads at consecutive addresses), and the next position's are prefetched into L2.
//  * The squared residual is summed in FP64 over the CTA in a fixed order: one partial per position, no atomics, bitwise
//    reproducible.
//  * The probe gradient (conj(O[patch]) dpsi and |O|^2, Ptychography.swift:356-357) is accumulated here, in tensor
//    memory: every thread owns 16 fixed detector pixels, so each CTA sums its positions in order and writes one
//    partial; a fixed-order FP64 reduction over the 148 partials follows.  This replaces a second pass over dpsi (0.35
//    ms at 16,384 positions, against 0.19 ms here).
//
// Bound by the LSU pipe (0.76 of its wavefronts) and instruction issue (0.59 of the slots) together, HBM at 20 %.  16,384
// positions take 1.79 ms (150 Gpixel/s); before, 2.81 ms: 512 threads of 128 registers, each line pass a register-resident
// four-step transform with an exchange in a padded tile and four CTA barriers a position (1.95 ms without the probe
// gradient in this form against 2.30 with a CTA barrier at every stage, 2.45 without the fused ends).
#include "engine.h"
#include "project.cuh"
#include "regdft.cuh"
#include "umma.cuh"

namespace cubo {

namespace {

constexpr int kN = 128;          // detector side
constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ int wrap_once(int v, int size) { return v < 0 ? v + size : (v >= size ? v - size : v); }

// x[q] *= W_128^{jq} (conjugate when INV)
template <bool INV, int R>
__device__ __forceinline__ void twiddle_line(float2 (&x)[R], int j, const float2 *tw) {
#pragma unroll
    for (int q = 1; q < R; q++) x[q] = regdft::turn<float2, INV>(x[q], tw[q * j]);
}

__device__ __forceinline__ float2 &at(char *plane, int offset) { return *reinterpret_cast<float2 *>(plane + offset); }

// The row's part of a slot's place.
__device__ __forceinline__ int row_turn(int row) { return 4 * ((row ^ (row >> 3)) & 3); }

// Second row stage, in place: the 16 adjacent slots of one block (byte offset b, 128-byte aligned but for the turn).
template <bool INV>
__device__ __forceinline__ void row_block(char *plane, int b) {
    float2 x[16];
#pragma unroll
    for (int r = 0; r < 16; r++) x[r] = at(plane, b ^ (r << 3));
    regdft::dft<float, INV, 16>(x);
#pragma unroll
    for (int r = 0; r < 16; r++) at(plane, b ^ (r << 3)) = x[r];
}

// First column stage, in place: rows j + 8 r of one column slot.
template <bool INV>
__device__ __forceinline__ void column_outer(char *plane, int b, int j, const float2 *tw) {
    float2 x[16];
#pragma unroll
    for (int r = 0; r < 16; r++) x[r] = at(plane, (b ^ ((r & 3) << 5)) + r * 8 * kN * 8);
    if (INV) twiddle_line<true, 16>(x, j, tw);
    regdft::dft<float, INV, 16>(x);
    if (!INV) twiddle_line<false, 16>(x, j, tw);
#pragma unroll
    for (int r = 0; r < 16; r++) at(plane, (b ^ ((r & 3) << 5)) + r * 8 * kN * 8) = x[r];
}

// Tensor-memory columns of this thread's probe-gradient accumulators for its k-th row: 8 detector pixels, real, imaginary
// and weight planes of 8 columns each; the eight warps that share a lane quadrant take 48 columns each.
__device__ __forceinline__ uint32_t accumulators(uint32_t tmem, int warp, int k) {
    return umma::tmem_addr(tmem, 32 * (warp & 3), 48 * (warp >> 2) + 24 * k);
}

__global__ void __launch_bounds__(kThreads, 1) fast128_kernel(const __grid_constant__ Fast128Args a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ double scratch[kWarps];
    __shared__ uint32_t tmem_base;
    char *plane = reinterpret_cast<char *>(smem_raw);
    float2 *tw = reinterpret_cast<float2 *>(plane + kN * kN * sizeof(float2));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid < kN) tw[tid] = a.tw128[tid];
    if (warp == 0) {
        umma::tmem_alloc(&tmem_base, 512);
        umma::tmem_relinquish();
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    const uint32_t tmem = tmem_base;

    // the ends of a row: samples j1 + 16 r of rows 4 warp + (lane >> 4) + 2 k, k = 0, 1
    const int j1 = lane & 15, row0 = 4 * warp + (lane >> 4);
    // the inner row stage: one block of one of the warp's rows (a half-warp takes rows two apart, eight blocks of each)
    const int blk = lane & 7, rs = lane >> 3, row_in = 4 * warp + (((rs & 1) << 1) | (rs >> 1));
    const int row_at = row_in * (kN * 8) + blk * 128 + ((blk ^ row_turn(row_in)) << 3);
    // the columns: slot 4 warp + (lane & 3), outer rows j + 8 r, inner row blocks j + 8 k
    const int slot = 4 * warp + (lane & 3), j = lane >> 2;
    const int slot_at = (slot & 0x70) * 8 + (((slot & 15) ^ (slot >> 4)) << 3);
    const int column_at = j * (kN * 8) + (slot_at ^ ((j & 3) << 5));

    // the exit wave of one row end (Ptychography.swift:321-336) and its first stage into the plane.  Column j1 + 16 r
    // lies left of the centre for r >= 4; when the whole window is inside the object no wrap is needed.
    auto object_row = [&](int p, int row) {
        return a.object + (size_t)wrap_once(a.scan.rr[p] + (row < kN / 2 ? row : row - kN), a.object_rows) *
                              a.object_columns;
    };
    auto patch = [&](int p, int row, float2 (&o)[8]) {
        const int cc = a.scan.cc[p];
        const float2 *orow = object_row(p, row);
        if (cc >= kN / 2 && cc + kN / 2 <= a.object_columns) {
#pragma unroll
            for (int r = 0; r < 8; r++) o[r] = orow[cc + j1 + (r < 4 ? 16 * r : 16 * r - kN)];
        } else {
#pragma unroll
            for (int r = 0; r < 8; r++)
                o[r] = orow[wrap_once(cc + j1 + (r < 4 ? 16 * r : 16 * r - kN), a.object_columns)];
        }
    };
    auto exit_wave = [&](int p, int row) {
        const float2 *S = a.shifted + (size_t)a.scan.cls[p] * (kN * kN) + row * kN + j1;
        float2 x[8], o[8];
#pragma unroll
        for (int r = 0; r < 8; r++) x[r] = S[16 * r];
        patch(p, row, o);
#pragma unroll
        for (int r = 0; r < 8; r++) x[r] = regdft::turn<float2, false>(x[r], o[r]);
        regdft::dft<float, false, 8>(x);
        twiddle_line<false, 8>(x, j1, tw);
        const int b = row * (kN * 8) + ((j1 ^ row_turn(row)) << 3);
#pragma unroll
        for (int q = 0; q < 8; q++) at(plane, (b ^ (q << 3)) + q * 128) = x[q];
    };

#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const uint32_t acc = accumulators(tmem, warp, k);
        float v[8];
#pragma unroll
        for (int part = 0; part < 3; part++) {  // an earlier band's partial of this CTA, or zero
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const size_t at_pixel = (size_t)blockIdx.x * (kN * kN) + (row0 + 2 * k) * kN + j1 + 16 * r;
                v[r] = !a.accumulate ? 0.f : part == 0 ? a.partial_grad[at_pixel].x
                                           : part == 1 ? a.partial_grad[at_pixel].y : a.partial_weight[at_pixel];
            }
            umma::tmem_st8(acc + 8 * part, v);
        }
        umma::tmem_wait_st();
    }
    const float inv_n = 1.0f / (float)(kN * kN);
    const int end = a.first + a.count;
    int p = a.first + blockIdx.x;
    if (p < end) {
#pragma unroll 1
        for (int k = 0; k < 2; k++) exit_wave(p, row0 + 2 * k);
    }
    for (; p < end; p += gridDim.x) {
        const float4 *A = reinterpret_cast<const float4 *>(a.amplitudes + (size_t)p * (kN * kN)) + tid;
        const int next = p + gridDim.x;
        if (tid == 0 && next < end)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(A + (size_t)gridDim.x * (kN * kN / 4)),
                         "r"((unsigned)(kN * kN * sizeof(float)))
                         : "memory");
        __syncwarp();
        row_block<false>(plane, row_at);
        __syncthreads();
        column_outer<false>(plane, column_at, j, tw);
        __syncwarp();
        // last column stage, projection (Ptychography.swift:338-349) and its inverse: rows 8 q + r of the slot, outputs
        // s = frequency q + 16 s
        double err = 0;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int q = j + 8 * k;
            const int b = q * (8 * kN * 8) + (slot_at ^ ((q & 3) << 5));
            const float4 m0 = A[(2 * k) * kThreads], m1 = A[(2 * k + 1) * kThreads];
            const float measured[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
            float2 x[8];
#pragma unroll
            for (int r = 0; r < 8; r++) x[r] = at(plane, (b ^ ((r & 3) << 5)) + r * (kN * 8));
            regdft::dft<float, false, 8>(x);
            project_values<float, 8>(x, measured, inv_n, err);
            regdft::dft<float, true, 8>(x);
#pragma unroll
            for (int r = 0; r < 8; r++) at(plane, (b ^ ((r & 3) << 5)) + r * (kN * 8)) = x[r];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) err += __shfl_down_sync(0xffffffffu, err, o);
        if (lane == 0) scratch[warp] = err;
        __syncwarp();
        column_outer<true>(plane, column_at, j, tw);
        __syncthreads();
        if (warp == 0) {
            double total = scratch[lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) total += __shfl_down_sync(0xffffffffu, total, o);
            if (lane == 0) a.error[p] = total;
        }
        row_block<true>(plane, row_at);
        __syncwarp();
        float2 *out = a.dpsi + (size_t)(p - a.dpsi_first) * (kN * kN) + j1;
#pragma unroll 1
        for (int k = 0; k < 2; k++) {
            const int row = row0 + 2 * k;
            const int b = row * (kN * 8) + ((j1 ^ row_turn(row)) << 3);
            float2 x[8], o[8];
            patch(p, row, o);
#pragma unroll
            for (int q = 0; q < 8; q++) x[q] = at(plane, (b ^ (q << 3)) + q * 128);
            twiddle_line<true, 8>(x, j1, tw);
            regdft::dft<float, true, 8>(x);
#pragma unroll
            for (int r = 0; r < 8; r++) out[row * kN + r * 16] = x[r];
            // probe gradient: conj(O[patch]) dpsi and |O|^2 added to this thread's pixels, in this CTA's position order
            const uint32_t acc = accumulators(tmem, warp, k);
            float v[8];
            umma::tmem_ld8(acc, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] += o[r].x * x[r].x + o[r].y * x[r].y;
            umma::tmem_st8(acc, v);
            umma::tmem_ld8(acc + 8, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] += o[r].x * x[r].y - o[r].y * x[r].x;
            umma::tmem_st8(acc + 8, v);
            umma::tmem_ld8(acc + 16, v);
            umma::tmem_wait_ld();
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] += o[r].x * o[r].x + o[r].y * o[r].y;
            umma::tmem_st8(acc + 16, v);
            umma::tmem_wait_st();
            if (next < end) exit_wave(next, row);
        }
    }
    // this CTA's probe-gradient partial, natural pixel order
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
        const uint32_t acc = accumulators(tmem, warp, k);
        float gr[8], gi[8], gw[8];
        umma::tmem_ld8(acc, gr);
        umma::tmem_ld8(acc + 8, gi);
        umma::tmem_ld8(acc + 16, gw);
        umma::tmem_wait_ld();
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const size_t at_pixel = (size_t)blockIdx.x * (kN * kN) + (row0 + 2 * k) * kN + j1 + 16 * r;
            a.partial_grad[at_pixel] = make_float2(gr[r], gi[r]);
            a.partial_weight[at_pixel] = gw[r];
        }
    }
    umma::fence_before_sync();
    __syncthreads();
    umma::fence_after_sync();
    if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

// [position][row][column] -> [position][h][thread][e]: the thread's amplitude i = 4 h + e is output s = i & 7 of its block
// k = i >> 3.
__global__ void permute_amplitudes_kernel(const float *in, float *out, long long positions) {
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= positions * kN * kN) return;
    const long long p = i / (kN * kN);
    const int rem = (int)(i - p * kN * kN);
    const int h = rem >> 12, t = (rem >> 2) & (kThreads - 1), e = rem & 3;
    const int k = h >> 1, s = 4 * (h & 1) + e, lane = t & 31;
    const int slot = 4 * (t >> 5) + (lane & 3), q = (lane >> 2) + 8 * k;
    const int row = q + 16 * s, column = (slot >> 4) + 8 * (slot & 15);
    out[i] = in[p * kN * kN + row * kN + column];
}

}  // namespace

bool fast128_applicable(int rows, int columns) { return rows == kN && columns == kN; }

int fast128_partials_per_position() { return 1; }

size_t fast128_smem() { return (size_t)(kN * kN + kN) * sizeof(float2); }

int fast128_ctas() { return 148; }  // fixed, so the probe-gradient summation order does not depend on the device

cudaError_t configure_fast128() {
    int device = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    if ((size_t)optin < fast128_smem()) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(fast128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fast128_smem());
}

cudaError_t launch_fast128(const Fast128Args &a, int ctas, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    (void)ctas;
    const int grid = a.count < fast128_ctas() ? a.count : fast128_ctas();
    fast128_kernel<<<grid, kThreads, fast128_smem(), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_permute_amplitudes(const float *in, float *out, long long positions, cudaStream_t s) {
    const long long total = positions * kN * kN;
    permute_amplitudes_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(in, out, positions);
    return cudaGetLastError();
}

}  // namespace cubo
