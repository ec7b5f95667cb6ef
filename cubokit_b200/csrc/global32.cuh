// The FP32 position pass for detectors whose plane does not fit one CTA's shared memory (more than 16,384 pixels, sides
// up to 4096, e.g. 256 x 256), or any detector with CUBO_PTYCHO_VARIANT_GLOBAL.
//
// Same arithmetic as the shared-memory pass (exit wave, forward 2-D FFT, Fourier-modulus projection with the 1/n of
// ifft2 folded in, inverse 2-D FFT; Ptychography.swift:321-350, the Float path PtychographySingle.swift:137-176), in
// three launches per batch of positions, each reading and writing the residual plane once:
//
//  1. rows:    the exit wave X = S O[patch] of nl rows of one position and their forward row transforms, into dpsi;
//  2. columns: nl columns of one position: forward column transforms, the projection and its squared residual (one
//              FP64 partial per CTA, summed over the CTA in a fixed order), inverse column transforms;
//  3. rows:    the inverse row transforms.
//
// Lines are transformed as the any-size shared-memory pass does it (anypass.cuh): in-place stages of up to 16 samples in
// registers, decimation in frequency forward, in time back.  The first stage reads global memory and the last writes it,
// so a line of two stages (up to 256) crosses shared memory once, a column three times around the projection, with one
// and two barriers.  Rows leave in natural order: output s of block K is the frequency K + s L / r, so consecutive
// threads on consecutive K write consecutive addresses; a row's blocks are padded to an odd length in shared memory,
// which keeps both its stages free of bank conflicts.  128, 192 and 256 have their geometry fixed at compile time.  Lines
// with a prime factor above 31 take the direct DFT (g32_rows_direct, g32_columns_direct).
//
// 44 bytes a pixel cross HBM over the three launches (the shifted probe and the object come from L2), 2.24 ms per pass of 4,096
// positions of 256 x 256 = 0.80 of the measured copy rate (120 Gpixel/s).  The exit wave's rows are bound by LSU wavefronts (78 %
// of the pipe), the columns by issue (71 %) beside HBM (60), the inverse rows by HBM (79).  The Stockham stages before (lines
// staged whole, two barriers a stage; a run-time plan that spilled beyond four lengths, line counts that had to divide the
// side) took 4.08 ms; 128 x 225 4.59 -> 0.80 (2,500 positions), 160 x 200 5.86 -> 1.13 (2,500), 128 x 248 22.1 -> 0.91 (1,600), 96 x
// 211 5.78 -> 2.45 (400).
#pragma once

#include "anypass.cuh"

namespace cubo {


constexpr int kG32Threads = 256;
constexpr int kG32MaxN = 4096;  // the longest side; complex64 elements of the lines one CTA holds where the line allows it
constexpr size_t kG32Smem = 200 * 1024;

__device__ __forceinline__ int g32_wrap(int v, int size) { return v < 0 ? v + size : (v >= size ? v - size : v); }

// Fixed-order sum over the CTA: warps by shuffles, then thread 0 adds the warp sums in warp order.
static __device__ double g32_block_sum(double v, double *scratch) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    double total = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kG32Threads / 32; w++) total += scratch[w];
    __syncthreads();
    return total;  // valid in thread 0
}

struct G32Args {
    PositionPassArgs<float> p;
    AnyLine line;        // of the launch's lines: `columns` samples (rows launches) or `rows` samples (columns launch)
    Divisor by_nl;       // lines per CTA
    Divisor by_block[kAnyStages];  // blocks of a line, L / r, of each stage
    int nl, per;         // lines per CTA, CTAs per position
};

// Position of sample e of a row in shared memory: blocks of the last radix padded to an odd length.
__device__ __forceinline__ int padded(int e, const AnyLine &l) {
    const int last = l.r[l.stages - 1];
    return (last & 1) ? e : e + quotient(e, l.sub[l.stages >= 2 ? l.stages - 2 : 0]);
}

// ---------------------------------------------------------------------------------------------- rows, run-time plan

// Forward rows r0 .. of position p from the exit wave.  (Stage m - 2's sub is the last radix, so `padded` divides by it.)
template <bool WIDE>
__global__ void __launch_bounds__(kG32Threads, WIDE ? 1 : 4) g32_rows_forward(const __grid_constant__ G32Args g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const PositionPassArgs<float> &a = g.p;
    const AnyLine &l = g.line;
    const int L = l.L, m = l.stages, last = l.r[m - 1], nb = L / last, rl = last | 1, pitch = nb * rl;
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = D + (size_t)g.nl * pitch;
    unsigned short *base = reinterpret_cast<unsigned short *>(tw + L);  // block holding frequency K, 0 <= K < nb
    const int p = a.first + (int)(blockIdx.x / g.per), r0 = (int)(blockIdx.x % g.per) * g.nl;
    const int rows = min(g.nl, a.rows - r0);
    for (int i = threadIdx.x; i < L; i += kG32Threads) tw[i] = a.tw_columns[i];
    for (int b = threadIdx.x; b < nb; b += kG32Threads) base[slot_frequency(l, b * last)] = (unsigned short)b;
    const int rr = a.scan.rr[p], cc = a.scan.cc[p], cls = a.scan.cls[p];
    float2 *out = a.dpsi + (size_t)p * a.n + (size_t)r0 * L;
    __syncthreads();
    with_radix<WIDE>(l.r[0], [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int sub = (int)l.sub[0].d, step = m > 1 ? padded(sub, l) : 1;
        for (int i = threadIdx.x; i < rows * sub; i += kG32Threads) {
            const int row = quotient(i, l.sub[0]), j = i - row * sub;
            const float2 *S = a.shifted + (size_t)cls * a.n + (size_t)(r0 + row) * L + j;
            const float2 *o = a.object + (size_t)g32_wrap(rr + corner_offset(r0 + row, a.rows), a.object_rows) *
                                             a.object_columns;
            float2 x[R], q[R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                x[r] = S[r * sub];
                q[r] = o[g32_wrap(cc + corner_offset(j + r * sub, L), a.object_columns)];
            }
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = regdft::turn<float2, false>(x[r], q[r]);
            regdft::dft<float, false, R>(x);
            if (m == 1) {
#pragma unroll
                for (int r = 0; r < R; r++) out[(size_t)row * L + r] = x[r];
                continue;
            }
            twiddle<float, false, R>(x, j, 1, tw);
            float2 *y = D + row * pitch + padded(j, l);
#pragma unroll
            for (int r = 0; r < R; r++) y[r * step] = x[r];
        }
    });
    if (m == 1) return;
    __syncthreads();
    for (int s = 1; s + 1 < m; s++) {
        with_radix<WIDE>(l.r[s], [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int sub = (int)l.sub[s].d, step = padded(sub, l), blocks = (int)g.by_block[s].d;
            for (int i = threadIdx.x; i < rows * blocks; i += kG32Threads) {
                const int row = quotient(i, g.by_block[s]), b = i - row * blocks;
                const int blk = quotient(b, l.sub[s]), j = b - blk * sub;
                float2 *y = D + row * pitch + padded(blk * sub * R + j, l);
                float2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = y[r * step];
                regdft::dft<float, false, R>(x);
                twiddle<float, false, R>(x, j, l.before[s], tw);
#pragma unroll
                for (int r = 0; r < R; r++) y[r * step] = x[r];
            }
        });
        __syncthreads();
    }
    with_radix<WIDE>(last, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = threadIdx.x; i < rows * nb; i += kG32Threads) {
            const int row = quotient(i, g.by_block[m - 1]), K = i - row * nb;
            const float2 *y = D + row * pitch + (int)base[K] * rl;
            float2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[r];
            regdft::dft<float, false, R>(x);
            float2 *o = out + (size_t)row * L + K;
#pragma unroll
            for (int r = 0; r < R; r++) o[r * nb] = x[r];
        }
    });
}

// Inverse rows, in place in dpsi.
template <bool WIDE>
__global__ void __launch_bounds__(kG32Threads, WIDE ? 1 : 4) g32_rows_inverse(const __grid_constant__ G32Args g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const PositionPassArgs<float> &a = g.p;
    const AnyLine &l = g.line;
    const int L = l.L, m = l.stages, last = l.r[m - 1], nb = L / last, rl = last | 1, pitch = nb * rl;
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = D + (size_t)g.nl * pitch;
    unsigned short *base = reinterpret_cast<unsigned short *>(tw + L);
    const int p = a.first + (int)(blockIdx.x / g.per), r0 = (int)(blockIdx.x % g.per) * g.nl;
    const int rows = min(g.nl, a.rows - r0);
    for (int i = threadIdx.x; i < L; i += kG32Threads) tw[i] = a.tw_columns[i];
    for (int b = threadIdx.x; b < nb; b += kG32Threads) base[slot_frequency(l, b * last)] = (unsigned short)b;
    float2 *io = a.dpsi + (size_t)p * a.n + (size_t)r0 * L;
    __syncthreads();
    with_radix<WIDE>(last, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = threadIdx.x; i < rows * nb; i += kG32Threads) {
            const int row = quotient(i, g.by_block[m - 1]), K = i - row * nb;
            float2 *o = io + (size_t)row * L + K;
            float2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = o[r * nb];
            regdft::dft<float, true, R>(x);
            float2 *y = m == 1 ? o : D + row * pitch + (int)base[K] * rl;
#pragma unroll
            for (int r = 0; r < R; r++) y[r] = x[r];  // m == 1: nb = 1, the row itself
        }
    });
    if (m == 1) return;
    __syncthreads();
    for (int s = m - 2; s >= 1; s--) {
        with_radix<WIDE>(l.r[s], [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int sub = (int)l.sub[s].d, step = padded(sub, l), blocks = (int)g.by_block[s].d;
            for (int i = threadIdx.x; i < rows * blocks; i += kG32Threads) {
                const int row = quotient(i, g.by_block[s]), b = i - row * blocks;
                const int blk = quotient(b, l.sub[s]), j = b - blk * sub;
                float2 *y = D + row * pitch + padded(blk * sub * R + j, l);
                float2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = y[r * step];
                twiddle<float, true, R>(x, j, l.before[s], tw);
                regdft::dft<float, true, R>(x);
#pragma unroll
                for (int r = 0; r < R; r++) y[r * step] = x[r];
            }
        });
        __syncthreads();
    }
    with_radix<WIDE>(l.r[0], [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int sub = (int)l.sub[0].d, step = padded(sub, l);
        for (int i = threadIdx.x; i < rows * sub; i += kG32Threads) {
            const int row = quotient(i, l.sub[0]), j = i - row * sub;
            const float2 *y = D + row * pitch + padded(j, l);
            float2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[r * step];
            twiddle<float, true, R>(x, j, 1, tw);
            regdft::dft<float, true, R>(x);
            float2 *o = io + (size_t)row * L + j;
#pragma unroll
            for (int r = 0; r < R; r++) o[r * sub] = x[r];
        }
    });
}

// ------------------------------------------------------------------------------------------- columns, run-time plan

// Columns c0 .. of position p, sample e of column c at D[e nl + c].  The CTA's squared residual goes to
// error[p per + c0 / nl].
template <bool WIDE>
__global__ void __launch_bounds__(kG32Threads, WIDE ? 1 : 4) g32_columns(const __grid_constant__ G32Args g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double scratch[kG32Threads / 32];
    const PositionPassArgs<float> &a = g.p;
    const AnyLine &l = g.line;
    const int L = l.L, C = a.columns, m = l.stages, last = l.r[m - 1], nb = L / last, nl = g.nl;
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = D + (size_t)nl * L;
    unsigned short *freq = reinterpret_cast<unsigned short *>(tw + L);  // frequency of output 0 of each last-stage block
    const int p = a.first + (int)(blockIdx.x / g.per), c0 = (int)(blockIdx.x % g.per) * nl;
    const int lines = min(nl, C - c0);
    float2 *io = a.dpsi + (size_t)p * a.n + c0;
    const float *A = a.amplitudes + (size_t)p * a.n + c0;
    for (int i = threadIdx.x; i < L; i += kG32Threads) {
        tw[i] = a.tw_rows[i];
        asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (size_t)i * C));  // the amplitudes, for the centre step
    }
    for (int b = threadIdx.x; b < nb; b += kG32Threads) freq[b] = (unsigned short)slot_frequency(l, b * last);
    __syncthreads();
    if (m > 1) {
        with_radix<WIDE>(l.r[0], [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int sub = (int)l.sub[0].d;
            for (int i = threadIdx.x; i < nl * sub; i += kG32Threads) {
                const int j = quotient(i, g.by_nl), c = i - j * nl;
                if (c >= lines) continue;
                const float2 *o = io + (size_t)j * C + c;
                float2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = o[(size_t)r * sub * C];
                regdft::dft<float, false, R>(x);
                twiddle<float, false, R>(x, j, 1, tw);
                float2 *y = D + j * nl + c;
#pragma unroll
                for (int r = 0; r < R; r++) y[r * sub * nl] = x[r];
            }
        });
        __syncthreads();
    }
    for (int s = 1; s + 1 < m; s++) {
        with_radix<WIDE>(l.r[s], [&](auto rc) {
            inner_stage<float, false, decltype(rc)::value>(D, l, s, l.before[s], g.by_nl, 1, nl, tw);
        });
        __syncthreads();
    }
    double err = 0;
    with_radix<WIDE>(last, [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = threadIdx.x; i < nl * nb; i += kG32Threads) {
            const int b = quotient(i, g.by_nl), c = i - b * nl;
            if (c >= lines) continue;
            const float *am = A + (size_t)freq[b] * C + c;
            float measured[R];
#pragma unroll
            for (int q = 0; q < R; q++) measured[q] = am[(size_t)q * nb * C];
            float2 *y = m == 1 ? io + c : D + b * R * nl + c;
            const int step = m == 1 ? C : nl;
            float2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[(size_t)r * step];
            regdft::dft<float, false, R>(x);
            project_values<float, R>(x, measured, a.inv_n, err);
            regdft::dft<float, true, R>(x);
#pragma unroll
            for (int r = 0; r < R; r++) y[(size_t)r * step] = x[r];
        }
    });
    const double total = g32_block_sum(err, scratch);  // its barriers also order the centre step before the inverse ones
    if (threadIdx.x == 0) a.error[(size_t)p * g.per + c0 / nl] = total;
    if (m == 1) return;
    for (int s = m - 2; s >= 1; s--) {
        with_radix<WIDE>(l.r[s], [&](auto rc) {
            inner_stage<float, true, decltype(rc)::value>(D, l, s, l.before[s], g.by_nl, 1, nl, tw);
        });
        __syncthreads();
    }
    with_radix<WIDE>(l.r[0], [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int sub = (int)l.sub[0].d;
        for (int i = threadIdx.x; i < nl * sub; i += kG32Threads) {
            const int j = quotient(i, g.by_nl), c = i - j * nl;
            if (c >= lines) continue;
            const float2 *y = D + j * nl + c;
            float2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[r * sub * nl];
            twiddle<float, true, R>(x, j, 1, tw);
            regdft::dft<float, true, R>(x);
            float2 *o = io + (size_t)j * C + c;
#pragma unroll
            for (int r = 0; r < R; r++) o[(size_t)r * sub * C] = x[r];
        }
    });
}

using G32Kernel = void (*)(G32Args);
// The instances with the primes above 13, compiled in a file of their own.
G32Kernel g32_wide_rows_forward();
G32Kernel g32_wide_rows_inverse();
G32Kernel g32_wide_columns();

}  // namespace cubo
