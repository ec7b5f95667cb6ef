// The shared-memory position pass for any detector size whose side lengths have no prime factor above 31 (sm_100a).
//
// Same arithmetic as the other passes (exit wave, forward 2-D FFT, Fourier-modulus projection with the 1/n of ifft2
// folded in, inverse 2-D FFT; Ptychography.swift:321-350).  One CTA holds one position's plane in shared memory and
// every line transform runs in place:
//
//  * A line of length L = r_1 r_2 ... r_m (m the fewest factors of at most 16, or a prime up to 31) is transformed by
//    decimation in frequency: stage i takes blocks of B = L / (r_1 .. r_{i-1}) samples, sub = B / r_i, reads the r_i
//    samples j + r sub of a block, transforms them in registers, multiplies output q by W_B^{jq} and writes it back to
//    j + q sub.  Reads and writes of a butterfly are the same places, so a thread needs only its own butterfly in
//    registers and one barrier a stage (the Stockham form holds every value of the plane in registers across two).
//    The spectrum ends in digit-reversed order; the projection is pointwise and looks its frequency up, and the inverse
//    (decimation in time, the mirrored stages with conjugate twiddles) starts from that order.
//  * Fused ends: the first row stage forms the exit wave from global memory, the last column stage, the projection and
//    the first inverse column stage are one step on the same registers, and the last inverse row stage writes dpsi.  At
//    two stages a side the plane crosses shared memory six times each way instead of eleven.
//  * Consecutive threads take consecutive columns in the column stages and consecutive rows (odd pitch) in the inner row
//    stages, so shared memory is free of bank conflicts whatever the lengths; the ends take consecutive samples of a
//    row, as global memory wants it.
//  * Index divisions are multiplications by reciprocals made on the host.
//
// Bound by shared-memory wavefronts and issue together (FP32 120 x 112: 70 and 56 %; FP64 100 x 90, one CTA an SM: 56 and 35 %,
// FP64 pipe 36 %), not by HBM.  Against the run-time Stockham plan (one 512-thread CTA per SM, its per-stage arrays in local
// memory, a run-time modulo per twiddle), 3,180 positions of 120 x 112: 5.76 -> 0.39 ms per FP32 pass, 7 -> 110 Gpixel/s;
// 3,600 of 100 x 100 in FP64 3.21 -> 0.70.
#pragma once

#include "engine.h"
#include "project.cuh"
#include "regdft.cuh"

namespace cubo {

template <typename T> constexpr int kAnyThreads = sizeof(T) == 4 ? 1024 : 512;  // most threads of a CTA: 64 / 128 registers
constexpr int kAnyStages = 12;

// Exact i / d for i, d < 65536 as umulhi(i, ceil(2^32 / d)); d = 1 has no 32-bit reciprocal and is told by 0.
struct Divisor {
    unsigned d, m;
};
__host__ __device__ inline Divisor divisor(int d) {
    return Divisor{(unsigned)d, d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0u};
}
__device__ __forceinline__ int quotient(int i, const Divisor &v) {
    return v.m ? (int)__umulhi((unsigned)i, v.m) : i;
}

struct AnyLine {
    int L, stages;
    int r[kAnyStages];        // radix of each stage
    int before[kAnyStages];   // r_1 .. r_{i-1}
    Divisor sub[kAnyStages];  // L / (r_1 .. r_i)
};

template <typename T>
struct AnyPassArgs {
    PositionPassArgs<T> p;
    AnyLine rows, columns;   // the line of `rows` samples (along a column) and of `columns` samples (along a row)
    Divisor by_rows, by_columns;
    int pitch;
};

__device__ __forceinline__ int awrap(int v, int size) { return v < 0 ? v + size : (v >= size ? v - size : v); }

// The frequency slot e of a transformed line holds: e = sum q_i sub_i, k = sum q_i r_1 .. r_{i-1}.
static __device__ int slot_frequency(const AnyLine &l, int e) {
    int k = 0;
    for (int i = 0; i < l.stages; i++) {
        const int q = quotient(e, l.sub[i]);
        e -= q * (int)l.sub[i].d;
        k += q * l.before[i];
    }
    return k;
}

// x[q] *= W_B^{jq} (conjugate when INV); step = L / B, tw = W_L^t
template <typename T, bool INV, int R>
__device__ __forceinline__ void twiddle(C2<T> (&x)[R], int j, int step, const C2<T> *tw) {
    const int e = j * step;
#pragma unroll
    for (int q = 1; q < R; q++) x[q] = regdft::turn<C2<T>, INV>(x[q], tw[q * e]);
}

// An inner stage of every line: lines `line` apart, samples `elem` apart, stage s of plan l, whose twiddles are powers of
// W_B = tw[scale] (B the stage's block).
template <typename T, bool INV, int R>
__device__ __forceinline__ void inner_stage(C2<T> *D, const AnyLine &l, int s, int scale, const Divisor &lines,
                                            int line, int elem, const C2<T> *tw) {
    const int sub = (int)l.sub[s].d, block = sub * R, total = (int)lines.d * (l.L / R);
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int b = quotient(i, lines), ln = i - b * (int)lines.d;
        const int blk = quotient(b, l.sub[s]), j = b - blk * sub;
        C2<T> *x0 = D + ln * line + (blk * block + j) * elem;
        const int step = sub * elem;
        C2<T> x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = x0[r * step];
        if (INV) {
            if (sub > 1) twiddle<T, true, R>(x, j, scale, tw);  // blocks of one sample each have none
            regdft::dft<T, true, R>(x);
        } else {
            regdft::dft<T, false, R>(x);
            if (sub > 1) twiddle<T, false, R>(x, j, scale, tw);
        }
#pragma unroll
        for (int r = 0; r < R; r++) x0[r * step] = x[r];
    }
}

// The first row stage, from the exit wave S O[patch] (Ptychography.swift:321-336).
template <typename T, int R>
__device__ __forceinline__ void first_stage(C2<T> *D, const AnyPassArgs<T> &g, int rr, int cc, const C2<T> *S,
                                            const C2<T> *tw) {
    const PositionPassArgs<T> &a = g.p;
    const Divisor per = g.columns.sub[0];
    const int sub = (int)per.d, total = a.rows * sub;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int row = quotient(i, per), j = i - row * sub;
        const C2<T> *orow = a.object + (size_t)awrap(rr + corner_offset(row, a.rows), a.object_rows) * a.object_columns;
        const C2<T> *s = S + row * a.columns + j;
        C2<T> x[R], o[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            x[r] = s[r * sub];
            o[r] = orow[awrap(cc + corner_offset(j + r * sub, a.columns), a.object_columns)];
        }
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = regdft::turn<C2<T>, false>(x[r], o[r]);
        regdft::dft<T, false, R>(x);
        if (sub > 1) twiddle<T, false, R>(x, j, 1, tw);
        C2<T> *y = D + row * g.pitch + j;
#pragma unroll
        for (int q = 0; q < R; q++) y[q * sub] = x[q];
    }
}

// The last inverse row stage, into dpsi.
template <typename T, int R>
__device__ __forceinline__ void last_stage(const C2<T> *D, const AnyPassArgs<T> &g, C2<T> *out, const C2<T> *tw) {
    const PositionPassArgs<T> &a = g.p;
    const Divisor per = g.columns.sub[0];
    const int sub = (int)per.d, total = a.rows * sub;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int row = quotient(i, per), j = i - row * sub;
        const C2<T> *y = D + row * g.pitch + j;
        C2<T> x[R];
#pragma unroll
        for (int q = 0; q < R; q++) x[q] = y[q * sub];
        if (sub > 1) twiddle<T, true, R>(x, j, 1, tw);
        regdft::dft<T, true, R>(x);
        C2<T> *o = out + row * a.columns + j;
#pragma unroll
        for (int r = 0; r < R; r++) o[r * sub] = x[r];
    }
}

// The last column stage (blocks of R adjacent slots, no twiddle), the projection (Ptychography.swift:338-349) and the
// first inverse column stage; returns this thread's squared residual.
template <typename T, int R>
__device__ __forceinline__ double centre_stage(C2<T> *D, const AnyPassArgs<T> &g, const float *A,
                                               const unsigned short *kr0, const unsigned short *kc) {
    const PositionPassArgs<T> &a = g.p;
    const int blocks = a.rows / R, total = blocks * a.columns;
    const int step = blocks * a.columns;  // output q of a block is the frequency kr0 + q rows / R
    double err = 0;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int blk = quotient(i, g.by_columns), c = i - blk * a.columns;
        C2<T> *x0 = D + (blk * R) * g.pitch + c;
        const float *am = A + (int)kr0[blk] * a.columns + (int)kc[c];
        float measured[R];
#pragma unroll
        for (int q = 0; q < R; q++) measured[q] = am[q * step];
        C2<T> x[R];
#pragma unroll
        for (int r = 0; r < R; r++) x[r] = x0[r * g.pitch];
        regdft::dft<T, false, R>(x);
        project_values<T, R>(x, measured, a.inv_n, err);
        regdft::dft<T, true, R>(x);
#pragma unroll
        for (int r = 0; r < R; r++) x0[r * g.pitch] = x[r];
    }
    return err;
}

// Runs `f` with the radix as a compile-time constant.  WIDE adds the primes above 13.
template <int R>
struct Radix {
    static constexpr int value = R;
};
template <bool WIDE, typename F>
__device__ __forceinline__ void with_radix(int r, const F &f) {
    switch (r) {
        case 2: f(Radix<2>()); break;
        case 3: f(Radix<3>()); break;
        case 4: f(Radix<4>()); break;
        case 5: f(Radix<5>()); break;
        case 6: f(Radix<6>()); break;
        case 7: f(Radix<7>()); break;
        case 8: f(Radix<8>()); break;
        case 9: f(Radix<9>()); break;
        case 10: f(Radix<10>()); break;
        case 11: f(Radix<11>()); break;
        case 12: f(Radix<12>()); break;
        case 13: f(Radix<13>()); break;
        case 14: f(Radix<14>()); break;
        case 15: f(Radix<15>()); break;
        case 16: f(Radix<16>()); break;
        default:
            if constexpr (WIDE) {
                switch (r) {
                    case 17: f(Radix<17>()); break;
                    case 19: f(Radix<19>()); break;
                    case 23: f(Radix<23>()); break;
                    case 29: f(Radix<29>()); break;
                    default: f(Radix<31>()); break;
                }
            }
    }
}

template <typename T, bool WIDE>
__global__ void __launch_bounds__(kAnyThreads<T>, 1) any_pass_kernel(const __grid_constant__ AnyPassArgs<T> g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double scratch[kAnyThreads<T> / 32];
    const PositionPassArgs<T> &a = g.p;
    C2<T> *D = reinterpret_cast<C2<T> *>(smem_raw);
    C2<T> *twr = D + (size_t)a.rows * g.pitch;  // W_rows^t
    C2<T> *twc = twr + a.rows;                  // W_columns^t
    unsigned short *kr0 = reinterpret_cast<unsigned short *>(twc + a.columns);
    unsigned short *kc = kr0 + a.rows;
    const int tid = threadIdx.x, p = a.first + blockIdx.x;
    const int last = g.rows.r[g.rows.stages - 1], blocks = a.rows / last;
    for (int i = tid; i < a.rows; i += blockDim.x) twr[i] = a.tw_rows[i];
    for (int i = tid; i < a.columns; i += blockDim.x) {
        twc[i] = a.tw_columns[i];
        kc[i] = (unsigned short)slot_frequency(g.columns, i);
    }
    for (int i = tid; i < blocks; i += blockDim.x) kr0[i] = (unsigned short)slot_frequency(g.rows, i * last);
    const int rr = a.scan.rr[p], cc = a.scan.cc[p], cls = a.scan.cls[p];
    __syncthreads();
    with_radix<WIDE>(g.columns.r[0], [&](auto r) {
        first_stage<T, decltype(r)::value>(D, g, rr, cc, a.shifted + (size_t)cls * a.n, twc);
    });
    __syncthreads();
    for (int s = 1; s < g.columns.stages; s++) {
        with_radix<WIDE>(g.columns.r[s], [&](auto r) {
            inner_stage<T, false, decltype(r)::value>(D, g.columns, s, g.columns.before[s], g.by_rows, g.pitch, 1, twc);
        });
        __syncthreads();
    }
    for (int s = 0; s + 1 < g.rows.stages; s++) {
        with_radix<WIDE>(g.rows.r[s], [&](auto r) {
            inner_stage<T, false, decltype(r)::value>(D, g.rows, s, g.rows.before[s], g.by_columns, 1, g.pitch, twr);
        });
        __syncthreads();
    }
    double err = 0;
    with_radix<WIDE>(last, [&](auto r) {
        err = centre_stage<T, decltype(r)::value>(D, g, a.amplitudes + (size_t)p * a.n, kr0, kc);
    });
    __syncthreads();
    for (int s = g.rows.stages - 2; s >= 0; s--) {
        with_radix<WIDE>(g.rows.r[s], [&](auto r) {
            inner_stage<T, true, decltype(r)::value>(D, g.rows, s, g.rows.before[s], g.by_columns, 1, g.pitch, twr);
        });
        __syncthreads();
    }
    for (int s = g.columns.stages - 1; s >= 1; s--) {
        with_radix<WIDE>(g.columns.r[s], [&](auto r) {
            inner_stage<T, true, decltype(r)::value>(D, g.columns, s, g.columns.before[s], g.by_rows, g.pitch, 1, twc);
        });
        __syncthreads();
    }
    with_radix<WIDE>(g.columns.r[0], [&](auto r) {
        last_stage<T, decltype(r)::value>(D, g, a.dpsi + (size_t)p * a.n, twc);
    });
    // the position's squared residual, summed over the CTA in a fixed order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) err += __shfl_down_sync(0xffffffffu, err, o);
    if ((tid & 31) == 0) scratch[tid >> 5] = err;
    __syncthreads();
    if (tid == 0) {
        double total = 0;
        for (int w = 0; w < (int)blockDim.x / 32; w++) total += scratch[w];
        a.error[p] = total;
    }
}

// The fewest allowed factors whose product is L, the largest factor as small as possible, ascending; count 0: L has a
// prime factor above 31 (or does not fit the stages).
inline int best_factors(int L, int most, int *out) {
    static const int radices[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 19, 23, 29, 31};
    if (L < 2) return 0;
    for (int count = 1; count <= kAnyStages; count++) {
        // factors not above `cap`, the cap raised until the length splits into `count` of them
        for (int cap : radices) {
            if (cap > most) break;
            int f[kAnyStages], rest = L, depth = 0;
            int at[kAnyStages];  // index of the factor tried at each depth, descending
            at[0] = (int)(sizeof(radices) / sizeof(radices[0])) - 1;
            while (depth >= 0) {
                bool down = false;
                for (int &i = at[depth]; i >= 0; i--) {
                    const int r = radices[i];
                    if (r > cap || rest % r != 0) continue;
                    f[depth] = r;
                    if (depth + 1 == count) {
                        if (rest != r) continue;
                        for (int k = 0; k < count; k++) out[k] = f[count - 1 - k];  // ascending
                        return count;
                    }
                    rest /= r;
                    at[depth + 1] = i;
                    down = true;
                    break;
                }
                if (down) depth++;
                else {
                    depth--;
                    if (depth >= 0) { rest *= f[depth]; at[depth]--; }
                }
            }
        }
    }
    return 0;
}

// Ascending radices give the row ends (stage 1) the longest contiguous runs of global memory; the column lines take them
// descending, so that the centre step, which holds the amplitudes too, has the smallest.
inline bool plan_line(int L, int most, bool ascending, AnyLine *l) {
    int f[kAnyStages] = {};
    const int count = L == 1 ? 0 : best_factors(L, most, f);
    if (count == 0 && L != 1) return false;
    l->L = L;
    l->stages = count;
    int done = 1;
    for (int i = 0; i < count; i++) {
        l->r[i] = ascending ? f[i] : f[count - 1 - i];
        l->before[i] = done;
        done *= l->r[i];
        l->sub[i] = divisor(L / done);
    }
    return true;
}

using AnyKernelF = void (*)(AnyPassArgs<float>);
using AnyKernelD = void (*)(AnyPassArgs<double>);
// The instances with the primes above 13, each compiled in a file of its own (their unrolled prime DFTs take the
// compiler as long as the rest of the library).
AnyKernelF any_wide_f32();
AnyKernelD any_wide_f64();

}  // namespace cubo
