// The Fourier-modulus projection of far-field values (Ptychography.swift:338-349): f becomes (A / |f| - 1) f / n, the
// residual of giving f the measured modulus A, with the squared error (A - |f|)^2 summed; a zero value becomes A / n.
//
// |f| and A / |f| from one reciprocal square root r of |f|^2, each corrected by the residual of its FMA (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990): with
// g = |f|^2 r, |f| = g + (|f|^2 - g g) r / 2, and with t = A r, A / |f| = t + (A - t |f|) r, for an eighth of the square root's
// and the division's instructions.  The residuals carry their own rounding, so a result whose exact value lies next to the middle
// of two numbers can come out as the other one: none of 3.4e7 values of either type did, and tests/test_gpu_project.py holds
// them to one unit in the last place, in at most 1 % of the values.  The general functions were a fifth of the passes; ms per pass before and after: FP32 120 x
// 112 0.534 -> 0.435 and 64 x 64 0.109 -> 0.089 (3,600 positions), 256 x 256 2.51 -> 2.24 (4,096), 128 x 128 2.135 -> 1.79
// (16,384), FP64 100 x 100 0.978 -> 0.696.  Powers outside [1e-30, 1e30] (1e-280, 1e280), where r or a residual leaves the
// normal range, not finite ones and zeros take the general functions, decided for all R values of a thread at once.
#pragma once

#include "common.cuh"

namespace cubo {

template <typename T> struct ProjectRange;
template <> struct ProjectRange<float> { static constexpr float low = 1e-30f, high = 1e30f, measured = 1e20f; };
template <> struct ProjectRange<double> { static constexpr double low = 1e-280, high = 1e280, measured = 1e100; };

template <typename T>
__device__ __forceinline__ bool modulus_in_range(T power, T measured) {
    using L = ProjectRange<T>;
    return power > L::low && power < L::high && measured < L::measured;
}

// |f| and measured / |f| of a power in range.
__device__ __forceinline__ void modulus_and_ratio(float power, float measured, float &modulus, float &ratio) {
    const float r = rsqrtf(power), g = power * r, t = measured * r;
    modulus = fmaf(fmaf(-g, g, power), 0.5f * r, g);
    ratio = fmaf(fmaf(-t, modulus, measured), r, t);
}
__device__ __forceinline__ void modulus_and_ratio(double power, double measured, double &modulus, double &ratio) {
    const double r = rsqrt(power), g = power * r, t = measured * r;
    modulus = fma(fma(-g, g, power), 0.5 * r, g);
    ratio = fma(fma(-t, modulus, measured), r, t);
}

template <typename T, int R>
__device__ __forceinline__ void project_values(C2<T> (&x)[R], const float (&measured)[R], T inv_n, double &err) {
    T power[R];
    bool plain = true;
#pragma unroll
    for (int i = 0; i < R; i++) {
        power[i] = x[i].x * x[i].x + x[i].y * x[i].y;
        plain = plain && modulus_in_range<T>(power[i], (T)measured[i]);
    }
    if (plain) {
#pragma unroll
        for (int i = 0; i < R; i++) {
            T modulus, ratio;
            modulus_and_ratio(power[i], (T)measured[i], modulus, ratio);
            const T miss = (T)measured[i] - modulus;
            err += (double)(miss * miss);
            const T s = (ratio - (T)1) * inv_n;
            x[i].x *= s;
            x[i].y *= s;
        }
        return;
    }
#pragma unroll 1
    for (int i = 0; i < R; i++) {
        // (dynamic indices would put the arrays in local memory: select)
        C2<T> f = x[0];
        T want = (T)measured[0];
#pragma unroll
        for (int k = 1; k < R; k++)
            if (k == i) { f = x[k]; want = (T)measured[k]; }
        const T mag = sqrt(f.x * f.x + f.y * f.y);
        const T miss = want - mag;
        err += (double)(miss * miss);
        if (mag > (T)0) {
            const T s = (want / mag - (T)1) * inv_n;
            f.x *= s;
            f.y *= s;
        } else {
            f = mk<T>(want * inv_n, (T)0);
        }
#pragma unroll
        for (int k = 0; k < R; k++)
            if (k == i) x[k] = f;
    }
}

// The mixed states' common factor of a pixel of summed intensity `power`, (A / sqrt(power) - 1) / n, and its squared error;
// a zero intensity has factor 0 and adds an infinite term or, on request, A^2 (PtychographyEngines.swift:188-195).
__device__ __forceinline__ double mixed_factor(double power, double measured, double inv_n, bool zero_infinite,
                                               double &err) {
    double modulus, ratio;
    if (modulus_in_range<double>(power, measured)) {
        modulus_and_ratio(power, measured, modulus, ratio);
    } else {
        modulus = sqrt(power);
        if (modulus == 0.0) {
            err += zero_infinite ? __longlong_as_double(0x7ff0000000000000ll) : measured * measured;
            return 0.0;
        }
        ratio = measured / modulus;
    }
    err += (measured - modulus) * (measured - modulus);
    return (ratio - 1.0) * inv_n;
}

}  // namespace cubo
