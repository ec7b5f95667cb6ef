// Small complex DFTs in registers for any radix up to 31, natural order in and out (sm_100a).
//
// Composite radices split once (R = A B, A-point DFTs, the twiddle W_R^{bc}, B-point DFTs); odd primes pair the samples
// k and R - k, so an R-point DFT costs (R - 1)^2 / 2 real-by-complex multiply-adds.  Every constant is cos / sin of
// 2 pi k / R evaluated at compile time and rounded to the nearest double (tests/test_regdft_constants.py).  Forward is e^{-2 pi i}, both directions unnormalised.
#pragma once

#include "common.cuh"

namespace cubo {
namespace regdft {

// cos and sin of 2 pi k / n, 0 <= k < n, rounded to the nearest double (compile time only): Taylor series on the first
// octant in pairs of doubles (T. J. Dekker, "A floating-point technique for extending the available precision", Numer.
// Math. 18, 1971), some 100 bits.  In plain double the sums' own roundings left half the constants of radix 8 and 16 one
// unit off, and a constant that is short acts on every plane as the same small gain: with them the errors of four mixed states
// of 128 x 128 were 1.4e-15 from 64 bits after four iterations, 3.4e-16 with these (objects 1.7e-16, 1.4e-16; four slices'
// errors 1.0e-15, 3.4e-16).
struct Pair {
    double hi, lo;
};
constexpr Pair two_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return Pair{s, (a - (s - t)) + (b - t)};
}
constexpr Pair two_product(double a, double b) {
    constexpr double kSplit = 134217729.0;  // 2^27 + 1
    const double ah = kSplit * a - (kSplit * a - a), al = a - ah, bh = kSplit * b - (kSplit * b - b), bl = b - bh;
    const double p = a * b;
    return Pair{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr Pair add(Pair a, Pair b) {
    const Pair s = two_sum(a.hi, b.hi);
    return two_sum(s.hi, s.lo + (a.lo + b.lo));
}
constexpr Pair multiply(Pair a, Pair b) {
    const Pair p = two_product(a.hi, b.hi);
    return two_sum(p.hi, p.lo + (a.hi * b.lo + a.lo * b.hi));
}
constexpr Pair divide(Pair a, int d) {
    const double q = a.hi / d;
    const Pair p = two_product(q, (double)d);
    return two_sum(q, (((a.hi - p.hi) - p.lo) + a.lo) / d);
}
// sum of (-1)^i x^(2 i + first) / (2 i + first)!, first = 0 (cosine) or 1 (sine)
constexpr double taylor(Pair x, int first) {
    const Pair square = multiply(x, x);
    Pair term = first ? x : Pair{1, 0}, sum = term;
    for (int i = 1; i < 16; i++) {
        term = divide(multiply(term, Pair{-square.hi, -square.lo}), (2 * i - 1 + first) * (2 * i + first));
        sum = add(sum, term);
    }
    return sum.hi;
}
// 2 pi k / n
constexpr Pair angle(int k, int n) {
    return divide(multiply(Pair{6.283185307179586, 2.4492935982947064e-16}, Pair{(double)k, 0}), n);
}
constexpr double turn_cos(int k, int n) {
    k %= n;
    if (2 * k > n) k = n - k;                              // cos(2 pi - a) = cos a
    if (4 * k > n) return -turn_cos(n - 2 * k, 2 * n);     // cos a = -cos(pi - a); the angle 2 pi (n - 2k) / (2n)
    return 8 * k > n ? taylor(angle(n - 4 * k, 4 * n), 1) : taylor(angle(k, n), 0);
}
constexpr double turn_sin(int k, int n) {
    k %= n;
    if (2 * k > n) return -turn_sin(n - k, n);
    if (4 * k > n) return turn_sin(n - 2 * k, 2 * n);      // sin a = sin(pi - a)
    return 8 * k > n ? taylor(angle(n - 4 * k, 4 * n), 0) : taylor(angle(k, n), 1);
}
template <int R>
struct Turns {
    double c[R], s[R];
    constexpr Turns() : c(), s() {
        for (int k = 0; k < R; k++) { c[k] = turn_cos(k, R); s[k] = turn_sin(k, R); }
    }
};

// Packed FP32x2 add / subtract / multiply-add (one instruction for both parts, each rounded as the scalar one).
__device__ __forceinline__ float2 add(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "add.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 sub(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// a * s + c with a real factor s
__device__ __forceinline__ float2 mad(float2 a, float s, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\tmov.b64 rc, {%5, %6};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(s), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 mad(double2 a, double s, double2 c) {
    return make_double2(fma(a.x, s, c.x), fma(a.y, s, c.y));
}

// a W forward, a conj(W) inverse
template <typename V, bool INV>
__device__ __forceinline__ V turn(V a, V w) {
    V r;
    if (INV) { r.x = a.x * w.x + a.y * w.y; r.y = a.y * w.x - a.x * w.y; }
    else { r.x = a.x * w.x - a.y * w.y; r.y = a.x * w.y + a.y * w.x; }
    return r;
}
template <typename V, bool INV>
__device__ __forceinline__ V quarter(V a) {  // a W_4
    V r;
    if (INV) { r.x = -a.y; r.y = a.x; } else { r.x = a.y; r.y = -a.x; }
    return r;
}

// The first factor A of the split R = A B (0: R is 2, 4 or an odd prime).
constexpr int split(int r) {
    return r == 6 ? 2 : r == 8 ? 2 : r == 9 ? 3 : r == 10 ? 2 : r == 12 ? 3 : r == 14 ? 2 : r == 15 ? 3 : r == 16 ? 4 : 0;
}

template <typename T, bool INV, int R>
__device__ __forceinline__ void dft(C2<T> (&x)[R]) {
    using V = C2<T>;
    if constexpr (R == 2) {
        const V a = x[0], b = x[1];
        x[0] = add(a, b);
        x[1] = sub(a, b);
    } else if constexpr (R == 4) {
        const V t0 = add(x[0], x[2]), t1 = sub(x[0], x[2]), t2 = add(x[1], x[3]), t3 = quarter<V, INV>(sub(x[1], x[3]));
        x[0] = add(t0, t2);
        x[2] = sub(t0, t2);
        x[1] = add(t1, t3);
        x[3] = sub(t1, t3);
    } else if constexpr (split(R) > 0) {
        constexpr int A = split(R), B = R / A;
        constexpr Turns<R> w;
        V y[B][A];
        // n = B a + b, k = c + A d: X[c + A d] = sum_b W_B^{bd} W_R^{bc} sum_a W_A^{ac} x[B a + b]
#pragma unroll
        for (int b = 0; b < B; b++) {
#pragma unroll
            for (int a = 0; a < A; a++) y[b][a] = x[B * a + b];
            dft<T, INV, A>(y[b]);
        }
#pragma unroll
        for (int c = 0; c < A; c++) {
            V z[B];
#pragma unroll
            for (int b = 0; b < B; b++) {
                const int e = b * c;  // < R
                if (e == 0) z[b] = y[b][c];
                else if (4 * e == R) z[b] = quarter<V, INV>(y[b][c]);
                else z[b] = turn<V, INV>(y[b][c], mk<T>((T)w.c[e], (T)-w.s[e]));
            }
            dft<T, INV, B>(z);
#pragma unroll
            for (int d = 0; d < B; d++) x[c + A * d] = z[d];
        }
    } else {
        constexpr int H = (R - 1) / 2;
        constexpr Turns<R> w;
        V p[H], m[H], sum = x[0];
#pragma unroll
        for (int k = 1; k <= H; k++) {
            p[k - 1] = add(x[k], x[R - k]);
            m[k - 1] = sub(x[k], x[R - k]);
        }
        const V x0 = x[0];
#pragma unroll
        for (int k = 0; k < H; k++) sum = add(sum, p[k]);
        x[0] = sum;
#pragma unroll
        for (int q = 1; q <= H; q++) {
            V u = x0, v = mk<T>(0, 0);
#pragma unroll
            for (int k = 1; k <= H; k++) {
                u = mad(p[k - 1], (T)w.c[(k * q) % R], u);
                v = mad(m[k - 1], (T)w.s[(k * q) % R], v);
            }
            v = quarter<V, INV>(v);  // -i v forward, +i v inverse
            x[q] = add(u, v);
            x[R - q] = sub(u, v);
        }
    }
}

}  // namespace regdft
}  // namespace cubo
