// The compile-time DFT constants of cubokit_b200/csrc/regdft.cuh, for tests/test_regdft_constants.py (host code only).
#include "regdft.cuh"

namespace {
template <int R>
void fill(double *c, double *s) {
    constexpr cubo::regdft::Turns<R> w;
    for (int k = 0; k < R; k++) {
        c[k] = w.c[k];
        s[k] = w.s[k];
    }
}
template <int R>
int find(int radix, double *c, double *s) {
    if (radix == R) return fill<R>(c, s), 0;
    if constexpr (R < 31) return find<R + 1>(radix, c, s);
    return 1;
}
}  // namespace

// cos and sin of 2 pi k / radix, 0 <= k < radix; 1: the radix is not one of 2 .. 31.
extern "C" int turns(int radix, double *c, double *s) { return find<2>(radix, c, s); }
