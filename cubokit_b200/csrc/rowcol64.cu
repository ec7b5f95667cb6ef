// FP64 planes as row and column launches through global memory, for every FP64 engine whose planes do not stay in one CTA
// (sm_100a): the single-slice pass above 12,288 pixels, the far fields of position correction, the mixed states and the
// multislice propagation, for detectors whose sides have no prime factor above 13.
//
//   rows forward   nl rows of one plane: the input (a shifted probe by class, or a wave or residual by position) times the
//                  object patch (or its conjugate, optionally a row or a column further), transformed along the row
//   columns        nl columns of one position: forward column transforms of its planes, the pointwise step, inverse column
//                  transforms.  The step is the modulus projection of one plane, the summed-intensity projection of the
//                  mixed states' planes, a separable Fresnel propagator, or (no inverse, nothing written back) the normal
//                  equations of position correction from three planes
//   rows inverse   the inverse row transforms; multislice joins them with the next slice's forward rows (rc_through_kernel)
//
// Line transforms as in the any-size pass (anypass.cuh): in-place stages in registers, the first stage of a launch read from
// and the last written to global memory, so a line of two stages crosses shared memory once each way.  128 has its
// geometry (8 x 16) at compile time, other lengths the run-time plan.  Sums over a CTA and over a position's CTAs have a
// fixed order.
//
// Each launch reads and writes a plane once (96 n bytes a transform pair, against 32 n for a plane that stays on chip), yet it
// is quicker than the clustered launch that kept a 128 x 128 plane in two SMs and exchanged halves between them: there one
// CTA an SM loaded, transformed and stored in turn, with HBM busy 15 % of the time; here two to six CTAs an SM overlap those.
// 1,600 positions of 128 x 128, per iteration: four mixed states 3.5 -> 2.0 ms (their columns meet in one CTA, so the summed
// projection needs no factor plane and no launch of its own), four slices forward 2.6 -> 1.84 and back 1.87 -> 1.38 ms; the
// three far fields and normal equations of 2,304 positions 2.7 -> 1.15 ms (the third field's columns end in the equations'
// sums, which no field is written for).  Rows run at 4.6 TB/s, single columns at 4.5.  No unit is full: FP64 pipe 19 to 42 %,
// LSU wavefronts 38 to 58, HBM 30 to 60; at 88 to 128 registers two CTAs fit an SM (22 % of its warps), and each one's phases
// follow one another.  Against the batched line transforms, which the generic variant, longer primes and sides up to 16 keep:
// four slices of 980 positions of 96 x 96 58 -> 17 ms per seven iterations, two mixed states of 1,035 14.9 -> 4.7 per six.
#include <algorithm>
#include <type_traits>

#include "anypass.cuh"
#include "position_step.cuh"

namespace cubo {

namespace {

constexpr int kRcThreads = 256;
// complex128 values of the lines one CTA holds, where the line allows it: eight a thread, 32 KB, so that registers and not
// shared memory set the CTAs an SM
constexpr int kRcValues = 2048;
constexpr size_t kRcSmem = 200 * 1024;

enum { kRcProject, kRcPropagate, kRcMixed, kRcSolve };

struct RcArgs {
    int rows, columns, n, object_rows, object_columns;
    int first;                            // the launch's first position
    ScanTables scan;
    AnyLine line;                         // of the launch's lines
    Divisor by_nl, by_block[kAnyStages];  // lines per CTA; blocks of a line, L / r, of each stage
    int nl, per;                          // lines per CTA, CTAs per plane
    const double2 *tw;                    // W_L^t
    // rows: plane (position p, layer y) is read at in + y in_layer + (class or p) n and written at
    // out + y out_layer + (p - out_first) out_stride
    const double2 *in;
    int by_class;
    long long in_layer;
    const double2 *object, *object_after; // null: no factor; object_after: position correction, whose layers are the object
    int conj_object;                      // before the update at the centre, after it a row and after it a column further
    double2 *out;                         // (columns: the planes in place)
    double2 *next;                        // rows through: the next spectrum, laid out by position
    const double2 *from;                  // rows inverse: the spectrum, by position (null: out itself)
    long long out_layer, out_stride;
    int out_first;
    int layers;
    // columns
    const float *amplitudes;
    double inv_n;
    double *error;                        // [position][per]
    const double2 *prop_rows, *prop_columns;
    int conj_prop, zero_infinite;
    double *terms;                        // [position - out_first][per][5]
};

__device__ __forceinline__ int rc_wrap(int v, int size) { return v < 0 ? v + size : (v >= size ? v - size : v); }

// A line's plan, at run time or as RA x RB at compile time.  `padded` places sample e of a row in shared memory with
// blocks of the last radix padded to an odd length; base(K) is the block that holds frequency K.
struct RunTimeLine {
    const RcArgs &g;
    const unsigned short *blocks_of;
    __device__ int length() const { return g.line.L; }
    __device__ int last() const { return g.line.r[g.line.stages - 1]; }
    __device__ int sub() const { return (int)g.line.sub[0].d; }
    __device__ int by_sub(int i) const { return quotient(i, g.line.sub[0]); }
    __device__ int blocks() const { return (int)g.by_block[g.line.stages - 1].d; }
    __device__ int by_blocks(int i) const { return quotient(i, g.by_block[g.line.stages - 1]); }
    __device__ int padded(int e) const {
        return (last() & 1) ? e : e + quotient(e, g.line.sub[g.line.stages - 2]);
    }
    __device__ int base(int K) const { return blocks_of[K]; }
    __device__ int lines() const { return g.nl; }
    __device__ int by_lines(int i) const { return quotient(i, g.by_nl); }
    template <typename F> __device__ void outer(const F &f) const { with_radix<false>(g.line.r[0], f); }
    template <typename F> __device__ void inner_most(const F &f) const { with_radix<false>(last(), f); }
    template <typename F> __device__ void between(bool inverse, const F &f) const {
        const int m = g.line.stages;
        for (int i = 1; i + 1 < m; i++) {
            const int s = inverse ? m - 1 - i : i;
            with_radix<false>(g.line.r[s], [&](auto r) { f(r, s); });
            __syncthreads();
        }
    }
};
template <int RA, int RB, int NL>
struct FixedLine {
    static_assert(RB % 2 == 0, "one pad a block");
    const RcArgs &g;
    const unsigned short *blocks_of;
    __device__ int length() const { return RA * RB; }
    __device__ int last() const { return RB; }
    __device__ int sub() const { return RB; }
    __device__ int by_sub(int i) const { return i / RB; }
    __device__ int blocks() const { return RA; }
    __device__ int by_blocks(int i) const { return i / RA; }
    __device__ int padded(int e) const { return e + e / RB; }
    __device__ int base(int K) const { return K; }
    __device__ int lines() const { return NL; }
    __device__ int by_lines(int i) const { return i / NL; }
    template <typename F> __device__ void outer(const F &f) const { f(Radix<RA>()); }
    template <typename F> __device__ void inner_most(const F &f) const { f(Radix<RB>()); }
    template <typename F> __device__ void between(bool, const F &) const {}
};

// The middle stages of a row line in shared memory (run-time plans of three stages and more).
template <bool INV, typename Line>
__device__ __forceinline__ void rows_between(const Line &l, double2 *D, int rows, int pitch, const double2 *tw) {
    l.between(INV, [&](auto rc, int s) {
        constexpr int R = decltype(rc)::value;
        const AnyLine &a = l.g.line;
        const int sub = (int)a.sub[s].d, step = l.padded(sub), blocks = (int)l.g.by_block[s].d;
        for (int i = threadIdx.x; i < rows * blocks; i += kRcThreads) {
            const int row = quotient(i, l.g.by_block[s]), b = i - row * blocks;
            const int blk = quotient(b, a.sub[s]), j = b - blk * sub;
            double2 *y = D + row * pitch + l.padded(blk * sub * R + j);
            double2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[r * step];
            if (INV) twiddle<double, true, R>(x, j, a.before[s], tw);
            regdft::dft<double, INV, R>(x);
            if (!INV) twiddle<double, false, R>(x, j, a.before[s], tw);
#pragma unroll
            for (int r = 0; r < R; r++) y[r * step] = x[r];
        }
    });
}

template <typename Line, bool INV>
__global__ void __launch_bounds__(kRcThreads, 2) rc_rows_kernel(const __grid_constant__ RcArgs g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *D = reinterpret_cast<double2 *>(smem_raw);
    const Line shape{g, nullptr};
    const int L = shape.length(), nb = shape.blocks(), rl = shape.last() | 1, pitch = nb * rl;
    double2 *tw = D + (size_t)shape.lines() * pitch;
    unsigned short *blocks_of = reinterpret_cast<unsigned short *>(tw + L);
    const Line l{g, blocks_of};
    // a position's layers follow one another: they share its input or its object patch in L2
    const int plane = (int)(blockIdx.x / g.per), r0 = (int)(blockIdx.x % g.per) * l.lines();
    const int p = g.first + plane / g.layers, layer = plane % g.layers;
    const int rows = min(l.lines(), g.rows - r0);
    for (int i = threadIdx.x; i < L; i += kRcThreads) tw[i] = g.tw[i];
    for (int b = threadIdx.x; b < nb; b += kRcThreads) blocks_of[slot_frequency(g.line, b * l.last())] = (unsigned short)b;
    double2 *out = g.out + layer * g.out_layer + (long long)(p - g.out_first) * g.out_stride + (size_t)r0 * L;
    const double2 *in = INV ? (g.from ? g.from + (long long)p * g.n + (size_t)r0 * L : out)
                            : g.in + layer * g.in_layer +
                                        (size_t)(g.by_class ? g.scan.cls[p] : p) * g.n + (size_t)r0 * L;
    __syncthreads();
    if constexpr (!INV) {
        const double2 *object = g.object_after && layer > 0 ? g.object_after : g.object;
        const int rr = object ? g.scan.rr[p] + (g.object_after && layer == 1) : 0;
        const int cc = object ? g.scan.cc[p] + (g.object_after && layer == 2) : 0;
        l.outer([&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int sub = l.sub(), step = l.padded(sub);
            for (int i = threadIdx.x; i < rows * sub; i += kRcThreads) {
                const int row = l.by_sub(i), j = i - row * sub;
                const double2 *s = in + (size_t)row * L + j;
                double2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = s[r * sub];
                if (object) {
                    const double2 *orow = object + (size_t)rc_wrap(rr + corner_offset(r0 + row, g.rows), g.object_rows) *
                                                       g.object_columns;
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        double2 o = orow[rc_wrap(cc + corner_offset(j + r * sub, L), g.object_columns)];
                        if (g.conj_object) o.y = -o.y;
                        x[r] = cmul(x[r], o);
                    }
                }
                regdft::dft<double, false, R>(x);
                twiddle<double, false, R>(x, j, 1, tw);
                double2 *y = D + row * pitch + l.padded(j);
#pragma unroll
                for (int r = 0; r < R; r++) y[r * step] = x[r];
            }
        });
        __syncthreads();
        rows_between<false>(l, D, rows, pitch, tw);
        l.inner_most([&](auto rc) {
            constexpr int R = decltype(rc)::value;
            for (int i = threadIdx.x; i < rows * nb; i += kRcThreads) {
                const int row = l.by_blocks(i), K = i - row * nb;
                const double2 *y = D + row * pitch + l.base(K) * rl;
                double2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = y[r];
                regdft::dft<double, false, R>(x);
                double2 *o = out + (size_t)row * L + K;
#pragma unroll
                for (int r = 0; r < R; r++) o[r * nb] = x[r];
            }
        });
    } else {
        l.inner_most([&](auto rc) {
            constexpr int R = decltype(rc)::value;
            for (int i = threadIdx.x; i < rows * nb; i += kRcThreads) {
                const int row = l.by_blocks(i), K = i - row * nb;
                const double2 *o = in + (size_t)row * L + K;
                double2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = o[r * nb];
                regdft::dft<double, true, R>(x);
                double2 *y = D + row * pitch + l.base(K) * rl;
#pragma unroll
                for (int r = 0; r < R; r++) y[r] = x[r];
            }
        });
        __syncthreads();
        rows_between<true>(l, D, rows, pitch, tw);
        l.outer([&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int sub = l.sub(), step = l.padded(sub);
            for (int i = threadIdx.x; i < rows * sub; i += kRcThreads) {
                const int row = l.by_sub(i), j = i - row * sub;
                const double2 *y = D + row * pitch + l.padded(j);
                double2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = y[r * step];
                twiddle<double, true, R>(x, j, 1, tw);
                regdft::dft<double, true, R>(x);
                double2 *o = out + (size_t)row * L + j;
#pragma unroll
                for (int r = 0; r < R; r++) o[r * sub] = x[r];
            }
        });
    }
}

// Multislice, between two slices: the inverse rows of one (whose wave or residual is written to out) and, while a row's samples
// are in registers, their product with the object patch and the next slice's forward rows (written to next).  The last stage of
// the one and the first of the other hold the same samples in the same thread.  `in` may be out or next.  A plane is read once
// and written twice in place of two of each: four slices of 1,600 positions of 128 x 128, an iteration, forward 2.08 -> 1.84 ms,
// back 1.55 -> 1.38.
template <typename Line>
__global__ void __launch_bounds__(kRcThreads, 2) rc_through_kernel(const __grid_constant__ RcArgs g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *D = reinterpret_cast<double2 *>(smem_raw);
    const Line shape{g, nullptr};
    const int L = shape.length(), nb = shape.blocks(), rl = shape.last() | 1, pitch = nb * rl;
    double2 *tw = D + (size_t)shape.lines() * pitch;
    unsigned short *blocks_of = reinterpret_cast<unsigned short *>(tw + L);
    const Line l{g, blocks_of};
    const int p = g.first + (int)(blockIdx.x / g.per), r0 = (int)(blockIdx.x % g.per) * l.lines();
    const int rows = min(l.lines(), g.rows - r0);
    for (int i = threadIdx.x; i < L; i += kRcThreads) tw[i] = g.tw[i];
    for (int b = threadIdx.x; b < nb; b += kRcThreads) blocks_of[slot_frequency(g.line, b * l.last())] = (unsigned short)b;
    const long long at = (long long)p * g.n + (size_t)r0 * L;
    const double2 *in = g.in + at;
    double2 *out = g.out + at, *next = g.next + at;
    const int rr = g.scan.rr[p], cc = g.scan.cc[p];
    __syncthreads();
    l.inner_most([&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = threadIdx.x; i < rows * nb; i += kRcThreads) {
            const int row = l.by_blocks(i), K = i - row * nb;
            const double2 *o = in + (size_t)row * L + K;
            double2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = o[r * nb];
            regdft::dft<double, true, R>(x);
            double2 *y = D + row * pitch + l.base(K) * rl;
#pragma unroll
            for (int r = 0; r < R; r++) y[r] = x[r];
        }
    });
    __syncthreads();
    rows_between<true>(l, D, rows, pitch, tw);
    l.outer([&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int sub = l.sub(), step = l.padded(sub);
        for (int i = threadIdx.x; i < rows * sub; i += kRcThreads) {
            const int row = l.by_sub(i), j = i - row * sub;
            double2 *y = D + row * pitch + l.padded(j);
            double2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[r * step];
            twiddle<double, true, R>(x, j, 1, tw);
            regdft::dft<double, true, R>(x);
            double2 *o = out + (size_t)row * L + j;
            const double2 *orow = g.object + (size_t)rc_wrap(rr + corner_offset(r0 + row, g.rows), g.object_rows) *
                                                 g.object_columns;
#pragma unroll
            for (int r = 0; r < R; r++) {
                o[r * sub] = x[r];
                double2 f = orow[rc_wrap(cc + corner_offset(j + r * sub, L), g.object_columns)];
                if (g.conj_object) f.y = -f.y;
                x[r] = cmul(x[r], f);
            }
            regdft::dft<double, false, R>(x);
            twiddle<double, false, R>(x, j, 1, tw);
#pragma unroll
            for (int r = 0; r < R; r++) y[r * step] = x[r];
        }
    });
    __syncthreads();
    rows_between<false>(l, D, rows, pitch, tw);
    l.inner_most([&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = threadIdx.x; i < rows * nb; i += kRcThreads) {
            const int row = l.by_blocks(i), K = i - row * nb;
            const double2 *y = D + row * pitch + l.base(K) * rl;
            double2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = y[r];
            regdft::dft<double, false, R>(x);
            double2 *o = next + (size_t)row * L + K;
#pragma unroll
            for (int r = 0; r < R; r++) o[r * nb] = x[r];
        }
    });
}

// The columns of one position: plane y's sample e of column c at D[(y L + e) lines + c].
template <typename Line, int MODE>
__global__ void __launch_bounds__(kRcThreads, 2) rc_columns_kernel(const __grid_constant__ RcArgs g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double scratch[5][kRcThreads / 32];
    double2 *D = reinterpret_cast<double2 *>(smem_raw);
    const Line shape{g, nullptr};
    const int L = shape.length(), C = g.columns, nl = shape.lines(), nb = shape.blocks();
    const int layers = MODE == kRcMixed ? g.layers : MODE == kRcSolve ? 3 : 1;
    const int threads = MODE == kRcProject || MODE == kRcPropagate ? kRcThreads : (int)blockDim.x;
    double2 *tw = D + (size_t)layers * L * nl;
    unsigned short *freq = reinterpret_cast<unsigned short *>(tw + L);  // frequency of output 0 of each last block
    const Line l{g, freq};
    const int p = g.first + (int)(blockIdx.x / g.per), part = (int)(blockIdx.x % g.per), c0 = part * nl;
    const int lines = min(nl, C - c0);
    double2 *io = g.out + (long long)(p - g.out_first) * g.out_stride + c0;
    const float *A = MODE == kRcPropagate ? nullptr : g.amplitudes + (size_t)p * g.n + c0;
    for (int i = threadIdx.x; i < L; i += threads) {
        tw[i] = g.tw[i];
        if (MODE != kRcPropagate) asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (size_t)i * C));
    }
    for (int b = threadIdx.x; b < nb; b += threads) freq[b] = (unsigned short)slot_frequency(g.line, b * l.last());
    __syncthreads();
    l.outer([&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int sub = l.sub();
        for (int i = threadIdx.x; i < layers * nl * sub; i += threads) {  // (layer, sample, column)
            const int e = l.by_lines(i), c = i - e * nl, y = layers > 1 ? l.by_sub(e) : 0, j = e - y * sub;
            if (c >= lines) continue;
            const double2 *o = io + y * g.out_layer + (size_t)j * C + c;
            double2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = o[(size_t)r * sub * C];
            regdft::dft<double, false, R>(x);
            twiddle<double, false, R>(x, j, 1, tw);
            double2 *z = D + ((size_t)y * L + j) * nl + c;
#pragma unroll
            for (int r = 0; r < R; r++) z[r * sub * nl] = x[r];
        }
    });
    __syncthreads();
    for (int y = 0; y < layers; y++)
        l.between(false, [&](auto rc, int s) {
            inner_stage<double, false, decltype(rc)::value>(D + (size_t)y * L * nl, g.line, s, g.line.before[s], g.by_nl, 1,
                                                            nl, tw);
        });
    double sums[5] = {0, 0, 0, 0, 0};  // [0]: the squared residual; all five: the normal equations
    l.inner_most([&](auto rc) {
        constexpr int R = decltype(rc)::value;
        for (int i = threadIdx.x; i < nl * nb; i += threads) {
            const int b = l.by_lines(i), c = i - b * nl;
            if (c >= lines) continue;
            double2 *z = D + b * R * nl + c;
            const int kr = freq[b];
            float measured[R];
            if (MODE != kRcPropagate) {
                const float *am = A + (size_t)kr * C + c;
#pragma unroll
                for (int q = 0; q < R; q++) measured[q] = am[(size_t)q * nb * C];
            }
            if constexpr (MODE == kRcSolve) {
                double2 f[R], x[R];
                double dx[R];
#pragma unroll
                for (int r = 0; r < R; r++) f[r] = z[r * nl];
                regdft::dft<double, false, R>(f);
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = z[(r + L) * nl];
                regdft::dft<double, false, R>(x);
#pragma unroll
                for (int r = 0; r < R; r++) dx[r] = 2 * ((f[r].x - x[r].x) * f[r].x + (f[r].y - x[r].y) * f[r].y);
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = z[(r + 2 * L) * nl];
                regdft::dft<double, false, R>(x);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const double want = (double)measured[r];
                    position_products(dx[r], 2 * ((f[r].x - x[r].x) * f[r].x + (f[r].y - x[r].y) * f[r].y),
                                      want * want - (f[r].x * f[r].x + f[r].y * f[r].y), sums);
                }
            } else if constexpr (MODE == kRcMixed) {
                double power[R];
#pragma unroll
                for (int r = 0; r < R; r++) power[r] = 0;
                for (int y = 0; y < layers; y++) {
                    double2 *zy = z + (size_t)y * L * nl;
                    double2 x[R];
#pragma unroll
                    for (int r = 0; r < R; r++) x[r] = zy[r * nl];
                    regdft::dft<double, false, R>(x);
#pragma unroll
                    for (int r = 0; r < R; r++) {
                        power[r] += x[r].x * x[r].x + x[r].y * x[r].y;
                        zy[r * nl] = x[r];
                    }
                }
#pragma unroll
                for (int r = 0; r < R; r++)  // the factor takes the intensity's place
                    power[r] = mixed_factor(power[r], (double)measured[r], g.inv_n, g.zero_infinite != 0, sums[0]);
                for (int y = 0; y < layers; y++) {
                    double2 *zy = z + (size_t)y * L * nl;
                    double2 x[R];
#pragma unroll
                    for (int r = 0; r < R; r++) x[r] = cscale(zy[r * nl], power[r]);
                    regdft::dft<double, true, R>(x);
#pragma unroll
                    for (int r = 0; r < R; r++) zy[r * nl] = x[r];
                }
            } else {
                double2 x[R];
#pragma unroll
                for (int r = 0; r < R; r++) x[r] = z[r * nl];
                regdft::dft<double, false, R>(x);
                if constexpr (MODE == kRcProject) {
                    project_values<double, R>(x, measured, g.inv_n, sums[0]);
                } else {
                    double2 wc = g.prop_columns[c0 + c];
                    wc.x *= g.inv_n;
                    wc.y *= g.conj_prop ? -g.inv_n : g.inv_n;
#pragma unroll
                    for (int q = 0; q < R; q++) {
                        double2 wr = g.prop_rows[kr + q * nb];
                        if (g.conj_prop) wr.y = -wr.y;
                        x[q] = cmul(x[q], cmul(wr, wc));
                    }
                }
                regdft::dft<double, true, R>(x);
#pragma unroll
                for (int r = 0; r < R; r++) z[r * nl] = x[r];
            }
        }
    });
    constexpr int kSums = MODE == kRcSolve ? 5 : MODE == kRcPropagate ? 0 : 1;
    if constexpr (kSums > 0) {  // over the CTA in a fixed order
#pragma unroll
        for (int q = 0; q < kSums; q++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sums[q] += __shfl_down_sync(0xffffffffu, sums[q], o);
            if ((threadIdx.x & 31) == 0) scratch[q][threadIdx.x >> 5] = sums[q];
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < kSums) {
        double total = 0;
        for (int w = 0; w < threads / 32; w++) total += scratch[threadIdx.x][w];
        if (MODE == kRcSolve) g.terms[((long long)(p - g.out_first) * g.per + part) * 5 + threadIdx.x] = total;
        else g.error[(long long)p * g.per + part] = total;
    }
    if constexpr (MODE == kRcSolve) return;
    for (int y = 0; y < layers; y++)
        l.between(true, [&](auto rc, int s) {
            inner_stage<double, true, decltype(rc)::value>(D + (size_t)y * L * nl, g.line, s, g.line.before[s], g.by_nl, 1,
                                                           nl, tw);
        });
    l.outer([&](auto rc) {
        constexpr int R = decltype(rc)::value;
        const int sub = l.sub();
        for (int i = threadIdx.x; i < layers * nl * sub; i += threads) {
            const int e = l.by_lines(i), c = i - e * nl, y = layers > 1 ? l.by_sub(e) : 0, j = e - y * sub;
            if (c >= lines) continue;
            const double2 *z = D + ((size_t)y * L + j) * nl + c;
            double2 x[R];
#pragma unroll
            for (int r = 0; r < R; r++) x[r] = z[r * sub * nl];
            twiddle<double, true, R>(x, j, 1, tw);
            regdft::dft<double, true, R>(x);
            double2 *o = io + y * g.out_layer + (size_t)j * C + c;
#pragma unroll
            for (int r = 0; r < R; r++) o[(size_t)r * sub * C] = x[r];
        }
    });
}

// Position correction: a position's terms summed over its column CTAs in order, and its move.
__global__ void __launch_bounds__(128) rc_move_kernel(const double *terms, int per, int first, int m, double *positions,
                                                      const double *initial, int count, double step, double limit_update,
                                                      double limit_total, int *bad) {
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= m) return;
    double v[5] = {0, 0, 0, 0, 0};
    for (int part = 0; part < per; part++)
        for (int q = 0; q < 5; q++) v[q] += terms[((long long)i * per + part) * 5 + q];
    position_step(v, first + i, positions, initial, count, step, limit_update, limit_total, bad);
}

// -------------------------------------------------------------------------------------------------------- host side

using RcKernel = void (*)(RcArgs);
using Row128 = FixedLine<8, 16, 16>;
using Column128 = FixedLine<16, 8, 16>;
// several planes a CTA: eight columns (64 KB at four states) measured 0.83 ms against 1.2 with the sixteen of one plane
using Columns128 = FixedLine<16, 8, 8>;
constexpr int kMostLayers128 = 11;       // whose planes fit kRcSmem

// Lines per CTA: the power of two that fills kRcValues values over all layers; for columns at least 4 (64-byte segments)
// where those fit.
int rc_lines(int length, int layers, bool columns) {
    int nl = 1;
    while (2 * nl * length * layers <= kRcValues) nl *= 2;
    if (columns)
        while (nl < (layers == 1 ? 8 : 4) && 2ull * nl * length * layers * sizeof(double2) <= 100 * 1024) nl *= 2;
    return nl;
}

bool rc_line(int L, bool columns, AnyLine *line) { return L > 16 && L <= 4096 && plan_line(L, 16, !columns, line) && line->stages >= 2; }

// The launch's geometry over lines of `L` samples, `count` lines a plane.
bool rc_setup(RcArgs *g, int L, int count, int layers, bool columns, size_t *smem) {
    if (!rc_line(L, columns, &g->line)) return false;
    g->nl = L != 128 || layers > kMostLayers128 ? rc_lines(L, layers, columns) : layers == 1 ? 16 : 8;
    g->by_nl = divisor(g->nl);
    for (int i = 0; i < g->line.stages; i++) g->by_block[i] = divisor(L / g->line.r[i]);
    g->per = (count + g->nl - 1) / g->nl;
    const size_t last = (size_t)g->line.r[g->line.stages - 1];
    const size_t values = columns ? (size_t)layers * L * g->nl : (size_t)g->nl * (L / last) * (last | 1);
    *smem = (values + L) * sizeof(double2) + L * sizeof(unsigned short);
    return *smem <= kRcSmem;
}

template <int MODE>
RcKernel columns_kernel(int L, int layers) {
    using Line = std::conditional_t<MODE == kRcMixed || MODE == kRcSolve, Columns128, Column128>;
    return L == 128 && layers <= kMostLayers128 ? rc_columns_kernel<Line, MODE> : rc_columns_kernel<RunTimeLine, MODE>;
}

RcArgs base_args(const RcGeometry &q) {
    RcArgs g{};
    g.rows = q.rows; g.columns = q.columns; g.n = q.rows * q.columns;
    g.object_rows = q.object_rows; g.object_columns = q.object_columns;
    g.scan = q.scan;
    g.inv_n = 1.0 / ((double)q.rows * q.columns);
    return g;
}

// Launches over positions [first, first + count), `planes` planes' CTAs each, in batches whose CTAs fit one grid dimension.
cudaError_t launch_rc(RcKernel kernel, RcArgs g, int first, int count, int planes, int threads, size_t smem,
                      cudaStream_t s) {
    const int chunk = (int)std::max<long long>(1, (1LL << 30) / ((long long)g.per * planes));
    for (int done = 0; done < count; done += chunk) {
        const int m = std::min(chunk, count - done);
        g.first = first + done;
        kernel<<<(unsigned)((long long)m * planes * g.per), threads, smem, s>>>(g);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

bool rowcol64_applicable(int rows, int columns, int layers) {
    RcArgs g{};
    size_t smem = 0;
    return rc_setup(&g, columns, rows, 1, false, &smem) && rc_setup(&g, rows, columns, layers, true, &smem) && g.nl >= 2;
}

int rowcol64_parts(int rows, int columns, int layers) {
    RcArgs g{};
    size_t smem = 0;
    return rc_setup(&g, rows, columns, layers, true, &smem) ? g.per : 0;
}

cudaError_t configure_rowcol64() {
    const RcKernel kernels[] = {rc_rows_kernel<RunTimeLine, false>, rc_rows_kernel<RunTimeLine, true>,
                                rc_rows_kernel<Row128, false>, rc_rows_kernel<Row128, true>,
                                rc_through_kernel<RunTimeLine>, rc_through_kernel<Row128>,
                                rc_columns_kernel<RunTimeLine, kRcProject>, rc_columns_kernel<RunTimeLine, kRcPropagate>,
                                rc_columns_kernel<RunTimeLine, kRcMixed>, rc_columns_kernel<RunTimeLine, kRcSolve>,
                                rc_columns_kernel<Column128, kRcProject>, rc_columns_kernel<Column128, kRcPropagate>,
                                rc_columns_kernel<Columns128, kRcMixed>, rc_columns_kernel<Columns128, kRcSolve>};
    for (RcKernel k : kernels) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRcSmem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_rc_rows(const RcGeometry &q, const RcRows &r, bool inverse, cudaStream_t s) {
    if (r.count <= 0) return cudaSuccess;
    RcArgs g = base_args(q);
    size_t smem = 0;
    if (!rc_setup(&g, q.columns, q.rows, 1, false, &smem)) return cudaErrorInvalidValue;
    g.tw = q.tw_columns;
    g.in = r.in; g.by_class = r.by_class; g.in_layer = r.in_layer; g.from = r.from;
    g.object = r.object; g.object_after = r.object_after; g.conj_object = r.conj_object;
    g.out = r.out; g.out_layer = r.out_layer; g.out_stride = r.out_stride; g.out_first = r.out_first;
    const bool fixed = q.columns == 128;
    const RcKernel k = inverse ? (fixed ? rc_rows_kernel<Row128, true> : rc_rows_kernel<RunTimeLine, true>)
                               : (fixed ? rc_rows_kernel<Row128, false> : rc_rows_kernel<RunTimeLine, false>);
    g.layers = r.layers;
    return launch_rc(k, g, r.first, r.count, r.layers, kRcThreads, smem, s);
}

cudaError_t launch_rc_through(const RcGeometry &q, const RcRows &r, double2 *next, cudaStream_t s) {
    if (r.count <= 0) return cudaSuccess;
    RcArgs g = base_args(q);
    size_t smem = 0;
    if (!rc_setup(&g, q.columns, q.rows, 1, false, &smem)) return cudaErrorInvalidValue;
    g.tw = q.tw_columns;
    g.in = r.in; g.object = r.object; g.conj_object = r.conj_object; g.out = r.out; g.next = next;
    return launch_rc(q.columns == 128 ? rc_through_kernel<Row128> : rc_through_kernel<RunTimeLine>, g, r.first, r.count, 1,
                     kRcThreads, smem, s);
}

cudaError_t launch_rc_columns(const RcGeometry &q, const RcColumns &c, cudaStream_t s) {
    if (c.count <= 0) return cudaSuccess;
    RcArgs g = base_args(q);
    size_t smem = 0;
    if (!rc_setup(&g, q.rows, q.columns, c.layers, true, &smem)) return cudaErrorInvalidValue;
    g.tw = q.tw_rows;
    g.out = c.planes; g.out_layer = c.layer; g.out_stride = c.stride; g.out_first = c.plane_first;
    g.layers = c.layers;
    g.amplitudes = c.amplitudes;
    g.error = c.error;
    g.prop_rows = c.prop_rows; g.prop_columns = c.prop_columns; g.conj_prop = c.conj_prop;
    g.zero_infinite = c.zero_infinite;
    g.terms = c.terms;
    const RcKernel k = c.terms ? columns_kernel<kRcSolve>(q.rows, c.layers)
                       : c.prop_rows ? columns_kernel<kRcPropagate>(q.rows, c.layers)
                       : c.layers > 1 ? columns_kernel<kRcMixed>(q.rows, c.layers)
                                      : columns_kernel<kRcProject>(q.rows, c.layers);
    // several layers: a thread per block of the centre step, which walks them
    const int centre = g.nl * (int)g.by_block[g.line.stages - 1].d;
    const int threads = c.layers == 1 ? kRcThreads : std::max(64, std::min(kRcThreads, (centre + 31) / 32 * 32));
    return launch_rc(k, g, c.first, c.count, 1, threads, smem, s);
}

cudaError_t launch_rc_move(const double *terms, int per, int first, int m, double *positions, const double *initial,
                           int count, double step, double limit_update, double limit_total, int *bad, cudaStream_t s) {
    if (m <= 0) return cudaSuccess;
    rc_move_kernel<<<(m + 127) / 128, 128, 0, s>>>(terms, per, first, m, positions, initial, count, step, limit_update,
                                                   limit_total, bad);
    return cudaGetLastError();
}

}  // namespace cubo
