// The shifted-probe table: ifft2(spectrum x ramp) of every fractional shift class (Ptychography.swift:303-320), computed
// in FP64 and written in the plan's type, one launch (sm_100a).
//
// An FP64 plane does not fit one CTA from 14,000 pixels on (128 x 128: 256 KB), but a Fourier shift needs no plane
// exchange between CTAs: output rows y = b + f y' (b < f, f a divisor of the row count) depend on the spectrum only
// through the fold
//     V_b[k', c] = sum_{r < f} w_b[k' + r R/f] F[k' + r R/f, c],   w_b[k] = ramp_row[k] e^{2 pi i k b / R} / n,
// after which they are a plain (R/f) x C inverse transform of V_b x ramp_column.  So CTA (class, b) reads the spectrum
// (the same for every class: from L2), keeps an (R/f) x C plane in shared memory and writes whole output rows; the fold
// costs f complex multiply-adds a sample.  The smallest f that fits is the fastest (3,364 classes of 128 x 128: f = 2
// 0.99 ms, 4 1.26, 8 2.0, before the two changes below).  The transform is the in-place
// decimation in time of the any-size position pass (anypass.cuh): the fold writes the samples straight into
// digit-reversed slots, and the last row stage writes natural order.
//
// Bound by shared-memory wavefronts (59 % of the pipe; FP64 pipe 26 %), the phases of one CTA in sequence.  Four samples'
// fold loads in flight a thread and the spectrum's columns put in slot order once per table (scattered 16-byte reads took
// 16 wavefronts a warp instead of 4) took the same table from 0.99 to 0.68 ms.  Before, each class took a ramp product, a
// batched line FFT through HBM in two passes, a scaling and a conversion: 2.05 ms, and one FP64 plane of scratch per
// class (3,600 classes of 96 x 96: 1.93 -> 0.46 ms; 576 of 256 x 256: 1.37 -> 0.85 ms; the FP64 form at 128 x 128, which
// ran the clustered plane kernel's inverse: 0.82 -> 0.76 ms).
#include "anypass.cuh"

namespace cubo {

namespace {

constexpr int kShiftThreads = 512;
constexpr int kShiftUnroll = 4;
constexpr size_t kShiftSmem = 226 * 1024;

struct ShiftArgs {
    int rows, columns, fold;
    const double2 *spectrum;          // [row frequency][column slot]
    const double2 *ramp_rows;         // [class][rows]
    const double2 *ramp_columns;      // [class][columns]
    const double2 *tw_rows, *tw_columns;
    double scale;
    void *out;                        // [class][rows][columns], complex of the plan's type
    AnyLine lines, columns_line;      // the folded column line (rows / fold) and the row line (columns)
    Divisor by_lines, by_columns;     // rows / fold, columns
    int pitch;
};

// The last row stage (inverse), into output rows b + fold y'.
template <typename T, int R>
__device__ __forceinline__ void store_stage(const double2 *D, const ShiftArgs &g, C2<T> *out, const double2 *tw) {
    const Divisor per = g.columns_line.sub[0];
    const int sub = (int)per.d, total = (int)g.by_lines.d * sub;
    for (int i = threadIdx.x; i < total; i += blockDim.x) {
        const int row = quotient(i, per), j = i - row * sub;
        const double2 *y = D + row * g.pitch + j;
        double2 x[R];
#pragma unroll
        for (int q = 0; q < R; q++) x[q] = y[q * sub];
        twiddle<double, true, R>(x, j, 1, tw);
        regdft::dft<double, true, R>(x);
        C2<T> *o = out + (size_t)row * g.fold * g.columns + j;
#pragma unroll
        for (int r = 0; r < R; r++) o[r * sub] = mk<T>((T)x[r].x, (T)x[r].y);
    }
}

// The spectrum with each row's columns in slot order, so that every class reads it in order.
__global__ void __launch_bounds__(256) shift_order_kernel(const double2 *in, double2 *out, int n,
                                                          AnyLine line) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int row = i / line.L, slot = i - row * line.L;
    out[i] = in[row * line.L + slot_frequency(line, slot)];
}

template <typename T>
__global__ void __launch_bounds__(kShiftThreads, 1) shift_kernel(const __grid_constant__ ShiftArgs g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int R = g.rows, C = g.columns, folded = (int)g.by_lines.d, tid = threadIdx.x;
    double2 *D = reinterpret_cast<double2 *>(smem_raw);
    double2 *twr = D + (size_t)folded * g.pitch;  // W_rows^t
    double2 *twc = twr + R;                       // W_columns^t
    double2 *w = twc + C;                         // w_b
    double2 *ramp = w + R;                        // ramp_column in slot order
    unsigned short *kr = reinterpret_cast<unsigned short *>(ramp + C);  // frequency of each row slot
    const int cls = blockIdx.x / g.fold, b = blockIdx.x - cls * g.fold;
    for (int i = tid; i < R; i += blockDim.x) {
        twr[i] = g.tw_rows[i];
        const double2 v = regdft::turn<double2, true>(g.ramp_rows[(size_t)cls * R + i], g.tw_rows[(i * b) % R]);
        w[i] = make_double2(v.x * g.scale, v.y * g.scale);
    }
    for (int i = tid; i < C; i += blockDim.x) {
        twc[i] = g.tw_columns[i];
        ramp[i] = g.ramp_columns[(size_t)cls * C + slot_frequency(g.columns_line, i)];
    }
    for (int i = tid; i < folded; i += blockDim.x) kr[i] = (unsigned short)slot_frequency(g.lines, i);
    __syncthreads();
    const int total = folded * C;
    for (int i0 = tid; i0 < total; i0 += kShiftUnroll * blockDim.x) {  // several samples' loads in flight per thread
        const double2 *F[kShiftUnroll];
        int at[kShiftUnroll], k[kShiftUnroll], c[kShiftUnroll];
        double2 v[kShiftUnroll];
#pragma unroll
        for (int u = 0; u < kShiftUnroll; u++) {
            const int i = min(i0 + u * (int)blockDim.x, total - 1), e = quotient(i, g.by_columns);
            c[u] = i - e * C;
            k[u] = kr[e];
            at[u] = e * g.pitch + c[u];
            F[u] = g.spectrum + (size_t)k[u] * C + c[u];
            v[u] = make_double2(0, 0);
        }
        for (int r = 0; r < g.fold; r++) {
            double2 f[kShiftUnroll];
#pragma unroll
            for (int u = 0; u < kShiftUnroll; u++) f[u] = F[u][(size_t)r * total];
#pragma unroll
            for (int u = 0; u < kShiftUnroll; u++) {
                const double2 q = w[k[u] + r * folded];
                v[u].x += f[u].x * q.x - f[u].y * q.y;
                v[u].y += f[u].x * q.y + f[u].y * q.x;
            }
        }
#pragma unroll
        for (int u = 0; u < kShiftUnroll; u++)
            if (i0 + u * (int)blockDim.x < total) D[at[u]] = cmul(v[u], ramp[c[u]]);
    }
    __syncthreads();
    for (int s = g.lines.stages - 1; s >= 0; s--) {  // W_(R/fold)^t = W_R^(fold t)
        with_radix<false>(g.lines.r[s], [&](auto r) {
            inner_stage<double, true, decltype(r)::value>(D, g.lines, s, g.fold * g.lines.before[s], g.by_columns, 1,
                                                          g.pitch, twr);
        });
        __syncthreads();
    }
    for (int s = g.columns_line.stages - 1; s >= 1; s--) {
        with_radix<false>(g.columns_line.r[s], [&](auto r) {
            inner_stage<double, true, decltype(r)::value>(D, g.columns_line, s, g.columns_line.before[s], g.by_lines,
                                                          g.pitch, 1, twc);
        });
        __syncthreads();
    }
    C2<T> *out = static_cast<C2<T> *>(g.out) + (size_t)cls * R * C + (size_t)b * C;
    with_radix<false>(g.columns_line.r[0], [&](auto r) { store_stage<T, decltype(r)::value>(D, g, out, twc); });
}

size_t shift_smem(int rows, int columns, int fold) {
    const size_t folded = (size_t)(rows / fold), pitch = (size_t)(columns | 1);
    return (folded * pitch + 2 * (size_t)(rows + columns)) * sizeof(double2) +
           folded * sizeof(unsigned short);
}

// The fold of a rows x columns table: the smallest divisor of the rows whose folded plane fits one CTA and whose lines
// have plans (0: none, the table takes the line transforms through HBM).
int shift_fold(int rows, int columns, AnyLine *lines, AnyLine *columns_line) {
    if (rows < 2 || columns < 2 || columns > 4096 || rows > 4096 || !plan_line(columns, 16, true, columns_line)) return 0;
    for (int f = 1; f <= 32; f++)
        if (rows % f == 0 && (long long)(rows / f) * columns < 65536 && shift_smem(rows, columns, f) <= kShiftSmem &&
            plan_line(rows / f, 16, false, lines))
            return f;
    return 0;
}

}  // namespace

bool shift_applicable(int rows, int columns) {
    AnyLine l{}, c{};
    return shift_fold(rows, columns, &l, &c) > 0;
}

cudaError_t configure_shift() {
    cudaError_t e = cudaFuncSetAttribute(shift_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShiftSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(shift_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShiftSmem);
    return e;
}

template <typename T>
cudaError_t launch_shift_table(const Fft2Plan64 &p, const double2 *spectrum, double2 *scratch,
                               const double2 *ramps_rows, const double2 *ramps_columns, int classes, C2<T> *out,
                               cudaStream_t s) {
    if (classes <= 0) return cudaSuccess;
    ShiftArgs g{};
    g.rows = p.rows;
    g.columns = p.columns;
    g.fold = shift_fold(p.rows, p.columns, &g.lines, &g.columns_line);
    if (g.fold == 0) return cudaErrorInvalidValue;
    g.spectrum = scratch;
    g.ramp_rows = ramps_rows;
    g.ramp_columns = ramps_columns;
    g.tw_rows = p.tw_rows;
    g.tw_columns = p.tw_columns;
    g.scale = 1.0 / ((double)p.rows * p.columns);
    g.out = out;
    g.by_lines = divisor(p.rows / g.fold);
    g.by_columns = divisor(p.columns);
    g.pitch = p.columns | 1;
    const size_t smem = shift_smem(p.rows, p.columns, g.fold);
    // the SM's 512 threads (at 128 registers) over the CTAs whose planes fit it: 3,600 classes of 96 x 96 (one fits) 0.46
    // ms at 512 threads, 0.50 at 256; of 64 x 64 (three) 0.19 at 256, 0.25 at 512; of 40 x 48 (seven) 0.13 at 128, 0.15
    // at 256
    const int threads = smem > kShiftSmem / 2 ? kShiftThreads : smem > kShiftSmem / 4 ? 256 : 128;
    const int n = p.rows * p.columns;
    shift_order_kernel<<<(n + 255) / 256, 256, 0, s>>>(spectrum, scratch, n, g.columns_line);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    shift_kernel<T><<<(unsigned)classes * (unsigned)g.fold, threads, smem, s>>>(g);
    return cudaGetLastError();
}
template cudaError_t launch_shift_table<float>(const Fft2Plan64 &, const double2 *, double2 *, const double2 *,
                                               const double2 *, int, float2 *, cudaStream_t);
template cudaError_t launch_shift_table<double>(const Fft2Plan64 &, const double2 *, double2 *, const double2 *,
                                                const double2 *, int, double2 *, cudaStream_t);

}  // namespace cubo
