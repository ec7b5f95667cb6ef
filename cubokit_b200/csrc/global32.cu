// Host side of the FP32 position pass through global memory (global32.cuh), its instances with compile-time geometry and
// the direct DFT.
#include <algorithm>

#include "global32.cuh"

namespace cubo {

namespace {

// --------------------------------------------------------------------- 128, 192 and 256: geometry at compile time

// Rows of RA RB samples, NL a CTA: RA samples a thread in the outer stage, RB (even, padded by one) in the inner one.
template <int RA, int RB, int NL, bool INV>
__global__ void __launch_bounds__(kG32Threads, 4) g32_rows_fixed(const __grid_constant__ G32Args g) {
    constexpr int L = RA * RB, RL = RB + 1, P = RA * RL;
    static_assert(RB % 2 == 0, "one pad a block");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const PositionPassArgs<float> &a = g.p;
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = D + NL * P;
    const int tid = threadIdx.x;
    const int p = a.first + (int)(blockIdx.x / g.per), r0 = (int)(blockIdx.x % g.per) * NL;
    const int rows = min(NL, a.rows - r0);
    for (int i = tid; i < L; i += kG32Threads) tw[i] = a.tw_columns[i];
    float2 *io = a.dpsi + (size_t)p * a.n + (size_t)r0 * L;
    if constexpr (!INV) {
        const int rr = a.scan.rr[p], cc = a.scan.cc[p], cls = a.scan.cls[p];
        const float2 *S = a.shifted + (size_t)cls * a.n + (size_t)r0 * L;
        const bool interior = cc >= L / 2 && cc + L / 2 <= a.object_columns;
        __syncthreads();
#pragma unroll
        for (int i0 = 0; i0 < NL * RB; i0 += kG32Threads) {
            const int i = i0 + tid, row = i / RB, j = i % RB;
            if (row < rows) {
                const float2 *s = S + row * L + j;
                const float2 *o = a.object + (size_t)g32_wrap(rr + corner_offset(r0 + row, a.rows), a.object_rows) *
                                             a.object_columns;
                float2 x[RA], q[RA];
#pragma unroll
                for (int r = 0; r < RA; r++) {
                    const int c = j + r * RB, off = c < L / 2 ? c : c - L;
                    x[r] = s[r * RB];
                    q[r] = o[interior ? cc + off : g32_wrap(cc + off, a.object_columns)];
                }
#pragma unroll
                for (int r = 0; r < RA; r++) x[r] = regdft::turn<float2, false>(x[r], q[r]);
                regdft::dft<float, false, RA>(x);
                twiddle<float, false, RA>(x, j, 1, tw);
                float2 *y = D + row * P + j;
#pragma unroll
                for (int r = 0; r < RA; r++) y[r * RL] = x[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i0 = 0; i0 < NL * RA; i0 += kG32Threads) {
            const int i = i0 + tid, row = i / RA, K = i % RA;
            if (row < rows) {
                const float2 *y = D + row * P + K * RL;
                float2 x[RB];
#pragma unroll
                for (int r = 0; r < RB; r++) x[r] = y[r];
                regdft::dft<float, false, RB>(x);
                float2 *o = io + row * L + K;
#pragma unroll
                for (int r = 0; r < RB; r++) o[r * RA] = x[r];
            }
        }
    } else {
#pragma unroll
        for (int i0 = 0; i0 < NL * RA; i0 += kG32Threads) {
            const int i = i0 + tid, row = i / RA, K = i % RA;
            if (row < rows) {
                const float2 *o = io + row * L + K;
                float2 x[RB];
#pragma unroll
                for (int r = 0; r < RB; r++) x[r] = o[r * RA];
                regdft::dft<float, true, RB>(x);
                float2 *y = D + row * P + K * RL;
#pragma unroll
                for (int r = 0; r < RB; r++) y[r] = x[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int i0 = 0; i0 < NL * RB; i0 += kG32Threads) {
            const int i = i0 + tid, row = i / RB, j = i % RB;
            if (row < rows) {
                const float2 *y = D + row * P + j;
                float2 x[RA];
#pragma unroll
                for (int r = 0; r < RA; r++) x[r] = y[r * RL];
                twiddle<float, true, RA>(x, j, 1, tw);
                regdft::dft<float, true, RA>(x);
                float2 *o = io + row * L + j;
#pragma unroll
                for (int r = 0; r < RA; r++) o[r * RB] = x[r];
            }
        }
    }
}

// Columns of RA RB samples, NL a CTA: RA samples a thread in the outer stages, RB in the centre step.
template <int RA, int RB, int NL>
__global__ void __launch_bounds__(kG32Threads, 4) g32_columns_fixed(const __grid_constant__ G32Args g) {
    constexpr int L = RA * RB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double scratch[kG32Threads / 32];
    const PositionPassArgs<float> &a = g.p;
    const int C = a.columns, tid = threadIdx.x;
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    float2 *tw = D + NL * L;
    const int p = a.first + (int)(blockIdx.x / g.per), c0 = (int)(blockIdx.x % g.per) * NL;
    const int lines = min(NL, C - c0);
    float2 *io = a.dpsi + (size_t)p * a.n + c0;
    const float *A = a.amplitudes + (size_t)p * a.n + c0;
    for (int i = tid; i < L; i += kG32Threads) {
        tw[i] = a.tw_rows[i];
        asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (size_t)i * C));  // the amplitudes, for the centre step
    }
    __syncthreads();
#pragma unroll
    for (int i0 = 0; i0 < NL * RB; i0 += kG32Threads) {
        const int i = i0 + tid, j = i / NL, c = i % NL;
        if (i < NL * RB && c < lines) {
            const float2 *o = io + (size_t)j * C + c;
            float2 x[RA];
#pragma unroll
            for (int r = 0; r < RA; r++) x[r] = o[(size_t)r * RB * C];
            regdft::dft<float, false, RA>(x);
            twiddle<float, false, RA>(x, j, 1, tw);
            float2 *y = D + j * NL + c;
#pragma unroll
            for (int r = 0; r < RA; r++) y[r * RB * NL] = x[r];
        }
    }
    __syncthreads();
    double err = 0;
#pragma unroll
    for (int i0 = 0; i0 < NL * RA; i0 += kG32Threads) {
        const int i = i0 + tid, b = i / NL, c = i % NL;
        if (i < NL * RA && c < lines) {
            const float *am = A + (size_t)b * C + c;  // output q of block b is the frequency b + RA q
            float measured[RB];
#pragma unroll
            for (int q = 0; q < RB; q++) measured[q] = am[(size_t)q * RA * C];
            float2 *y = D + b * RB * NL + c;
            float2 x[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) x[r] = y[r * NL];
            regdft::dft<float, false, RB>(x);
            project_values<float, RB>(x, measured, a.inv_n, err);
            regdft::dft<float, true, RB>(x);
#pragma unroll
            for (int r = 0; r < RB; r++) y[r * NL] = x[r];
        }
    }
    const double total = g32_block_sum(err, scratch);  // its barriers also order the centre step before the inverse one
    if (tid == 0) a.error[(size_t)p * g.per + c0 / NL] = total;
#pragma unroll
    for (int i0 = 0; i0 < NL * RB; i0 += kG32Threads) {
        const int i = i0 + tid, j = i / NL, c = i % NL;
        if (i < NL * RB && c < lines) {
            const float2 *y = D + j * NL + c;
            float2 x[RA];
#pragma unroll
            for (int r = 0; r < RA; r++) x[r] = y[r * RB * NL];
            twiddle<float, true, RA>(x, j, 1, tw);
            regdft::dft<float, true, RA>(x);
            float2 *o = io + (size_t)j * C + c;
#pragma unroll
            for (int r = 0; r < RA; r++) o[(size_t)r * RB * C] = x[r];
        }
    }
}

// ---------------------------------------------------------------- direct DFT, lengths with a prime factor above 31

// nl rows of one position: the exit wave's (exit_wave) or dpsi's, transformed forward or (inv) back into dpsi.
__global__ void __launch_bounds__(kG32Threads, 2)
    g32_rows_direct(PositionPassArgs<float> a, int nl, int exit_wave, int inv) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    const int L = a.columns;
    float2 *tw = D + (size_t)nl * L;
    for (int i = threadIdx.x; i < L; i += kG32Threads) tw[i] = a.tw_columns[i];
    const int per = a.rows / nl;
    const int p = a.first + (int)(blockIdx.x / per), r0 = (int)(blockIdx.x % per) * nl;
    float2 *rows = a.dpsi + (size_t)p * a.n + (size_t)r0 * L;
    const int rr = a.scan.rr[p], cc = a.scan.cc[p], cls = a.scan.cls[p];
    const float2 *S = a.shifted + (size_t)cls * a.n + (size_t)r0 * L;
    for (int i = threadIdx.x; i < nl * L; i += kG32Threads) {
        if (!exit_wave) { D[i] = rows[i]; continue; }
        const int j = i / L, e = i - j * L;
        const int y = g32_wrap(rr + corner_offset(r0 + j, a.rows), a.object_rows);
        const int x = g32_wrap(cc + corner_offset(e, a.columns), a.object_columns);
        D[i] = cmul(S[i], a.object[(size_t)y * a.object_columns + x]);
    }
    __syncthreads();
    direct_lines<float, kG32Threads, kG32MaxN / kG32Threads>(D, LineGeom{L, nl, 1, L}, tw, inv != 0);
    for (int i = threadIdx.x; i < nl * L; i += kG32Threads) rows[i] = D[i];
}

// nl columns of one position, element e of column j at D[e nl + j].
__global__ void __launch_bounds__(kG32Threads, 2) g32_columns_direct(PositionPassArgs<float> a, int nl) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double scratch[kG32Threads / 32];
    float2 *D = reinterpret_cast<float2 *>(smem_raw);
    const int L = a.rows;
    float2 *tw = D + (size_t)nl * L;
    for (int i = threadIdx.x; i < L; i += kG32Threads) tw[i] = a.tw_rows[i];
    const int per = a.columns / nl;
    const int p = a.first + (int)(blockIdx.x / per), c0 = (int)(blockIdx.x % per) * nl;
    float2 *base = a.dpsi + (size_t)p * a.n + c0;
    const float *A = a.amplitudes + (size_t)p * a.n + c0;
    for (int i = threadIdx.x; i < nl * L; i += kG32Threads) {
        const int e = i / nl, j = i - e * nl;
        D[i] = base[(size_t)e * a.columns + j];
    }
    __syncthreads();
    const LineGeom geom{L, nl, nl, 1};
    direct_lines<float, kG32Threads, kG32MaxN / kG32Threads>(D, geom, tw, false);
    double err = 0;
    for (int i = threadIdx.x; i < nl * L; i += kG32Threads) {
        const int e = i / nl, j = i - e * nl;
        float2 f[1] = {D[i]};
        const float measured[1] = {A[(size_t)e * a.columns + j]};
        project_values<float, 1>(f, measured, a.inv_n, err);
        D[i] = f[0];
    }
    const double total = g32_block_sum(err, scratch);  // its barriers also order the projection before the inverse
    if (threadIdx.x == 0) a.error[(size_t)p * per + c0 / nl] = total;
    direct_lines<float, kG32Threads, kG32MaxN / kG32Threads>(D, geom, tw, true);
    for (int i = threadIdx.x; i < nl * L; i += kG32Threads) {
        const int e = i / nl, j = i - e * nl;
        base[(size_t)e * a.columns + j] = D[i];
    }
}

// -------------------------------------------------------------------------------------------------------- host side

// Direct: the largest divisor d of `lines` with d line_length <= kG32MaxN.
int g32_divisor_lines(int line_length, int lines) {
    int best = 1;
    for (int d = 1; d <= lines && (long long)d * line_length <= kG32MaxN; d++)
        if (lines % d == 0) best = d;
    return best;
}

// Lines per CTA of the planned launches: the power of two that fills kG32MaxN elements; for columns at least 16 (whole
// 128-byte segments of each row) while those fit a third of the SM.  The last CTA of a position may hold fewer.
int g32_lines(int line_length, bool columns) {
    int nl = 1;
    while (2 * nl * line_length <= kG32MaxN) nl *= 2;
    if (columns)
        while (nl < 16 && 2 * nl * line_length * sizeof(float2) <= 72 * 1024) nl *= 2;
    return nl;
}

struct G32Plan {
    AnyLine line{};
    bool planned = false;  // else the direct DFT
    int nl = 1;
    size_t smem = 0;
    G32Kernel forward = nullptr, inverse = nullptr, columns = nullptr;
};

G32Plan g32_plan(int L, bool columns) {
    G32Plan p;
    p.planned = L >= 2 && plan_line(L, 31, !columns, &p.line);
    if (!p.planned) return p;
    p.nl = g32_lines(L, columns);
    bool w = false;
    for (int i = 0; i < p.line.stages; i++) w = w || p.line.r[i] > 16;
    const size_t last = (size_t)p.line.r[p.line.stages - 1];
    p.smem = columns ? ((size_t)p.nl * L + L) * sizeof(float2) + L * sizeof(unsigned short)
                     : ((size_t)p.nl * (L / last) * (last | 1) + L) * sizeof(float2) + L * sizeof(unsigned short);
    if (columns) {
        p.columns = w ? g32_wide_columns() : g32_columns<false>;
        if (L == 128) p.columns = g32_columns_fixed<16, 8, 32>;
        if (L == 192) p.columns = g32_columns_fixed<16, 12, 16>;
        if (L == 256) p.columns = g32_columns_fixed<16, 16, 16>;
    } else {
        p.forward = w ? g32_wide_rows_forward() : g32_rows_forward<false>;
        p.inverse = w ? g32_wide_rows_inverse() : g32_rows_inverse<false>;
        if (L == 128) { p.forward = g32_rows_fixed<8, 16, 32, false>; p.inverse = g32_rows_fixed<8, 16, 32, true>; }
        if (L == 192) { p.forward = g32_rows_fixed<12, 16, 16, false>; p.inverse = g32_rows_fixed<12, 16, 16, true>; }
        if (L == 256) { p.forward = g32_rows_fixed<16, 16, 16, false>; p.inverse = g32_rows_fixed<16, 16, 16, true>; }
    }
    return p;
}

}  // namespace

bool global32_applicable(int rows, int columns) {
    return rows >= 1 && columns >= 1 && rows <= kG32MaxN && columns <= kG32MaxN;
}

int global32_partials_per_position(int rows, int columns) {
    const G32Plan p = g32_plan(rows, true);
    return p.planned ? (columns + p.nl - 1) / p.nl : columns / g32_divisor_lines(rows, columns);
}

cudaError_t configure_global32() {
    const G32Kernel kernels[] = {g32_rows_forward<false>, g32_rows_inverse<false>, g32_columns<false>,
                                 g32_wide_rows_forward(), g32_wide_rows_inverse(), g32_wide_columns(),
                                 g32_columns_fixed<16, 8, 32>, g32_columns_fixed<16, 12, 16>,
                                 g32_columns_fixed<16, 16, 16>, g32_rows_fixed<8, 16, 32, false>,
                                 g32_rows_fixed<8, 16, 32, true>, g32_rows_fixed<12, 16, 16, false>,
                                 g32_rows_fixed<12, 16, 16, true>, g32_rows_fixed<16, 16, 16, false>,
                                 g32_rows_fixed<16, 16, 16, true>};
    for (G32Kernel k : kernels) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kG32Smem);
        if (e != cudaSuccess) return e;
    }
    cudaError_t e = cudaFuncSetAttribute(g32_rows_direct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kG32Smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(g32_columns_direct, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kG32Smem);
    return e;
}

cudaError_t launch_position_pass_global32(const PositionPassArgs<float> &a, int *launches, cudaStream_t s) {
    if (launches) *launches = 0;
    if (a.count <= 0) return cudaSuccess;
    if (!global32_applicable(a.rows, a.columns)) return cudaErrorInvalidValue;
    const G32Plan pr = g32_plan(a.columns, false), pc = g32_plan(a.rows, true);
    const int nr = pr.planned ? pr.nl : g32_divisor_lines(a.columns, a.rows);
    const int nc = pc.planned ? pc.nl : g32_divisor_lines(a.rows, a.columns);
    const int per_r = (a.rows + nr - 1) / nr, per_c = (a.columns + nc - 1) / nc;
    const size_t direct_r = ((size_t)nr + 1) * a.columns * sizeof(float2);
    const size_t direct_c = ((size_t)nc + 1) * a.rows * sizeof(float2);
    auto args = [](const G32Plan &p, int per) {
        G32Args g{};
        g.line = p.line;
        g.nl = p.nl;
        g.per = per;
        g.by_nl = divisor(p.nl);
        for (int i = 0; i < p.line.stages; i++) g.by_block[i] = divisor(p.line.L / p.line.r[i]);
        return g;
    };
    G32Args gr = args(pr, per_r), gc = args(pc, per_c);
    // Batches of positions whose CTAs fit one grid dimension.  (Batches small enough to stay in L2 between their launches,
    // 19 to 111 MB of residuals, measured slower, before the projection's present form: 2.95 to 4.29 ms against 2.51 at 4,096 positions of 256 x 256; the gaps and
    // part waves of 3 launches a batch cost more than the HBM traffic they save.)
    const int chunk = (int)std::max<long long>(1, (1LL << 30) / std::max(per_r, per_c));
    int count = 0;
    for (int first = 0; first < a.count; first += chunk) {
        PositionPassArgs<float> b = a;
        b.first = a.first + first;
        gr.p = gc.p = b;
        const int m = std::min(chunk, a.count - first);
        const unsigned grid_r = (unsigned)((long long)m * per_r), grid_c = (unsigned)((long long)m * per_c);
        if (pr.planned) pr.forward<<<grid_r, kG32Threads, pr.smem, s>>>(gr);
        else g32_rows_direct<<<grid_r, kG32Threads, direct_r, s>>>(b, nr, 1, 0);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) {
            if (pc.planned) pc.columns<<<grid_c, kG32Threads, pc.smem, s>>>(gc);
            else g32_columns_direct<<<grid_c, kG32Threads, direct_c, s>>>(b, nc);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            if (pr.planned) pr.inverse<<<grid_r, kG32Threads, pr.smem, s>>>(gr);
            else g32_rows_direct<<<grid_r, kG32Threads, direct_r, s>>>(b, nr, 0, 1);
            e = cudaGetLastError();
        }
        if (e != cudaSuccess) return e;
        count += 3;
    }
    if (launches) *launches = count;
    return cudaSuccess;
}

}  // namespace cubo
