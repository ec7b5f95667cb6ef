// The split-BF16 position pass for a 128 x 128 detector: the 2-D DFT pair as products with a real 128 x 128 matrix on
// the tensor cores.
//
// Arithmetic (Ptychography.swift:321-350): exit wave X = S * O[patch], F = fft2(X), the Fourier-modulus projection with
// the 1/n of ifft2 folded in, then dpsi = ifft2(F').  The 128-point DFT matrix factors as W = T C with C real:
//
//   C row 0 = 1, row 1 = cos(pi k), rows 2j and 2j + 1 = cos(2 pi j k / 128) and sin(2 pi j k / 128)  (j = 1..63)
//
// and T combining row pairs: for z = C x, (W x)[j] = z[2j] - i z[2j+1] and (W x)[128 - j] = z[2j] + i z[2j+1]
// ((W x)[0] = z[0], (W x)[64] = z[1]); conj(W) swaps the two.  Every transform is therefore the real product D = C B of
// the re and the im plane separately, half the multiply-adds of a complex DFT matrix, and T is applied only where a
// stage's result is needed in the frequency or pixel basis: on a row of D inside one thread, and between the rows of
// TMEM lanes 2j and 2j + 1 (adjacent lanes of a warp) with one shuffle per value.  With D[m][n] = sum_k A[m][k] B[n][k]
// (A = C_sigma in tensor memory, B = data in shared memory):
//
//   stage 1  B[n = pos(r)][k = pos(c)]     = X                   K-major   D[raw c][pos r]
//   stage 2  B[n = raw c][k = pos(r)]      = D1                  K-major   D[raw r][raw c]  -> T both ways -> F[kr][kc]
//   stage 3  B[n = pos(kc)][k = pos(kr)]   = F'                  MN-major  D[raw r][pos kc]
//   stage 4  B[n = raw r][k = pos(kc)]     = D3                  K-major   D[raw c][raw r]  -> T both ways -> dpsi[r][c]
//
// pos orders samples and frequencies the way one thread holds the kc after T (8 consecutive positions per thread and row),
// sigma is its inverse, and C_sigma[m][pos] = C[m][sigma(pos)], the one A operand of all four stages, contracts in that
// order.  Each real product P Q is P_hi Q_hi + P_hi Q_lo + P_lo Q_hi in bf16 with FP32 accumulation in tensor memory: 3 x 8
// K-steps = 24 tcgen05.mma (M = N = 128, K = 16) per plane and stage.  The two planes run as a pipeline: the re plane's
// result is read out and its next stage issued while the tensor core still works on the im plane.
//
// One persistent CTA per SM with 210 KB of shared memory: the four B planes and the next position's amplitudes, bulk-copied
// in behind stages 3 to 2.  Tensor memory: C_sigma hi / lo (columns 0-127), the re-plane result (128-255), the im-plane
// result (256-383), and stage 1's re result (384-511), which is apart so that it can run while the last position's residual
// is still read out of the other two.  kThreads = 512 working threads: thread (warp w, lane i) owns TMEM lane
// 32 (w mod 4) + i and the kCols-column group w / 4 of each result (kCols = 32); the layout constants follow from kThreads.
// A thread of a fifth warpgroup issues the products.
//
// The tensor core is busy 12.3 K cycles a position and each scheduler issues 11 K, so what counts is that the phases
// overlap.  Issuing 24 products takes as long as running them: with a block barrier before each issue every warp waited about
// 1.2 K cycles five times a position for the warp that issued.  Now the working warps only arrive on an mbarrier and go on to
// the next wait for a product; nothing they do needs another warp's writes.  16,384 positions: 2.03-2.10 ms with barriers,
// 1.78 so (43 % tensor, 38 % issue; the exit wave takes 5 K cycles, the projection 4.9 K, the residual 4.7 K).  The
// registers are split 112 / 32 between working and issuing warpgroups, the launch's own total.  1024 working threads measured
// slower (the phases between the products need instructions more than latency), as did four rows of exit wave in flight
// instead of two (spills, 1.87 ms) and half the warps writing the residual before their exit wave (1.89).
//
// Amplitudes are pre-permuted into the order each thread consumes them (a warp reads 512 contiguous bytes per load); dpsi is
// written [position][row][column].  Waits are bounded: a wait that runs out sets *fault and the CTA stops after freeing its
// tensor memory.
#include "engine.h"
#include "umma.cuh"

namespace cubo {

namespace {

using namespace umma;

constexpr int kN = 128;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kLaunch = kThreads + 128;    // the working warps and one warpgroup that issues the products
constexpr int kGroups = kWarps / 4;        // warps per TMEM lane quadrant: column groups of a result
constexpr int kCols = kN / kGroups;        // result columns per thread (32)
constexpr int kSub = kCols / 16;           // sub-blocks of 4 column pairs per parity set (2)
constexpr int kRowsPerWarp = kN / kWarps;  // exit-wave rows per warp (8)
constexpr int kBatch = 1024 / kThreads;    // exit-wave rows whose loads are in flight at once (2)
static_assert(kCols % 16 == 0 && kRowsPerWarp % kBatch == 0, "thread layout");
// Canonical no-swizzle layout of a 128 x 128 bf16 plane with its core matrices (8 rows x 16 bytes) 144 bytes apart
// along K: the 16 bytes of padding put the K chunks of one row in different banks, so 4-byte stores along a row (the exit
// wave) and 16-byte stores of consecutive rows (the read-outs) are conflict-free.  The 32 bytes after each 8 rows do the same
// for the projection's stores, whose lane pairs are 16 columns apart.
constexpr uint32_t kLBO = 144, kSBO = 16 * kLBO + 32;
constexpr int kPlaneBytes = 16 * kSBO;          // 36.5 KB
constexpr uint64_t kWaitLimit = 2000000000ull;  // ns of wall time an mbarrier wait may take before giving up
// tensor-memory columns: C_sigma, the re and im results, and stage 1's re result
constexpr uint32_t kCSigma = 0, kSlotRe = 128, kSlotIm = 256, kSlotNext = 384;
constexpr int kReHi = 0, kImHi = 2;             // B planes: re hi, re lo, im hi, im lo
constexpr uint32_t kIdescK = idesc_bf16(128, 128, false, false), kIdescMN = idesc_bf16(128, 128, false, true);

__device__ __forceinline__ uint32_t kmajor_offset(int row, int k) {
    return (row >> 3) * kSBO + (k >> 3) * kLBO + (row & 7) * 16 + (k & 7) * 2;
}
__device__ __forceinline__ uint32_t mnmajor_offset(int k, int col) {
    return (col >> 3) * kSBO + (k >> 3) * kLBO + (k & 7) * 16 + (col & 7) * 2;
}

__device__ __forceinline__ int wrap_once(int v, int size) { return v < 0 ? v + size : (v >= size ? v - size : v); }

// Packed FP32x2 arithmetic (sm_100 mul / fma / sub .f32x2): one instruction for two values, each rounded as the scalar
// operation rounds it.
__device__ __forceinline__ float2 pmul(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "mul.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// The frequency paired with j by T: 128 - j, and 64 for j = 0.
__host__ __device__ __forceinline__ int mirror(int j) { return j == 0 ? 64 : kN - j; }
// The contraction position of sample or frequency J < 64 (side 0) or mirror(J) (side 1): the inverse of bf16_sigma.
__host__ __device__ __forceinline__ constexpr int position_of(int J, int side) { return 2 * (J & ~3) + 4 * side + (J & 3); }

// Writes 8 consecutive K (or MN) values of one row, split into bf16 hi and lo, into planes hi_plane and hi_plane + 1.
__device__ __forceinline__ void store_split8(uint8_t *planes, int hi_plane, uint32_t off, const float (&v)[8]) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; i++) split_bf16x2(v[2 * i], v[2 * i + 1], h[i], l[i]);
    *reinterpret_cast<uint4 *>(planes + hi_plane * kPlaneBytes + off) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(planes + (hi_plane + 1) * kPlaneBytes + off) = make_uint4(l[0], l[1], l[2], l[3]);
}

// The 24 MMAs of one plane: D (columns d_col) = A (hi at columns 0.., lo at 64..) * B (planes at b_hi, b_hi + one plane).  The
// accumulator cuts off what its exponent leaves no room for, so a step's small products come first and the contraction runs
// towards the centre of the probe and of the pattern (position 0).  After four iterations of 576 positions the object is
// 1.9e-7 from 64 bits so and 2.9e-7 in rising order with the large products first, the errors 3.5e-8 and 7.3e-7; the time is
// the same within 1 %.  Unrolled by two: more spills in the issuing thread's registers.
__device__ __forceinline__ void issue_plane(uint32_t tmem, uint32_t d_col, uint32_t b_hi, uint32_t idesc) {
    constexpr uint32_t kStep = (2 * kLBO) >> 4;
    const uint64_t top = smem_desc(b_hi, kLBO, kSBO) + (kN / 16 - 1) * kStep;
    const uint32_t a_hi = tmem + kCSigma + 8 * (kN / 16 - 1);
#pragma unroll 2
    for (int s = 0; s < kN / 16; s++) {
        const uint64_t dh = top - s * kStep;
        const uint32_t ah = a_hi - 8 * s;
        mma_ts(tmem + d_col, ah, dh + (kPlaneBytes >> 4), idesc, s > 0 ? 1u : 0u);
        mma_ts(tmem + d_col, ah + 64, dh, idesc, 1u);
        mma_ts(tmem + d_col, ah, dh, idesc, 1u);
    }
}

// Lane `row`'s kCols columns of one result (from taddr) -> kCols consecutive K of row `row` of a K-major B plane pair.
__device__ __forceinline__ void readout_kmajor(uint32_t taddr, uint8_t *planes, int hi_plane, int row, int k0) {
    float a[kCols];
#pragma unroll
    for (int c = 0; c < kCols / 16; c++) tmem_ld16(taddr + 16 * c, *reinterpret_cast<float(*)[16]>(a + 16 * c));
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < kCols / 8; c++) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = a[8 * c + i];
        store_split8(planes, hi_plane, kmajor_offset(row, k0 + 8 * c), v);
    }
}

// T on the columns of one lane: raw pairs (zc, zs) = columns (2J, 2J+1) -> the values at J (y0) and mirror(J) (y1).
// Forward: y0 = zc - i zs, y1 = zc + i zs; inverse the other way round; J = 0 passes (z0, z1) through.
template <bool kInverse>
__device__ __forceinline__ void combine(float zr, float zi, float sr, float si, bool passthrough, float &y0r, float &y0i,
                                        float &y1r, float &y1i) {
    if (passthrough) {
        y0r = zr; y0i = zi; y1r = sr; y1i = si;
    } else if (!kInverse) {
        y0r = zr + si; y0i = zi - sr; y1r = zr - si; y1i = zi + sr;
    } else {
        y0r = zr - si; y0i = zi + sr; y1r = zr + si; y1i = zi - sr;
    }
}

// The column index J of a thread's value i (0..3) of sub-block u: its column group g and parity h (= L & 1) own the
// raw result columns kCols g .. kCols g + kCols - 1, i.e. the column pairs (2J, 2J + 1) of J = (kCols / 2) g + 0 ..
// kCols / 2 - 1, of which it keeps, after the exchange with lane L ^ 1, the half of parity h.
__host__ __device__ __forceinline__ int column_of(int g, int h, int u, int i) {
    return (kCols / 2) * g + (kCols / 4) * h + 4 * u + i;
}

// A thread's part in T on the row pair (2j, 2j + 1), whose rows lanes L and L ^ 1 hold.  The odd lane turns its row by -i
// (forward) or i (inverse) before the exchange, so that T is y0 = own[0] mine + theirs[0] theirs and
// y1 = own[1] mine + theirs[1] theirs with factors 0, 1 and -1, alike for re and im.  For j = 0 T passes the rows through,
// so there y1 comes out turned: the user of y1 turns it back.
struct RowPair {
    float2 own[2], theirs[2];
};
__device__ __forceinline__ RowPair row_pair(int j, int h) {
    RowPair k;
    const float a = j == 0 && h ? 0.f : 1.f, b = j == 0 && !h ? 0.f : 1.f;
    const float c = j == 0 ? (h ? 1.f : 0.f) : (h ? -1.f : 1.f), d = j == 0 ? (h ? 0.f : 1.f) : (h ? 1.f : -1.f);
    k.own[0] = make_float2(a, a); k.theirs[0] = make_float2(b, b);
    k.own[1] = make_float2(c, c); k.theirs[1] = make_float2(d, d);
    return k;
}

// One thread's 16 values of a combined stage result for sub-block u: T on the columns (in the thread), then the
// exchange with lane L ^ 1, then T on the row pair (2j, 2j + 1).  out[side][4 s + i] is the value at row
// (side ? mirror(j) : j) and column (s ? mirror(J) : J), J = column_of(g, h, u, i), h = L & 1; at j = 0 side 1 is turned
// by -i (forward) or i (inverse).
template <bool kInverse>
__device__ __forceinline__ void combined_block(uint32_t lane_addr, int g, int u, int h, const RowPair &k,
                                               float (&out_re)[2][8], float (&out_im)[2][8]) {
    float r0[8], r1[8], i0[8], i1[8];  // raw columns of parity sets 0 and 1: kCols g + (kCols / 2) h' + 8 u .. + 8
    tmem_ld8(lane_addr + kSlotRe + kCols * g + 8 * u, r0);
    tmem_ld8(lane_addr + kSlotRe + kCols * g + kCols / 2 + 8 * u, r1);
    tmem_ld8(lane_addr + kSlotIm + kCols * g + 8 * u, i0);
    tmem_ld8(lane_addr + kSlotIm + kCols * g + kCols / 2 + 8 * u, i1);
    tmem_wait_ld();
    // T on the columns for both parity sets: a / b [s][i]
    float ar[2][4], ai[2][4], br[2][4], bi[2][4];
    const bool first = g == 0 && u == 0;  // J = 0 sits at i = 0 of parity set 0
#pragma unroll
    for (int i = 0; i < 4; i++) {
        combine<kInverse>(r0[2 * i], i0[2 * i], r0[2 * i + 1], i0[2 * i + 1], first && i == 0, ar[0][i], ai[0][i],
                          ar[1][i], ai[1][i]);
        combine<kInverse>(r1[2 * i], i1[2 * i], r1[2 * i + 1], i1[2 * i + 1], false, br[0][i], bi[0][i], br[1][i],
                          bi[1][i]);
    }
    // keep the own parity set, send the other: afterwards m is lane L's row (turned when odd) and t lane L ^ 1's, both
    // for the columns of set h
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            float mr[2], mi[2], tr[2], ti[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float a_r = ar[s][i + e], a_i = ai[s][i + e], b_r = br[s][i + e], b_i = bi[s][i + e];
                mr[e] = h ? (kInverse ? -b_i : b_i) : a_r;
                mi[e] = h ? (kInverse ? b_r : -b_r) : a_i;
                tr[e] = __shfl_xor_sync(0xffffffffu, h ? (kInverse ? -a_i : a_i) : b_r, 1);
                ti[e] = __shfl_xor_sync(0xffffffffu, h ? (kInverse ? a_r : -a_r) : b_i, 1);
            }
            const float2 m_r = make_float2(mr[0], mr[1]), m_i = make_float2(mi[0], mi[1]);
            const float2 t_r = make_float2(tr[0], tr[1]), t_i = make_float2(ti[0], ti[1]);
#pragma unroll
            for (int side = 0; side < 2; side++) {
                const float2 y_r = pfma(k.own[side], m_r, pmul(k.theirs[side], t_r));
                const float2 y_i = pfma(k.own[side], m_i, pmul(k.theirs[side], t_i));
                out_re[side][4 * s + i] = y_r.x; out_re[side][4 * s + i + 1] = y_r.y;
                out_im[side][4 * s + i] = y_i.x; out_im[side][4 * s + i + 1] = y_i.y;
            }
        }
}

__device__ __forceinline__ float rsqrt_normal(float x) {  // x normal: rsqrtf without its subnormal branch
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// The projection of eight frequencies (re, im) of one row, in place: (A / |F| - 1) F / n, at F = 0 the amplitude over n.
// |F| and A / |F| come through one reciprocal square root.  `turned` (row 64): the values are -i F; F' = i x (projected)
// leaves its real part in im and its imaginary part in re.
__device__ __forceinline__ void project_row(float (&re)[8], float (&im)[8], const float4 &lo, const float4 &hi, float inv_n,
                                            bool turned, float2 &err) {
    const float am[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    float2 m2[4];
    bool normal = true;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const float2 r = make_float2(re[2 * e], re[2 * e + 1]), i = make_float2(im[2 * e], im[2 * e + 1]);
        m2[e] = pfma(r, r, pmul(i, i));
        normal = normal && m2[e].x >= 1.17549435e-38f && m2[e].y >= 1.17549435e-38f;
    }
    const float sign = turned ? -inv_n : inv_n;
    if (normal) {
        const float2 minus_one = make_float2(-1.f, -1.f);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float2 r = make_float2(re[2 * e], re[2 * e + 1]), i = make_float2(im[2 * e], im[2 * e + 1]);
            const float2 a = make_float2(am[2 * e], am[2 * e + 1]);
            const float2 inv = make_float2(rsqrt_normal(m2[e].x), rsqrt_normal(m2[e].y));
            const float2 miss = psub(a, pmul(m2[e], inv));
            err = pfma(miss, miss, err);
            const float2 c = pfma(a, inv, minus_one);
            const float2 nr = pmul(r, pmul(c, make_float2(inv_n, inv_n))), ni = pmul(i, pmul(c, make_float2(sign, sign)));
            re[2 * e] = nr.x; re[2 * e + 1] = nr.y;
            im[2 * e] = ni.x; im[2 * e + 1] = ni.y;
        }
    } else {  // a zero, a subnormal or a NaN among them
#pragma unroll
        for (int e = 0; e < 8; e++) {
            const float m = (e & 1) ? m2[e >> 1].y : m2[e >> 1].x;
            const bool nonzero = m > 0.f;
            const float inv = rsqrtf(m), miss = am[e] - (nonzero ? m * inv : 0.f), c = fmaf(am[e], inv, -1.f);
            if (e & 1) err.y = fmaf(miss, miss, err.y);
            else err.x = fmaf(miss, miss, err.x);
            const float zero = am[e] * inv_n;
            re[e] = nonzero ? re[e] * (c * inv_n) : turned ? 0.f : zero;
            im[e] = nonzero ? im[e] * (c * sign) : turned ? zero : 0.f;
        }
    }
}

// The exit wave of one position: warp w takes rows kRowsPerWarp w .. + kRowsPerWarp - 1.  A lane holds the columns 2i,
// 2i + 1 of both halves of a row (i its index), the lower half first in lanes below 16 and second above, which keeps the
// stores below free of bank conflicts: 256 contiguous bytes of the object row and of the probe row per half-warp and load.
struct ExitWave {
    const float2 *S, *object;  // S: the probe's row row0
    int row0, y0, cc, object_rows, OC;
    bool aligned;
};
__device__ __forceinline__ ExitWave exit_wave(const Bf16Args &a, int p, int warp) {
    ExitWave w;
    w.row0 = kRowsPerWarp * warp;  // the warp's first patch row
    w.S = a.shifted + (size_t)a.scan.cls[p] * (kN * kN) + w.row0 * kN;
    w.object = a.object; w.object_rows = a.object_rows; w.OC = a.object_columns;
    // patch rows row0 .. row0 + kRowsPerWarp - 1 are object rows y0 .. (wrapped), y0 = rr + row0, or rr + row0 - 128 past
    // the centre row (a warp's rows never straddle it)
    w.y0 = a.scan.rr[p] + (w.row0 < kN / 2 ? w.row0 : w.row0 - kN);
    w.cc = a.scan.cc[p];
    // the patch row is the object row segment [cc - 64, cc + 64) (its columns 64..127, then 0..63): one aligned float4
    // per lane and half when it does not wrap and starts on an even complex
    w.aligned = w.cc >= kN / 2 && w.cc + kN / 2 <= w.OC && ((w.cc | w.OC) & 1) == 0;
    return w;
}
// The loads of kBatch rows from row0 + b0 of an aligned patch: 4 kBatch in flight.
__device__ __forceinline__ void exit_load(const ExitWave &w, int b0, int lane, float4 (&sv)[2 * kBatch],
                                          float4 (&ov)[2 * kBatch]) {
    const int low = 2 * lane, high = 2 * lane + kN / 2;
    const int ca = lane < 16 ? low : high, cb = lane < 16 ? high : low;
    const int xa = ca < kN / 2 ? ca : ca - kN, xb = cb < kN / 2 ? cb : cb - kN;
#pragma unroll
    for (int i = 0; i < kBatch; i++) {
        const float2 *orow = w.object + (size_t)wrap_once(w.y0 + b0 + i, w.object_rows) * w.OC + w.cc;
        sv[2 * i] = __ldg(reinterpret_cast<const float4 *>(w.S + (b0 + i) * kN + ca));
        sv[2 * i + 1] = __ldg(reinterpret_cast<const float4 *>(w.S + (b0 + i) * kN + cb));
        ov[2 * i] = __ldg(reinterpret_cast<const float4 *>(orow + xa));
        ov[2 * i + 1] = __ldg(reinterpret_cast<const float4 *>(orow + xb));
    }
}
// Stage 1's B operand of one row: n = the row's and k = the columns' contraction position.  The lower pair (2i, 2i + 1)
// lies on two consecutive k; of the upper half 2i + 65 pairs with 2i + 66, the next lane's.
__device__ __forceinline__ void exit_store(uint8_t *planes, int row, int lane, const float4 &sa, const float4 &oa,
                                           const float4 &sb, const float4 &ob) {
    const bool low = lane < 16;
    float a0r = sa.x * oa.x - sa.y * oa.y, a0i = sa.x * oa.y + sa.y * oa.x;
    const float a1r = sa.z * oa.z - sa.w * oa.w, a1i = sa.z * oa.w + sa.w * oa.z;
    float b0r = sb.x * ob.x - sb.y * ob.y, b0i = sb.x * ob.y + sb.y * ob.x;
    const float b1r = sb.z * ob.z - sb.w * ob.w, b1i = sb.z * ob.w + sb.w * ob.z;
    const float nr = __shfl_sync(0xffffffffu, low ? b0r : a0r, (lane + 1) & 31);
    const float ni = __shfl_sync(0xffffffffu, low ? b0i : a0i, (lane + 1) & 31);
    a0r = low ? a0r : nr; a0i = low ? a0i : ni;
    b0r = low ? nr : b0r; b0i = low ? ni : b0i;
    const int n = row <= kN / 2 ? position_of(row & (kN / 2 - 1), row >> 6) : position_of(kN - row, 1);
    const int kl = position_of(2 * lane, 0), ku = position_of(62 - 2 * lane, 1);
    const uint32_t offset_a = kmajor_offset(n, low ? kl : ku), offset_b = kmajor_offset(n, low ? ku : kl);
    uint32_t rh, rl, ih, il;
    split_bf16x2(a0r, a1r, rh, rl);
    split_bf16x2(a0i, a1i, ih, il);
    *reinterpret_cast<uint32_t *>(planes + (kReHi + 0) * kPlaneBytes + offset_a) = rh;
    *reinterpret_cast<uint32_t *>(planes + (kReHi + 1) * kPlaneBytes + offset_a) = rl;
    *reinterpret_cast<uint32_t *>(planes + (kImHi + 0) * kPlaneBytes + offset_a) = ih;
    *reinterpret_cast<uint32_t *>(planes + (kImHi + 1) * kPlaneBytes + offset_a) = il;
    split_bf16x2(b0r, b1r, rh, rl);
    split_bf16x2(b0i, b1i, ih, il);
    *reinterpret_cast<uint32_t *>(planes + (kReHi + 0) * kPlaneBytes + offset_b) = rh;
    *reinterpret_cast<uint32_t *>(planes + (kReHi + 1) * kPlaneBytes + offset_b) = rl;
    *reinterpret_cast<uint32_t *>(planes + (kImHi + 0) * kPlaneBytes + offset_b) = ih;
    *reinterpret_cast<uint32_t *>(planes + (kImHi + 1) * kPlaneBytes + offset_b) = il;
}
// Every row, the first batch of an aligned patch loaded before.
__device__ __forceinline__ void exit_rows(const ExitWave &w, uint8_t *planes, int lane, float4 (&sv)[2 * kBatch],
                                          float4 (&ov)[2 * kBatch]) {
    if (w.aligned) {
#pragma unroll
        for (int b0 = 0; b0 < kRowsPerWarp; b0 += kBatch) {
            if (b0 > 0) exit_load(w, b0, lane, sv, ov);
#pragma unroll
            for (int i = 0; i < kBatch; i++)
                exit_store(planes, w.row0 + b0 + i, lane, sv[2 * i], ov[2 * i], sv[2 * i + 1], ov[2 * i + 1]);
        }
        return;
    }
    // near the object's edge (or an odd row length): complex by complex, each column wrapped
#pragma unroll 1
    for (int i = 0; i < kRowsPerWarp; i++) {
        const float2 *orow = w.object + (size_t)wrap_once(w.y0 + i, w.object_rows) * w.OC;
        float4 s2[2], o2[2];
#pragma unroll
        for (int v = 0; v < 2; v++) {
            const int c = 2 * lane + ((lane < 16) == (v == 0) ? 0 : kN / 2), x = w.cc + (c < kN / 2 ? c : c - kN);
            s2[v] = __ldg(reinterpret_cast<const float4 *>(w.S + i * kN + c));
            const float2 o0 = __ldg(orow + wrap_once(x, w.OC)), o1 = __ldg(orow + wrap_once(x + 1, w.OC));
            o2[v] = make_float4(o0.x, o0.y, o1.x, o1.y);
        }
        exit_store(planes, w.row0 + i, lane, s2[0], o2[0], s2[1], o2[1]);
    }
}

__global__ void __launch_bounds__(kLaunch, 1) bf16_position_kernel(Bf16Args a) {
    extern __shared__ __align__(1024) uint8_t planes[];  // 4 x 36.5 KB: the B operand, then 64 KB of amplitudes
    __shared__ uint64_t mbar[2];                         // completion of the re / im plane's MMAs
    __shared__ uint64_t amp_bar;                         // arrival of the next position's amplitudes
    __shared__ uint64_t ready[2];                        // the working warps' arrivals, by turns
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int q = warp & 3, g = warp >> 2;
    const int L = 32 * q + lane;      // this thread's TMEM lane
    const int j = L >> 1, h = L & 1;  // its row pair and parity
    if (warp == 0) {
        tmem_alloc(&tmem_base, 512);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&mbar[0], 1);
        mbar_init(&mbar[1], 1);
        mbar_init(&amp_bar, 1);
        mbar_init(&ready[0], kWarps);
        mbar_init(&ready[1], kWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmem_base;
    const uint32_t lane_addr = tmem_addr(tmem, 32 * q, 0);
    const uint32_t smem = smem_u32(planes);
    float4 *amp_smem = reinterpret_cast<float4 *>(planes + 4 * kPlaneBytes);
    if (tid == 0)
        bulk_load(amp_smem, a.amplitudes + (size_t)(a.first + blockIdx.x) * (kN * kN), kN * kN * 4, &amp_bar);
    const int steps = (a.count - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // this CTA's positions, >= 1
    uint32_t phase = 0u;    // bit x: parity to wait for of plane x's barrier (working warps), of ready[x] (issuer)
    bool bad = false;       // a wait ran out: this thread stops
    if (warp >= kWarps) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 32;");
        if (tid == kThreads) {
            auto wait_ready = [&](int x) {
                bad = bad || !mbar_wait(&ready[x], (phase >> x) & 1u, kWaitLimit);
                phase ^= 1u << x;
                fence_after_sync();
                return !bad;
            };
            uint32_t commits = 0u;  // bit x: parity of the number of plane x's products issued
            auto issue = [&](int plane, uint32_t slot, uint32_t idesc) {
                issue_plane(tmem, slot, smem + (plane ? kImHi : kReHi) * kPlaneBytes, idesc);
                mma_commit(&mbar[plane]);
                commits ^= 1u << plane;
            };
            int copies = 1;
            for (int i = 0; i < steps && !bad; i++) {
                if (wait_ready(0)) issue(0, kSlotNext, kIdescK);  // stage 1
                if (wait_ready(1)) issue(1, kSlotIm, kIdescK);
                if (wait_ready(0)) issue(0, kSlotRe, kIdescK);    // stage 2
                if (wait_ready(1)) issue(1, kSlotIm, kIdescK);
                if (wait_ready(0)) {                              // stage 3; every warp has read this position's amplitudes
                    issue(0, kSlotRe, kIdescMN);
                    issue(1, kSlotIm, kIdescMN);
                    if (i + 1 < steps) {
                        copies++;
                        bulk_load(amp_smem, a.amplitudes + (size_t)(a.first + blockIdx.x + (i + 1) * gridDim.x) * (kN * kN),
                                  kN * kN * 4, &amp_bar);
                    }
                }
                if (wait_ready(1)) issue(0, kSlotRe, kIdescK);    // stage 4
                if (wait_ready(0)) issue(1, kSlotIm, kIdescK);
            }
            // the last products and copy end before the columns and the CTA go (at once, unless a wait ran out)
            for (int x = 0; x < 2; x++) mbar_wait(&mbar[x], ((commits >> x) & 1u) ^ 1u, kWaitLimit);
            mbar_wait(&amp_bar, (copies - 1) & 1, kWaitLimit);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
        uint32_t amp_phase = 0;
        // C_sigma hi and lo into tensor memory: plane v at columns 64 v, lane m, column c = the bf16 pair
        // (k = 2c, 2c + 1) of row m
#pragma unroll 1
        for (int v = 0; v < 2; v++) {
            constexpr int kw = 64 / kGroups;  // bf16 pairs of the plane's row per thread
            const uint32_t *src = reinterpret_cast<const uint32_t *>(a.c_planes + ((size_t)v * kN + L) * kN) + kw * g;
#pragma unroll
            for (int c0 = 0; c0 < kw; c0 += 8) {
                float r[8];
#pragma unroll
                for (int i = 0; i < 8; i++) r[i] = __uint_as_float(src[c0 + i]);
                tmem_st8(lane_addr + 64 * v + kw * g + c0, r);
            }
        }
        tmem_wait_st();
        // waits for plane x's product
        auto wait_plane = [&](int x) {
            bad = __any_sync(0xffffffffu, bad || !mbar_wait(&mbar[x], (phase >> x) & 1u, kWaitLimit));
            phase ^= 1u << x;
            fence_after_sync();
        };
        // hands this warp's B-operand writes and tensor-memory reads to the issuer
        auto publish = [&](int x) {
            fence_proxy_async();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[x]);
        };
        const float inv_n = 1.0f / (float)(kN * kN);
        const RowPair pair = row_pair(j, h);
        int p = a.first + blockIdx.x;
        float4 sv[2 * kBatch], ov[2 * kBatch];
        {  // stage 1 of the first position
            const ExitWave w = exit_wave(a, p, warp);
            if (w.aligned) exit_load(w, 0, lane, sv, ov);
            exit_rows(w, planes, lane, sv, ov);
            publish(0);
            publish(1);
        }
        for (int step = 0; step < steps && !bad; step++, p += gridDim.x) {
            // ---- stage 2: B[n = raw c][k = pos(r)] = D1, each plane as soon as its stage-1 product is done
            wait_plane(0);
            readout_kmajor(lane_addr + kSlotNext + kCols * g, planes, kReHi, L, kCols * g);
            publish(0);
            wait_plane(1);
            readout_kmajor(lane_addr + kSlotIm + kCols * g, planes, kImHi, L, kCols * g);
            publish(1);
            // ---- projection on F (rows kr = j, mirror(j); this thread's 16 columns kc); stage 3: B = F', MN-major
            wait_plane(0);
            wait_plane(1);
            bad = __any_sync(0xffffffffu, bad || !mbar_wait(&amp_bar, amp_phase, kWaitLimit));
            amp_phase ^= 1u;
            {
                // the squared residual of this thread's 32 frequencies in FP32 (two packed lanes), then in FP64 over the
                // threads, warps and positions, as the reference's Float path sums a pattern in Float and the patterns in
                // Double (PtychographySingle.swift:157-172)
                float2 errv = make_float2(0.f, 0.f);
#pragma unroll 1
                for (int u = 0; u < kSub; u++) {
                    float4 am4[4];
#pragma unroll
                    for (int e = 0; e < 4; e++) am4[e] = amp_smem[(4 * u + e) * kThreads + tid];
                    float fr[2][8], fi[2][8];
                    combined_block<false>(lane_addr, g, u, h, pair, fr, fi);
#pragma unroll
                    for (int side = 0; side < 2; side++) {
                        const bool turned = side == 1 && j == 0;
                        project_row(fr[side], fi[side], am4[2 * side], am4[2 * side + 1], inv_n, turned, errv);
                        const uint32_t off = mnmajor_offset(position_of(j, side), kCols * g + (kCols / 2) * h + 8 * u);
                        store_split8(planes, turned ? kImHi : kReHi, off, fr[side]);
                        store_split8(planes, turned ? kReHi : kImHi, off, fi[side]);
                    }
                }
                double err = (double)errv.x + (double)errv.y;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) err += __shfl_down_sync(0xffffffffu, err, o);
                if (lane == 0) a.error[(size_t)p * (kThreads / 32) + warp] = err;
            }
            publish(0);
            // ---- stage 4: B[n = raw r][k = pos(kc)] = D3
            wait_plane(0);
            readout_kmajor(lane_addr + kSlotRe + kCols * g, planes, kReHi, L, kCols * g);
            publish(1);
            wait_plane(1);
            readout_kmajor(lane_addr + kSlotIm + kCols * g, planes, kImHi, L, kCols * g);
            publish(0);
            // ---- stage 1 of the next position: its first loads fly while stage 4 finishes, and its re product runs behind
            // the residual's read-out
            const bool more = step + 1 < steps;
            ExitWave w{};
            if (more) {
                w = exit_wave(a, p + gridDim.x, warp);
                if (w.aligned) exit_load(w, 0, lane, sv, ov);
            }
            wait_plane(0);
            wait_plane(1);
            if (more) {
                exit_rows(w, planes, lane, sv, ov);
                publish(0);
            }
            // ---- dpsi[r][c]: columns c = j, mirror(j) of this lane pair, rows r = J, mirror(J)
            {
                float2 *out = a.dpsi + (size_t)(p - a.dpsi_first) * (kN * kN);
#pragma unroll 1
                for (int u = 0; u < kSub; u++) {
                    float dr[2][8], di[2][8];
                    combined_block<true>(lane_addr, g, u, h, pair, dr, di);
#pragma unroll
                    for (int side = 0; side < 2; side++) {
                        const int c = side ? mirror(j) : j;
                        const bool turned = side == 1 && j == 0;
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const int J = column_of(g, h, u, e & 3);
                            const int r = (e >> 2) ? mirror(J) : J;
                            out[r * kN + c] = make_float2(turned ? di[side][e] : dr[side][e],
                                                          turned ? -dr[side][e] : di[side][e]);
                        }
                    }
                }
            }
            if (more) publish(1);
        }
    }
    if (bad) *a.fault = 1;
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

// [position][row][column] -> [position][e4][thread][4]: thread T's float4 e4 = 4 u + 2 side + s holds the amplitudes of
// row (side ? mirror(j) : j), columns (s ? mirror(J) : J), J = column_of(g, h, u, i), i = 0..3, for T's lane pair j,
// parity h and column group g.
__global__ void permute_bf16_amplitudes_kernel(const float *in, float *out, long long positions) {
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    if (idx >= positions * kN * kN) return;
    const long long p = idx / (kN * kN);
    const int rem = (int)(idx - p * kN * kN);
    const int i = rem & 3, T = (rem >> 2) & (kThreads - 1), e4 = (rem >> 2) / kThreads;
    const int u = e4 >> 2, side = (e4 >> 1) & 1, s = e4 & 1;
    const int w = T >> 5, L = 32 * (w & 3) + (T & 31), g = w >> 2;
    const int jj = L >> 1, h = L & 1;
    const int J = column_of(g, h, u, i);
    const int kc = s ? mirror(J) : J, kr = side ? mirror(jj) : jj;
    out[idx] = in[p * kN * kN + kr * kN + kc];
}

size_t bf16_smem() { return 4 * (size_t)kPlaneBytes + (size_t)kN * kN * sizeof(float); }

}  // namespace

bool bf16_applicable(int rows, int columns) { return rows == kN && columns == kN; }
int bf16_partials_per_position() { return kThreads / 32; }

// Stage 3's contraction position pos = kCols g + (kCols / 2) h + 8 u + 4 s + i holds the frequency
// s ? mirror(J) : J, J = column_of(g, h, u, i): the order in which a thread stores its projected values.
int bf16_sigma(int pos) {
    const int g = pos / kCols, h = (pos % kCols) / (kCols / 2), r = pos % (kCols / 2);
    const int u = r >> 3, s = (r >> 2) & 1, i = r & 3;
    const int J = column_of(g, h, u, i);
    return s ? mirror(J) : J;
}

cudaError_t configure_bf16() {
    int device = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    if ((size_t)optin < bf16_smem() + 1024) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(bf16_position_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bf16_smem());
}

cudaError_t launch_bf16(const Bf16Args &a, int ctas, cudaStream_t s) {
    if (a.count <= 0) return cudaSuccess;
    const int grid = a.count < ctas ? a.count : ctas;
    bf16_position_kernel<<<grid, kLaunch, bf16_smem(), s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_permute_bf16_amplitudes(const float *in, float *out, long long positions, cudaStream_t s) {
    const long long total = positions * kN * kN;
    permute_bf16_amplitudes_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(in, out, positions);
    return cudaGetLastError();
}

}  // namespace cubo
