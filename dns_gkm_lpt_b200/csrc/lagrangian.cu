// Lagrangian side of the step on sm_100a: velocity splines, tricubic
// evaluation, Heun advection and the PrintStats reductions.
//
// Reference path replaced: generateSplines (src/update.cpp:1235-1247) ->
// get_bsplinep (src/Interpolation.cpp:3-31) -> einspline; Particle::
// updatePosition / track (src/ParticleTrack.cpp:42-73); the velocity part of
// getParticleProp (:99-113); PrintStats (src/update.cpp:688-842).
//
// Splines are uniform cubic B-splines built as batched 1-D line solves along
// each axis (axis 0 = y first, then x, then z).  Two end conditions:
//   natural_ghost3: the reference's grid (nt points from -3dx+dx/2, f''=0 at
//                   both ends), coefficients c_{-1}..c_{N} (N+2 per axis);
//   periodic:       the n interior cell centres, cyclic rows, stored N+3 per
//                   axis with wrapped copies so a 4-point window never wraps.
// The line solve and the evaluation use rounding-explicit intrinsics in the
// order of the CPU oracle, so both produce the same bits.  A solve's divisions
// by the pivots are multiplications by their reciprocals with a correction that
// rounds as the division does (pivot_div.cuh).  Lines short enough for a few
// warps of them per SM are solved in shared memory (resident_*), longer ones
// streamed through global memory (line_solve, pass2_group).
#include "gkm_internal.h"
#include "pivot_div.cuh"

#include <algorithm>

namespace gkm {
namespace {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

// One line: f (N points, stride fs) -> c (N+pad values, stride cs).
// The recurrences are sequential, but their inputs are not: the loops fetch U inputs ahead (data
// in the forward sweeps, those or the forward results in the backward sweeps) so that many loads are in
// flight per thread; the arithmetic and its order are unchanged.  Pass 1 stores one forward value in U, so
// longer batches pay there: of 8 / 16 / 24 points three components took 1.304 / 1.260 / 1.276 ms at 256^3, 8.89 /
// 8.51 / 8.55 at 512^3; one component per launch (FP32 coefficients, 512^3) 4 and 4 points in passes 0
// and 1 took 9.10 ms, 4 and 8 8.63, 4 and 16 8.67, 8 and 12 8.50.
constexpr int kLineBatch0 = 8, kLineBatch1Batched = 16, kLineBatch1Single = 12;
// the component-batched pass kernels hold six 128-thread CTAs per SM (80 registers): more lines
// in flight than the compiler's own choice (96-112 registers; 256^3 splines 1.57 -> 1.49 ms),
// where eight (64 registers) spill the fetch-ahead values
constexpr int kPassCtasPerSm = 6;

// The pivots and multipliers of the line solves reach the fixed point of d = 4 - 1/d to the last
// bit within 17 rows, whatever the number of points and the ends; from this row on (but for the
// last pivot of periodic lines) they are held in registers.
constexpr int kPivotRows = 24;

// x_i = (cv_u - x_{i+1}) / dp_i, i = i0 - u: the U rows of a back substitution down from i0
// (below the line's last row), solutions into cv.  False, with x as it was, where a numerator is
// out of pivot_quotient's range: the caller repeats the rows with divisions.
template <int U>
__device__ __forceinline__ bool back_rows(double (&cv)[U], int i0, const SplineTables& tb, double d_inf, double r_inf,
                                          double& x)
{
    const bool fixed = i0 - U + 1 >= kPivotRows;
    double y = x;
    bool ok = true;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const double d = fixed ? d_inf : tb.dp[i0 - u], r = fixed ? r_inf : tb.mt[i0 - u + 1];
        const double a = sub(cv[u], y);
        ok = ok && pivot_in_range(a);
        y = pivot_quotient(a, d, r);
        cv[u] = y;
    }
    if (ok) x = y;
    return ok;
}
// the fixed point, taken at row kPivotRows; shorter lines (last row N - 2, periodic N - 1) have no row
// that uses it
__device__ __forceinline__ void fixed_pivots(int N, const SplineTables& tb, double& d_inf, double& r_inf)
{
    const bool reached = N - 2 >= kPivotRows;
    d_inf = reached ? tb.dp[kPivotRows] : 0.0;
    r_inf = reached ? tb.mt[kPivotRows] : 0.0;
}

// IN_PLACE: the forward value of point i lies in slot i, where the input of point i was, instead of slot
// i + 1, so c may be the storage f reads (same stride) as long as slots N .. N+pad-1 exist.
// REREAD: the forward sweep stores one value in U, and the backward sweep forms the others again
// from the inputs: the line is read twice and written once instead of twice.  For inputs that cost
// no more than their load: with passes 1 and 2 so, all passes of three components went 1.44 -> 1.31 ms at
// 256^3, 9.99 -> 8.90 at 512^3.  Pass 0's inputs cost a division each (1.31 -> 1.40 ms).
template <int U, bool IN_PLACE, bool REREAD, class Src>
__device__ void line_solve(const Src& f, int N, int periodic, const SplineTables& tb, double* c, long long cs)
{
    double d_inf, r_inf;
    fixed_pivots(N, tb, d_inf, r_inf);
    const int lo = periodic ? 0 : 1, hi = periodic ? N - 1 : N - 2;   // the points solved for
    const double c0 = periodic ? 0.0 : f(0), cl = periodic ? 0.0 : f(N - 1);
    auto fwd = [&](int i) -> double& { return c[(long long)(i + (IN_PLACE ? 0 : 1)) * cs]; };
    double rp = 0.0;
    auto eliminate = [&](int i, double fi, double m) {
        double r = mul(6.0, fi);
        if (!periodic && i == 1) r = sub(r, c0);
        if (!periodic && i == N - 2) r = sub(r, cl);
        rp = (i == lo) ? r : sub(r, mul(m, rp));
    };
    int top = lo;   // batches of U points, the last point not among them, then the others one by one
    for (; top + U - 1 < hi; top += U) {
        double fv[U];
#pragma unroll
        for (int u = 0; u < U; u++) fv[u] = f(top + u);
#pragma unroll
        for (int u = 0; u < U; u++) {
            eliminate(top + u, fv[u], top > kPivotRows ? r_inf : tb.mt[top + u]);
            if (!REREAD || u == 0) fwd(top + u) = rp;
        }
    }
#pragma unroll 1
    for (int i = top; i <= hi; i++) {
        eliminate(i, f(i), tb.mt[i]);
        fwd(i) = rp;
    }
    double x = 0.0, xl = 0.0;
    if (hi >= lo) {
        x = xl = __ddiv_rn(rp, tb.dp[hi]);
        c[(long long)(hi + 1) * cs] = x;
    }
    auto divide = [&](int i) {
        x = __ddiv_rn(sub(fwd(i), x), tb.dp[i]);
        c[(long long)(i + 1) * cs] = x;
    };
#pragma unroll 1
    for (int i = hi - 1; i >= top; i--) divide(i);
    for (int s = top - U; s >= lo; s -= U) {   // points s + U - 1 down to s
        double cv[U];
        const bool fixed = s > kPivotRows;
        cv[U - 1] = fwd(s);
#pragma unroll
        for (int u = 1; u < U; u++) cv[U - 1 - u] = REREAD ? f(s + u) : fwd(s + u);
        if (REREAD) {
#pragma unroll
            for (int u = 1; u < U; u++)
                cv[U - 1 - u] = sub(mul(6.0, cv[U - 1 - u]), mul(fixed ? r_inf : tb.mt[s + u], cv[U - u]));
        }
        if (back_rows<U>(cv, s + U - 1, tb, d_inf, r_inf, x)) {
#pragma unroll
            for (int u = 0; u < U; u++) c[(long long)(s + U - u) * cs] = cv[u];
        } else {
            if (REREAD) {
                double r = fwd(s);
#pragma unroll 1
                for (int i = s + 1; i < s + U; i++) {
                    r = sub(mul(6.0, f(i)), mul(tb.mt[i], r));
                    fwd(i) = r;
                }
            }
#pragma unroll 1
            for (int i = s + U - 1; i >= s; i--) divide(i);
        }
    }
    if (!periodic) {
        // x: the solution of point 1, xl: of point N - 2 (the ends themselves when there is none)
        c[cs] = c0;
        c[(long long)N * cs] = cl;
        c[0] = sub(2.0 * c0, hi >= lo ? x : cl);
        c[(long long)(N + 1) * cs] = sub(2.0 * cl, hi >= lo ? xl : c0);
    } else {
        const double fac = __ddiv_rn(add(x, mul(-0.25, xl)), tb.denom);
        for (int i = 0; i < N; i++) c[(long long)(i + 1) * cs] = sub(c[(long long)(i + 1) * cs], mul(fac, tb.z[i]));
        c[0] = c[(long long)N * cs];
        c[(long long)(N + 1) * cs] = c[cs];
        c[(long long)(N + 2) * cs] = c[2 * cs];
    }
}

// Data of a spline at ghost-layout cell idx (generateSplines, src/update.cpp:1200-1210,1239-1241):
// q = 1..3 velocity rho u_q / rho; q = kSrcDensity rho; q = kSrcPressure
// (rho (gam-1)) (rho E / rho - |u|^2 / 2); q = kSrcPlain the array itself (one nt^3 component).
constexpr int kSrcDensity = 0, kSrcPressure = 4, kSrcPlain = 5;

__device__ __forceinline__ double spline_source(const double* __restrict__ W, long long comp, double gm1, int q,
                                                long long idx)
{
    if (q == kSrcDensity || q == kSrcPlain) return W[idx];
    const double d = W[idx];
    if (q != kSrcPressure) return __ddiv_rn(W[q * comp + idx], d);
    const double u = __ddiv_rn(W[comp + idx], d), v = __ddiv_rn(W[2 * comp + idx], d), w = __ddiv_rn(W[3 * comp + idx], d);
    const double vs = add(add(mul(u, u), mul(v, v)), mul(w, w));
    return mul(mul(d, gm1), sub(__ddiv_rn(W[4 * comp + idx], d), mul(0.5, vs)));
}

// pass 0: the data of source q along axis 0 (y) -> out [M0][N1][N2]; one line (i, k).  VEL: q is a
// velocity (1..3), whose source alone is compiled in.
template <int U, bool VEL>
__device__ __forceinline__ void pass0_line(const double* __restrict__ W, const FieldConst& fc, const SplineGrid& g,
                                           const SplineTables& tb, int q, double* __restrict__ out, long long L,
                                           long long stride = 0)
{
    const int N = g.npts;
    const long long lines = stride ? stride : (long long)N * N;   // output stride along axis 0
    const long long comp = fc.comp;
    const int off = g.periodic ? 3 : 0;
    const int i = (int)(L / N), k = (int)(L - (long long)i * N);
    const long long base = (long long)(i + off) * fc.pitch + (k + off);
    const long long sj = (long long)fc.nt * fc.pitch;
    auto f = [&](int j) {
        const long long idx = (long long)(j + off) * sj + base;
        if constexpr (VEL) return __ddiv_rn(W[q * comp + idx], W[idx]);
        else return spline_source(W, comp, fc.gm1, q, idx);
    };
    line_solve<U, false, false>(f, N, g.periodic, tb, out + L, lines);
}

template <bool VEL>
__global__ void spline_pass0(const double* __restrict__ W, FieldConst fc, SplineGrid g, SplineTables tb, int q,
                             double* __restrict__ out)
{
    const long long lines = (long long)g.npts * g.npts;
    for (long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x; L < lines; L += (long long)gridDim.x * blockDim.x)
        pass0_line<kLineBatch0, VEL>(W, fc, g, tb, q, out, L);
}

// pass 1: [M0][N1][N2] along axis 1 -> [M0][M1][N2]; one line (a, k)
template <int U>
__device__ __forceinline__ void pass1_line(const double* __restrict__ in, const SplineGrid& g, const SplineTables& tb,
                                           double* __restrict__ out, long long L)
{
    const int N = g.npts, M = N + g.pad;
    const int a = (int)(L / N), k = (int)(L - (long long)a * N);
    const double* src = in + (long long)a * N * N + k;
    auto f = [&](int i) { return src[(long long)i * N]; };
    line_solve<U, false, true>(f, N, g.periodic, tb, out + (long long)a * M * N + k, N);
}

__global__ void spline_pass1(const double* __restrict__ in, SplineGrid g, SplineTables tb, double* __restrict__ out)
{
    const long long lines = (long long)(g.npts + g.pad) * g.npts;
    for (long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x; L < lines; L += (long long)gridDim.x * blockDim.x)
        pass1_line<kLineBatch1Single>(in, g, tb, out, L);
}

// pass 2: [M0][M1][N2] along axis 2 -> [M0][M1][M2].  Lines are contiguous,
// so a thread per line would read 32 scattered addresses per warp access.
// Instead each warp owns 32 lines and moves 32-value chunks of them through
// shared memory (coalesced 256 B rows); lane j then runs line j's recurrence on
// its staged row.  The arithmetic per line is the one of line_solve, in the
// same order, so the coefficients are identical.
constexpr int kLineChunk = 32;
constexpr int kPass2Warps = 4;

// Rows of one line staged in shared memory: row[t] holds point i0 + t.  Forward elimination of the
// points [i_lo, i_hi] in that chunk (given: rp is the value of the point before i_lo), and back substitution of the same points downwards (the
// line's last row, whose pivot has no tabled reciprocal, divided first).
__device__ __forceinline__ void chunk_forward(double* row, int i0, int i_lo, int i_hi, int N, int periodic,
                                              const SplineTables& tb, double c0, double cl, double r_inf, double& rp,
                                              bool given = false)
{
    const int a = max(i_lo, i0), b = min(i_hi, i0 + kLineChunk - 1);
#pragma unroll 8
    for (int i = a; i <= b; i++) {
        double r = mul(6.0, row[i - i0]);
        if (!periodic) {
            if (i == 1) r = sub(r, c0);
            if (i == N - 2) r = sub(r, cl);
        }
        rp = (i == i_lo && !given) ? r : sub(r, mul(i > kPivotRows ? r_inf : tb.mt[i], rp));
        row[i - i0] = rp;
    }
}
__device__ __forceinline__ void chunk_back(double* row, int i0, int i_lo, int i_hi, const SplineTables& tb, double d_inf,
                                           double r_inf, double& x)
{
    const int a = max(i_lo, i0);
    int i = min(i_hi, i0 + kLineChunk - 1);
    if (i == i_hi && i >= a) {
        x = __ddiv_rn(row[i - i0], tb.dp[i]);
        row[i - i0] = x;
        i--;
    }
    constexpr int U = 8;
    for (; i - U + 1 >= a; i -= U) {
        double cv[U];
#pragma unroll
        for (int u = 0; u < U; u++) cv[u] = row[i - u - i0];
        if (back_rows<U>(cv, i, tb, d_inf, r_inf, x)) {
#pragma unroll
            for (int u = 0; u < U; u++) row[i - u - i0] = cv[u];
        } else {
#pragma unroll 1
            for (int k = i; k > i - U; k--) {
                x = __ddiv_rn(sub(row[k - i0], x), tb.dp[k]);
                row[k - i0] = x;
            }
        }
    }
#pragma unroll 1
    for (; i >= a; i--) {
        x = __ddiv_rn(sub(row[i - i0], x), tb.dp[i]);
        row[i - i0] = x;
    }
}

// lines [L0, L0 + 32) of a pass-2 input (lines total), by one warp with its staging rows sm.
// Chunks are 32 output slots [s0, s0 + 32), holding values s0 - 1 .. s0 + 30 of the line (value i
// lands in slot i + 1): the copies out, and the backward sweep's copies back in, then cover whole
// 32-byte sectors of the output rows (2,112 bytes, a multiple of 32) instead of starting 8 bytes
// into one.
__device__ __forceinline__ void pass2_group(const double* __restrict__ in, const SplineGrid& g, const SplineTables& tb,
                                            double* __restrict__ out, long long L0, long long lines,
                                            double (*sm)[kLineChunk + 1])
{
    const int N = g.npts, M = N + g.pad;
    const int lane = threadIdx.x & 31;
    const int nl = (int)min(32LL, lines - L0);   // lines of this warp
    const long long myL = L0 + lane;
    const bool mine = lane < nl;
    // values s0 - 1 + lane of the warp's lines from the input rows (N values each)
    auto load_in = [&](int s0) {
        const int e = s0 - 1 + lane;
        if (e >= 0 && e < N)
            for (int j = 0; j < nl; j++) sm[j][lane] = in[(L0 + j) * N + e];
        __syncwarp();
    };
    // slots s0 + lane (1..N) of the warp's output rows, in and out
    auto load_out = [&](int s0) {
        const int sl = s0 + lane;
        if (sl >= 1 && sl <= N)
            for (int j = 0; j < nl; j++) sm[j][lane] = out[(L0 + j) * M + sl];
        __syncwarp();
    };
    auto store_out = [&](int s0) {
        __syncwarp();
        const int sl = s0 + lane;
        if (sl >= 1 && sl <= N)
            for (int j = 0; j < nl; j++) out[(L0 + j) * M + sl] = sm[j][lane];
        __syncwarp();
    };
    const int s_last = (N / kLineChunk) * kLineChunk;   // the chunk holding slot N
    double d_inf, r_inf;
    fixed_pivots(N, tb, d_inf, r_inf);
    const double* src = in + myL * N;
    double* dst = out + myL * M;
    // The forward value before each chunk is kept in the output rows, 32 lanes side by side at the
    // first row's slots s0 .. s0 + 31 (beyond its end, in the next row's first slots), until the backward
    // sweep, which forms the chunk's forward values again, overwrites them with that chunk (the first
    // slots come last): the lines are read twice and written once instead of twice.
    double* keep = out + L0 * M + lane;
    if (!g.periodic) {
        const double c0 = mine ? src[0] : 0.0, cl = mine ? src[N - 1] : 0.0;
        // forward elimination of points 1..N-2 (values 0 and N-1 land in slots 1, N)
        double rp = 0.0;
        for (int s0 = 0; s0 <= s_last; s0 += kLineChunk) {
            load_in(s0);
            if (mine) {
                keep[s0] = rp;
                chunk_forward(sm[lane], s0 - 1, 1, N - 2, N, 0, tb, c0, cl, r_inf, rp);
            }
            __syncwarp();
        }
        // back substitution, chunks in descending order
        double x = 0.0, x1 = 0.0, xl2 = 0.0;
        for (int s0 = s_last; s0 >= 0; s0 -= kLineChunk) {
            load_in(s0);
            if (mine) {
                rp = keep[s0];
                chunk_forward(sm[lane], s0 - 1, 1, N - 2, N, 0, tb, c0, cl, r_inf, rp);
                chunk_back(sm[lane], s0 - 1, 1, N - 2, tb, d_inf, r_inf, x);
                if (s0 - 1 <= N - 2 && N - 2 < s0 - 1 + kLineChunk) xl2 = sm[lane][N - 2 - (s0 - 1)];
                x1 = x;   // the last chunk's last value is the solution of point 1
            }
            store_out(s0);
        }
        if (mine) {
            dst[1] = c0;
            dst[N] = cl;
            dst[0] = sub(2.0 * c0, x1);
            dst[N + 1] = sub(2.0 * cl, xl2);
        }
    } else {
        double rp = 0.0;
        for (int s0 = 0; s0 <= s_last; s0 += kLineChunk) {
            load_in(s0);
            if (mine) {
                keep[s0] = rp;
                chunk_forward(sm[lane], s0 - 1, 0, N - 1, N, 1, tb, 0.0, 0.0, r_inf, rp);
            }
            __syncwarp();
        }
        double x = 0.0, x0 = 0.0, xl = 0.0;
        for (int s0 = s_last; s0 >= 0; s0 -= kLineChunk) {
            load_in(s0);
            if (mine) {
                rp = keep[s0];
                chunk_forward(sm[lane], s0 - 1, 0, N - 1, N, 1, tb, 0.0, 0.0, r_inf, rp);
                chunk_back(sm[lane], s0 - 1, 0, N - 1, tb, d_inf, r_inf, x);
                if (s0 - 1 <= N - 1 && N - 1 < s0 - 1 + kLineChunk) xl = sm[lane][N - 1 - (s0 - 1)];
                x0 = x;   // the last chunk's last value is the solution of point 0
            }
            store_out(s0);
        }
        const double fac = mine ? __ddiv_rn(add(x0, mul(-0.25, xl)), tb.denom) : 0.0;
        double y0 = 0.0, y1 = 0.0, yl = 0.0;
        for (int s0 = 0; s0 <= s_last; s0 += kLineChunk) {
            load_out(s0);
            if (mine)
                for (int t = 0; t < kLineChunk; t++) {
                    const int i = s0 - 1 + t;
                    if (i < 0 || i > N - 1) continue;
                    const double v = sub(sm[lane][t], mul(fac, tb.z[i]));
                    sm[lane][t] = v;
                    if (i == 0) y0 = v;
                    if (i == 1) y1 = v;
                    if (i == N - 1) yl = v;
                }
            store_out(s0);
        }
        if (mine) {
            dst[0] = yl;
            dst[N + 1] = y0;
            dst[N + 2] = y1;
        }
    }
}

__global__ void __launch_bounds__(32 * kPass2Warps) spline_pass2(const double* __restrict__ in, SplineGrid g,
                                                                 SplineTables tb, double* __restrict__ out)
{
    __shared__ double stage[kPass2Warps][32][kLineChunk + 1];
    const int M = g.npts + g.pad;
    const long long lines = (long long)M * M;
    const int warp = threadIdx.x >> 5;
    const long long nwarps = (long long)gridDim.x * kPass2Warps;
    for (long long L0 = ((long long)blockIdx.x * kPass2Warps + warp) * 32; L0 < lines; L0 += nwarps * 32)
        pass2_group(in, g, tb, out, L0, lines, stage[warp]);
}

// ---- velocity splines with FP32 coefficients: the same FP64 line solves, only the stored
// coefficients are rounded to single precision.  Pass 0 writes [M0][M1][N2] with room along axis
// 1, pass 1 solves in place there, pass 2 solves each of its lines in place and writes the rounded
// coefficients: one FP64 buffer of M^2 N values serves all three components (instead of that
// scratch plus three FP64 coefficient arrays of M^3).
__global__ void spline_pass0_room(const double* __restrict__ W, FieldConst fc, SplineGrid g, SplineTables tb, int q,
                                  double* __restrict__ out)
{
    const long long lines = (long long)g.npts * g.npts;
    const long long stride = (long long)(g.npts + g.pad) * g.npts;
    for (long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x; L < lines; L += (long long)gridDim.x * blockDim.x)
        pass0_line<kLineBatch0, true>(W, fc, g, tb, q, out, L, stride);
}

// pass 1 in place on [M0][M1][N2]: line (a, k) reads rows 0..N-1 and writes rows 0..M-1
__global__ void spline_pass1_inplace(double* buf, SplineGrid g, SplineTables tb)
{
    const int N = g.npts, M = N + g.pad;
    const long long lines = (long long)M * N;
    for (long long L = blockIdx.x * (long long)blockDim.x + threadIdx.x; L < lines; L += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(L / N), k = (int)(L - (long long)a * N);
        double* line = buf + (long long)a * M * N + k;
        auto f = [&](int i) { return line[(long long)i * N]; };
        line_solve<kLineBatch1Single, true, true>(f, N, g.periodic, tb, line, N);
    }
}

// pass 2 with FP32 output: the lines of [M0][M1][N2] along axis 2, 32 per warp through shared
// memory as pass2_group, each chunk's first forward value kept in the place of its input; natural ends:
// the backward sweep writes each solution rounded as its coefficient; periodic: the solution of
// point i goes to slot i+1 (i <= N-2; the last one stays in a register) for the correction sweep,
// which writes the rounded coefficients.  Output [M0][M1][M2] floats.
__device__ __forceinline__ void pass2_group_f32(double* in, const SplineGrid& g, const SplineTables& tb,
                                                float* __restrict__ out, long long L0, long long lines,
                                                double (*sm)[kLineChunk + 1])
{
    const int N = g.npts, M = N + g.pad;
    const int lane = threadIdx.x & 31;
    const int nl = (int)min(32LL, lines - L0);
    const long long myL = L0 + lane;
    const bool mine = lane < nl;
    auto load = [&](int k0) {
        for (int j = 0; j < nl; j++) {
            const int k = k0 + lane;
            if (k < N) sm[j][lane] = in[(L0 + j) * N + k];
        }
        __syncwarp();
    };
    // staged solutions of points k < N - 1 into slots k + 1 of their lines
    auto store = [&](int k0) {
        __syncwarp();
        for (int j = 0; j < nl; j++) {
            const int k = k0 + lane;
            if (k < N - 1) in[(L0 + j) * N + k + 1] = sm[j][lane];
        }
        __syncwarp();
    };
    // staged values of slots k (kmin <= k < kmax) rounded into coefficients k + off
    auto emit = [&](int k0, int kmin, int kmax, int off) {
        __syncwarp();
        for (int j = 0; j < nl; j++) {
            const int k = k0 + lane;
            if (k >= kmin && k < kmax) out[(L0 + j) * M + k + off] = (float)sm[j][lane];
        }
        __syncwarp();
    };
    const double* src = in + myL * N;
    double* line = in + myL * N;
    float* dst = out + myL * M;
    const int top = ((N - 1) / kLineChunk) * kLineChunk;
    double d_inf, r_inf;
    fixed_pivots(N, tb, d_inf, r_inf);
    if (!g.periodic) {
        const double c0 = mine ? src[0] : 0.0, cl = mine ? src[N - 1] : 0.0;
        double rp = 0.0;
        for (int k0 = 0; k0 < N; k0 += kLineChunk) {
            load(k0);
            if (mine) {
                chunk_forward(sm[lane], k0, 1, N - 2, N, 0, tb, c0, cl, r_inf, rp);
                if (k0 > 0) line[k0] = sm[lane][0];
            }
            __syncwarp();
        }
        double x = 0.0, x1 = 0.0, xl2 = 0.0;
        for (int k0 = top; k0 >= 0; k0 -= kLineChunk) {
            load(k0);
            if (mine) {
                rp = sm[lane][0];
                chunk_forward(sm[lane], k0, k0 > 0 ? k0 + 1 : 1, N - 2, N, 0, tb, c0, cl, r_inf, rp, k0 > 0);
                chunk_back(sm[lane], k0, 1, N - 2, tb, d_inf, r_inf, x);
                if (k0 <= N - 2 && N - 2 < k0 + kLineChunk) xl2 = sm[lane][N - 2 - k0];
                x1 = x;
            }
            emit(k0, 1, N - 1, 1);   // the solution of point i is coefficient i + 1 (1 <= i <= N-2)
        }
        if (mine) {
            dst[1] = (float)c0;
            dst[0] = (float)sub(2.0 * c0, x1);
            dst[N] = (float)cl;
            dst[N + 1] = (float)sub(2.0 * cl, xl2);
        }
    } else {
        double rp = 0.0;
        for (int k0 = 0; k0 < N; k0 += kLineChunk) {
            load(k0);
            if (mine) {
                chunk_forward(sm[lane], k0, 0, N - 1, N, 1, tb, 0.0, 0.0, r_inf, rp);
                if (k0 > 0) line[k0] = sm[lane][0];
            }
            __syncwarp();
        }
        double x = 0.0, x0 = 0.0, xl = 0.0;
        for (int k0 = top; k0 >= 0; k0 -= kLineChunk) {
            load(k0);
            if (mine) {
                rp = sm[lane][0];
                chunk_forward(sm[lane], k0, k0 > 0 ? k0 + 1 : 0, N - 1, N, 1, tb, 0.0, 0.0, r_inf, rp, k0 > 0);
                chunk_back(sm[lane], k0, 0, N - 1, tb, d_inf, r_inf, x);
                if (k0 <= N - 1 && N - 1 < k0 + kLineChunk) xl = sm[lane][N - 1 - k0];
                x0 = x;
            }
            store(k0);
        }
        const double fac = mine ? __ddiv_rn(add(x0, mul(-0.25, xl)), tb.denom) : 0.0;
        double y0 = 0.0, y1 = 0.0;
        for (int k0 = 0; k0 < N; k0 += kLineChunk) {
            load(k0);
            if (mine)
                for (int t = 0; t < kLineChunk && k0 + t < N; t++) {
                    const int s = k0 + t;   // slot s holds point s-1
                    if (s < 1) continue;
                    const double v = sub(sm[lane][t], mul(fac, tb.z[s - 1]));
                    sm[lane][t] = v;
                    if (s == 1) y0 = v;
                    if (s == 2) y1 = v;
                }
            emit(k0, 1, N, 0);
        }
        if (mine) {
            const double yl = sub(xl, mul(fac, tb.z[N - 1]));
            dst[N] = (float)yl;
            dst[0] = (float)yl;
            dst[N + 1] = (float)y0;
            dst[N + 2] = (float)y1;
        }
    }
}

__global__ void __launch_bounds__(32 * kPass2Warps) spline_pass2_f32(double* in, SplineGrid g, SplineTables tb,
                                                                     float* __restrict__ out)
{
    __shared__ double stage[kPass2Warps][32][kLineChunk + 1];
    const int M = g.npts + g.pad;
    const long long lines = (long long)M * M;
    const int warp = threadIdx.x >> 5;
    const long long nwarps = (long long)gridDim.x * kPass2Warps;
    for (long long L0 = ((long long)blockIdx.x * kPass2Warps + warp) * 32; L0 < lines; L0 += nwarps * 32)
        pass2_group_f32(in, g, tb, out, L0, lines, stage[warp]);
}

// ---- lines resident in shared memory.  A warp (a CTA of its own, but for ensembles) takes 32 lines: their values come in at
// once, all loads in flight, each lane solves its line in place, and the coefficients go out, so a
// pass reads and writes global memory once.  The forward values of the kernels above make the round
// through global memory instead, and their loads wait on one another 4 or 8 at a time.  What
// remains is the lanes' serial chain, which pivot_quotient keeps short.
// How many warps of such lines an SM holds decides where it pays.  Velocity splines, ms, streaming
// kernels against these: three components per launch 64^3 0.099 -> 0.048, 128^3 0.270 -> 0.157, 160^3 0.371 ->
// 0.334, 192^3 0.763 -> 0.631, 224^3 0.99 -> 1.16, 256^3 1.26 -> 1.65; one component per launch (coefficients in
// FP32) 128^3 0.511 -> 0.198, 200^3 0.99 -> 0.76, 224^3 1.25 -> 1.09, 256^3 1.58 -> 1.50, 282^3 1.80 -> 1.90.
constexpr int kResidentBatched = 200, kResidentSingle = 264;
constexpr int kTableRows = kPivotRows + 2;   // rows of the tables a warp keeps beside its lines
__host__ __device__ inline int resident_bytes(int npts) { return (int)sizeof(double) * (2 * kTableRows + 32 * (npts | 1)); }

// 8-byte asynchronous copies, a thread's own (its wait covers them)
__device__ __forceinline__ void copy8_async(double* dst, const double* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait()
{
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

// the first rows of the pivot tables in shared memory (mt, then dp), the later ones' fixed point
struct LineTables {
    const double *mt, *dp;
    double d_inf, r_inf, d_last;
    __device__ __forceinline__ double m(int i) const { return i < kTableRows ? mt[i] : r_inf; }
    __device__ __forceinline__ double d(int i) const { return i < kTableRows ? dp[i] : d_inf; }
};
// issued with the lines' own copies; the caller waits and synchronises the warp
__device__ __forceinline__ LineTables line_tables(const SplineTables& tb, int N, int periodic, double* smem)
{
    const int lane = threadIdx.x & 31;
    if (lane < kTableRows && lane <= N) {
        copy8_async(smem + lane, tb.mt + lane);
        copy8_async(smem + kTableRows + lane, tb.dp + lane);
    }
    LineTables T;
    T.mt = smem;
    T.dp = smem + kTableRows;
    fixed_pivots(N, tb, T.d_inf, T.r_inf);
    T.d_last = tb.dp[periodic ? N - 1 : N - 2];
    return T;
}

// one line in place in shared memory, point i at s[i * st]: on return s holds the coefficients of points
// 0..N-1 (natural ends: lo and hi the ones outside).  The arithmetic and its order are line_solve's.
__device__ __forceinline__ void resident_solve(double* s, int st, int N, int periodic, const LineTables& T,
                                               const SplineTables& tb, double& lo, double& hi)
{
    const int i_lo = periodic ? 0 : 1, i_hi = periodic ? N - 1 : N - 2;
    const double c0 = s[0], cl = s[(N - 1) * st];
    double rp = 0.0;
    constexpr int U = 8;
    auto fwd = [&](int i, double fi) {
        double r = mul(6.0, fi);
        if (!periodic) {
            if (i == 1) r = sub(r, c0);
            if (i == N - 2) r = sub(r, cl);
        }
        rp = (i == i_lo) ? r : sub(r, mul(T.m(i), rp));
        s[i * st] = rp;
    };
    int i = i_lo;
    for (; i + U - 1 <= i_hi; i += U) {
        double fv[U];
#pragma unroll
        for (int u = 0; u < U; u++) fv[u] = s[(i + u) * st];
        if (i > kPivotRows && i + U - 1 < N - 2) {   // the inner rows
#pragma unroll
            for (int u = 0; u < U; u++) {
                rp = sub(mul(6.0, fv[u]), mul(T.r_inf, rp));
                s[(i + u) * st] = rp;
            }
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) fwd(i + u, fv[u]);
        }
    }
#pragma unroll 1
    for (; i <= i_hi; i++) fwd(i, s[i * st]);
    double x = __ddiv_rn(rp, T.d_last);
    s[i_hi * st] = x;
    const double x_hi = x;
    i = i_hi - 1;
    auto back = [&](int k) {
        const double a = sub(s[k * st], x), d = T.d(k);
        x = pivot_in_range(a) ? pivot_quotient(a, d, T.m(k + 1)) : __ddiv_rn(a, d);
        s[k * st] = x;
    };
    for (; i - U + 1 >= i_lo; i -= U) {
        const bool fixed = i - U + 1 >= kPivotRows;
        double cv[U], y = x;
        bool ok = true;
#pragma unroll
        for (int u = 0; u < U; u++) cv[u] = s[(i - u) * st];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const double d = fixed ? T.d_inf : T.d(i - u), r = fixed ? T.r_inf : T.m(i - u + 1);
            const double a = sub(cv[u], y);
            ok = ok && pivot_in_range(a);
            y = pivot_quotient(a, d, r);
            cv[u] = y;
        }
        if (ok) {
            x = y;
#pragma unroll
            for (int u = 0; u < U; u++) s[(i - u) * st] = cv[u];
        } else {
#pragma unroll 1
            for (int k = i; k > i - U; k--) back(k);
        }
    }
#pragma unroll 1
    for (; i >= i_lo; i--) back(i);
    if (!periodic) {
        // x is the solution of point 1 (N >= 4)
        lo = sub(2.0 * c0, x);
        hi = sub(2.0 * cl, x_hi);
    } else {
        const double fac = __ddiv_rn(add(x, mul(-0.25, x_hi)), tb.denom);
#pragma unroll 8
        for (int k = 0; k < N; k++) s[k * st] = sub(s[k * st], mul(fac, tb.z[k]));
        lo = hi = 0.0;
    }
}

// strided lines (passes 0 and 1): lane's column of s to c, stride cs
__device__ __forceinline__ void resident_store(const double* s, int N, int periodic, double lo, double hi, double* c,
                                               long long cs)
{
#pragma unroll 8
    for (int i = 0; i < N; i++) c[(long long)(i + 1) * cs] = s[i * 32];
    if (!periodic) {
        c[0] = lo;
        c[(long long)(N + 1) * cs] = hi;
    } else {
        c[0] = s[(N - 1) * 32];
        c[(long long)(N + 1) * cs] = s[0];
        c[(long long)(N + 2) * cs] = s[32];
    }
}

// pass 0, lines [32 group, 32 group + 32) of source q along axis 0 -> out, `stride` apart along axis 0
template <bool VEL>
__device__ __forceinline__ void resident_pass0(const double* __restrict__ W, const FieldConst& fc, const SplineGrid& g,
                                               const SplineTables& tb, int q, double* __restrict__ out, long long stride,
                                               long long group, double* smem)
{
    const int N = g.npts, lane = threadIdx.x & 31;
    const LineTables T = line_tables(tb, N, g.periodic, smem);
    const bool mine = group * 32 + lane < (long long)N * N;
    const long long L = mine ? group * 32 + lane : (long long)N * N - 1;   // a lane beyond the lines repeats the last
    const int off = g.periodic ? 3 : 0;
    const int i = (int)(L / N), k = (int)(L - (long long)i * N);
    const long long sj = (long long)fc.nt * fc.pitch, base = off * sj + (long long)(i + off) * fc.pitch + (k + off),
                    comp = fc.comp;
    double* s = smem + 2 * kTableRows + lane;
    if constexpr (VEL) {   // the next rows' loads are issued before this batch's divisions
        constexpr int U = 8;
        const double* pd = W + base;
        const double* pm = pd + q * comp;
        double d[U], m[U], dn[U], mn[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long o = min(u, N - 1) * sj;
            d[u] = pd[o];
            m[u] = pm[o];
        }
        for (int j = 0; j < N; j += U) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const long long o = min(j + U + u, N - 1) * sj;
                dn[u] = pd[o];
                mn[u] = pm[o];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (j + u < N) s[(j + u) * 32] = __ddiv_rn(m[u], d[u]);
                d[u] = dn[u];
                m[u] = mn[u];
            }
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < N; j++) s[j * 32] = spline_source(W, comp, fc.gm1, q, base + j * sj);
    }
    copy_async_wait();
    __syncwarp();
    if (!mine) return;
    double lo, hi;
    resident_solve(s, 32, N, g.periodic, T, tb, lo, hi);
    resident_store(s, N, g.periodic, lo, hi, out + L, stride);
}

// pass 1, lines of [M0][in_rows][N2] along axis 1 -> [M0][M1][N2] (in place where in == out and in_rows = M)
__device__ __forceinline__ void resident_pass1(const double* in, int in_rows, const SplineGrid& g, const SplineTables& tb,
                                               double* out, long long group, double* smem)
{
    const int N = g.npts, M = N + g.pad, lane = threadIdx.x & 31;
    const LineTables T = line_tables(tb, N, g.periodic, smem);
    const bool mine = group * 32 + lane < (long long)M * N;
    const long long L = mine ? group * 32 + lane : (long long)M * N - 1;
    const int a = (int)(L / N), k = (int)(L - (long long)a * N);
    const double* src = in + (long long)a * in_rows * N + k;
    double* s = smem + 2 * kTableRows + lane;
    if (mine) {
#pragma unroll 8
        for (int i = 0; i < N; i++) copy8_async(s + i * 32, src + (long long)i * N);
    }
    copy_async_wait();
    __syncwarp();
    if (!mine) return;
    double lo, hi;
    resident_solve(s, 32, N, g.periodic, T, tb, lo, hi);
    resident_store(s, N, g.periodic, lo, hi, out + (long long)a * M * N + k, N);
}

// pass 2, the contiguous lines of [M0][M1][N2] -> [M0][M1][M2]: rows move coalesced, lane j solves row j
// (rows an odd number of doubles apart: no bank conflicts); the stores start on the output's sectors
template <class OutT>
__device__ __forceinline__ void resident_pass2(const double* __restrict__ in, const SplineGrid& g, const SplineTables& tb,
                                               OutT* __restrict__ out, long long group, double* smem)
{
    const int N = g.npts, M = N + g.pad, S = N | 1, lane = threadIdx.x & 31;
    const long long lines = (long long)M * M, L0 = group * 32;
    const int nl = (int)min(32LL, lines - L0);
    const LineTables T = line_tables(tb, N, g.periodic, smem);
    smem += 2 * kTableRows;
    for (int j = 0; j < nl; j++)
        for (int k = lane; k < N; k += 32) copy8_async(smem + j * S + k, in + (L0 + j) * N + k);
    copy_async_wait();
    __syncwarp();
    if (lane < nl) {
        double lo, hi;
        double* s = smem + lane * S;
        resident_solve(s, 1, N, g.periodic, T, tb, lo, hi);
        OutT* dst = out + (L0 + lane) * M;
        if (!g.periodic) {
            dst[0] = (OutT)lo;
            dst[N + 1] = (OutT)hi;
        } else {
            dst[0] = (OutT)s[N - 1];
            dst[N + 1] = (OutT)s[0];
            dst[N + 2] = (OutT)s[1];
        }
    }
    __syncwarp();
    for (int j = 0; j < nl; j++)
        for (int sl = lane; sl <= N; sl += 32)
            if (sl > 0) out[(L0 + j) * M + sl] = (OutT)smem[j * S + sl - 1];
}

template <bool VEL>
__global__ void __launch_bounds__(32) spline_resident0(const double* __restrict__ W, FieldConst fc, SplineGrid g,
                                                       SplineTables tb, int q, double* __restrict__ out, long long stride)
{
    extern __shared__ double line_smem[];
    resident_pass0<VEL>(W, fc, g, tb, q, out, stride, blockIdx.x, line_smem);
}
__global__ void __launch_bounds__(32) spline_resident1(const double* in, int in_rows, SplineGrid g, SplineTables tb,
                                                       double* out)
{
    extern __shared__ double line_smem[];
    resident_pass1(in, in_rows, g, tb, out, blockIdx.x, line_smem);
}
template <class OutT>
__global__ void __launch_bounds__(32) spline_resident2(const double* __restrict__ in, SplineGrid g, SplineTables tb,
                                                       OutT* __restrict__ out)
{
    extern __shared__ double line_smem[];
    resident_pass2<OutT>(in, g, tb, out, blockIdx.x, line_smem);
}

struct Basis {
    double w[4];
};

__device__ __forceinline__ int locate(const SplineGrid& g, double x, double& t)
{
    const double u = mul(sub(x, g.start), g.dinv);
    const double fl = floor(u);
    int i = (int)fl;
    if (g.periodic) {
        t = sub(u, fl);
        i %= g.npts;
        if (i < 0) i += g.npts;
        return i;
    }
    if (i < 0) i = 0;
    if (i > g.npts - 2) i = g.npts - 2;
    t = sub(u, (double)i);
    return i;
}

__device__ __forceinline__ Basis basis(double t)
{
    const double t2 = mul(t, t), t3 = mul(t2, t), s = sub(1.0, t);
    const double c = 1.0 / 6.0;
    Basis b;
    b.w[0] = mul(c, mul(mul(s, s), s));
    b.w[1] = mul(c, add(sub(mul(3.0, t3), mul(6.0, t2)), 4.0));
    b.w[2] = mul(c, add(add(add(mul(-3.0, t3), mul(3.0, t2)), mul(3.0, t)), 1.0));
    b.w[3] = mul(c, t3);
    return b;
}

// Four consecutive coefficients from element idx on, by aligned pairs: two loads where idx is even, three
// where it is odd, instead of four (each costs L1 a pass per lane).  For arrays that start on 16 bytes,
// as allocations do; nothing outside [idx & ~1, idx + 4) is read, so no load leaves the array.
__device__ __forceinline__ void load_row(const double* __restrict__ C, long long idx, double r[4])
{
    const bool odd = idx & 1;
    const double* q = C + (idx - odd);
    const double2 a = *reinterpret_cast<const double2*>(q), b = *reinterpret_cast<const double2*>(q + 2);
    double c = 0.0;
    if (odd) c = q[4];
    r[0] = odd ? a.y : a.x;
    r[1] = odd ? b.x : a.y;
    r[2] = odd ? b.y : b.x;
    r[3] = odd ? c : b.y;
}

// value of one spline at a point (the oracle's contraction order: z, then x, then y); CT is the
// type the coefficients are stored in (double, or float for the FP32 velocity splines), the
// arithmetic is FP64.  PAIRS: FP64 coefficients by aligned pairs (the Heun kernel with 1M particles at 256^3
// 598 -> 552 us, at 128^3 461 -> 405; FP32 coefficients gain at 256^3 and lose at 512^3, particles in no order lose)
template <bool PAIRS, class CT>
__device__ __forceinline__ double spline_value(const CT* __restrict__ C, const SplineGrid& g, int ia, int ib, int ic,
                                               const Basis& A, const Basis& B, const Basis& Cz)
{
    const long long M = g.npts + g.pad;
    double v = 0.0;
#pragma unroll
    for (int x = 0; x < 4; x++) {
        double bw = 0.0;
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const CT* row = C + ((long long)(ia + x) * M + (ib + y)) * M + ic;
            double cw;
            if constexpr (PAIRS) {
                double r[4];
                load_row(C, row - C, r);
                cw = add(add(add(mul(Cz.w[0], r[0]), mul(Cz.w[1], r[1])), mul(Cz.w[2], r[2])), mul(Cz.w[3], r[3]));
            } else {
                cw = add(add(add(mul(Cz.w[0], (double)row[0]), mul(Cz.w[1], (double)row[1])),
                             mul(Cz.w[2], (double)row[2])),
                         mul(Cz.w[3], (double)row[3]));
            }
            bw = (y == 0) ? mul(B.w[0], cw) : add(bw, mul(B.w[y], cw));
        }
        v = add(v, mul(A.w[x], bw));
    }
    return v;
}

template <bool PAIRS, class CT>
__device__ __forceinline__ void eval3(const CT* const* coefs, const SplineGrid& g, double a, double b, double c,
                                      double out[3])
{
    double ta, tb, tc;
    const int ia = locate(g, a, ta), ib = locate(g, b, tb), ic = locate(g, c, tc);
    const Basis A = basis(ta), B = basis(tb), Cz = basis(tc);
#pragma unroll
    for (int f = 0; f < 3; f++) out[f] = spline_value<PAIRS, CT>(coefs[f], g, ia, ib, ic, A, B, Cz);
}

template <class CT>
struct Coefs3T {
    const CT* c[3];
};
using Coefs3 = Coefs3T<double>;

// ---------------------------------------------- values, gradients, Hessians --
// eval_UBspline_3d_d_vg / _vgl / _vgh as the CPU oracle evaluates them: basis
// weights w, first derivatives d and second derivatives h per axis, the 4x4x4
// window contracted along axis 2, then 1, then 0, every sum left to right.
struct BasisFull {
    double w[4], d[4], h[4];
};

__device__ __forceinline__ BasisFull basis_full(double t, double dinv)
{
    const double t2 = mul(t, t), t3 = mul(t2, t), s = sub(1.0, t);
    const double c = 1.0 / 6.0;
    BasisFull b;
    b.w[0] = mul(c, mul(mul(s, s), s));
    b.w[1] = mul(c, add(sub(mul(3.0, t3), mul(6.0, t2)), 4.0));
    b.w[2] = mul(c, add(add(add(mul(-3.0, t3), mul(3.0, t2)), mul(3.0, t)), 1.0));
    b.w[3] = mul(c, t3);
    b.d[0] = mul(mul(-0.5, mul(s, s)), dinv);
    b.d[1] = mul(mul(0.5, sub(mul(3.0, t2), mul(4.0, t))), dinv);
    b.d[2] = mul(mul(0.5, add(add(mul(-3.0, t2), mul(2.0, t)), 1.0)), dinv);
    b.d[3] = mul(mul(0.5, t2), dinv);
    const double d2 = mul(dinv, dinv);
    b.h[0] = mul(s, d2);
    b.h[1] = mul(sub(mul(3.0, t), 2.0), d2);
    b.h[2] = mul(add(mul(-3.0, t), 1.0), d2);
    b.h[3] = mul(t, d2);
    return b;
}

__device__ __forceinline__ double dot4(const double a[4], const double* r)
{
    return add(add(add(mul(a[0], r[0]), mul(a[1], r[1])), mul(a[2], r[2])), mul(a[3], r[3]));
}

__device__ __forceinline__ double dot4(const double a[4], double r0, double r1, double r2, double r3)
{
    return add(add(add(mul(a[0], r0), mul(a[1], r1)), mul(a[2], r2)), mul(a[3], r3));
}

struct SplineVal {
    double v, g[3], lap, h[6];   // h: 00 01 02 11 12 22
};

// WHAT 1: value + gradient; 2: + Laplacian; 3: + Hessian
template <int WHAT>
__device__ __forceinline__ SplineVal spline_eval(const double* __restrict__ C, const SplineGrid& g, double a, double b,
                                                 double c)
{
    double ta, tb, tc;
    const int ia = locate(g, a, ta), ib = locate(g, b, tb), ic = locate(g, c, tc);
    const BasisFull A = basis_full(ta, g.dinv), B = basis_full(tb, g.dinv), Z = basis_full(tc, g.dinv);
    const long long M = g.npts + g.pad;
    double v = 0, g0 = 0, g1 = 0, g2 = 0, h00 = 0, h01 = 0, h02 = 0, h11 = 0, h12 = 0, h22 = 0;
#pragma unroll
    for (int x = 0; x < 4; x++) {
        double cw[4], cd[4], ch[4];
#pragma unroll
        for (int y = 0; y < 4; y++) {
            const double* row = C + ((long long)(ia + x) * M + (ib + y)) * M + ic;
            const double r0 = row[0], r1 = row[1], r2 = row[2], r3 = row[3];
            cw[y] = dot4(Z.w, r0, r1, r2, r3);
            cd[y] = dot4(Z.d, r0, r1, r2, r3);
            ch[y] = (WHAT >= 2) ? dot4(Z.h, r0, r1, r2, r3) : 0.0;
        }
        const double bw = dot4(B.w, cw), bd = dot4(B.d, cw), bwd = dot4(B.w, cd);
        v = add(v, mul(A.w[x], bw));
        g0 = add(g0, mul(A.d[x], bw));
        g1 = add(g1, mul(A.w[x], bd));
        g2 = add(g2, mul(A.w[x], bwd));
        if (WHAT >= 2) {
            const double bh = dot4(B.h, cw), bwh = dot4(B.w, ch);
            h00 = add(h00, mul(A.h[x], bw));
            h11 = add(h11, mul(A.w[x], bh));
            h22 = add(h22, mul(A.w[x], bwh));
        }
        if (WHAT == 3) {
            const double bdd = dot4(B.d, cd);
            h01 = add(h01, mul(A.d[x], bd));
            h02 = add(h02, mul(A.d[x], bwd));
            h12 = add(h12, mul(A.w[x], bdd));
        }
    }
    SplineVal r;
    r.v = v;
    r.g[0] = g0;
    r.g[1] = g1;
    r.g[2] = g2;
    r.lap = (WHAT == 2) ? add(add(h00, h11), h22) : 0.0;
    r.h[0] = h00;
    r.h[1] = h01;
    r.h[2] = h02;
    r.h[3] = h11;
    r.h[4] = h12;
    r.h[5] = h22;
    return r;
}

// Laplacian of a velocity spline at every spline node, written at the node's
// ghost-layout cell (generateSplines, src/update.cpp:1217-1228): node (j, i, k)
// sits at ((j - 3) dx + dx/2, ...) on the reference grid.  The reference's
// loops visit interior nodes only; its ghost nodes keep the zeros of a fresh
// allocation and are splined as zeros, which this reproduces.
__global__ void lap_nodes_kernel(const double* __restrict__ C, SplineGrid g, FieldConst fc, double* __restrict__ out)
{
    const int N = g.npts, nt = fc.nt, off = g.periodic ? 3 : 0;
    const long long total = (long long)N * N * N;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(e / ((long long)N * N)), i = (int)((e / N) % N), k = (int)(e % N);
        const int J = j + off, I = i + off, K = k + off;
        const long long o = ((long long)J * nt + I) * fc.pitch + K;
        if (J < 3 || J >= nt - 3 || I < 3 || I >= nt - 3 || K < 3 || K >= nt - 3) {
            out[o] = 0.0;
            continue;
        }
        const double hx = mul(0.5, fc.dx);
        const double y = add(mul((double)(J - 3), fc.dx), hx);
        const double x = add(mul((double)(I - 3), fc.dx), hx);
        const double z = add(mul((double)(K - 3), fc.dx), hx);
        out[o] = spline_eval<2>(C, g, y, x, z).lap;
    }
}

struct Coefs8 {
    const double* c[8];   // rho, u, v, w, p, lap u, lap v, lap w
};

// getParticleProp (src/ParticleTrack.cpp:99-113) for every particle; props is the property table of
// include/gkm.h, [np][kPropCount] in upload order (a particle's 328 bytes lie together, so its scattered
// stores fill their sectors, and the host copies the table as it is).
__global__ void particle_props_kernel(Coefs8 cf, SplineGrid g, long long np, const double* __restrict__ py,
                                      const double* __restrict__ px, const double* __restrict__ pz,
                                      const long long* __restrict__ tag, double* __restrict__ props, DevClock* clock)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        const double a = py[p], b = px[p], c = pz[p];
        const long long t = tag[p];
        if (t < 0 || t >= np) {
            atomicOr(&clock->status, kStatusTags);
            continue;
        }
        double* o = props + t * kPropCount;
        auto put = [&](int slot, double v) { o[slot] = v; };
        const SplineVal d = spline_eval<1>(cf.c[0], g, a, b, c);
        put(0, d.v);
        for (int q = 0; q < 3; q++) put(1 + q, d.g[q]);
        for (int f = 0; f < 3; f++) {
            const SplineVal u = spline_eval<1>(cf.c[1 + f], g, a, b, c);
            put(4 + f, u.v);
            for (int q = 0; q < 3; q++) put(7 + 3 * f + q, u.g[q]);
        }
        const SplineVal P = spline_eval<3>(cf.c[4], g, a, b, c);
        put(16, P.v);
        for (int q = 0; q < 3; q++) put(17 + q, P.g[q]);
        const int hmap[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
        for (int q = 0; q < 9; q++) put(20 + q, P.h[hmap[q]]);
        for (int f = 0; f < 3; f++) {
            const SplineVal l = spline_eval<1>(cf.c[5 + f], g, a, b, c);
            put(29 + f, l.v);
            for (int q = 0; q < 3; q++) put(32 + 3 * f + q, l.g[q]);
        }
    }
}

// GetParticleStats (src/update.cpp:1111-1162): per-CTA sums of U.U, S_ij S_ij,
// (du/dx)^2, (du/dx)^3, (dw/dz)^2, (dw/dz)^3 over the particles (gradients are
// (d/dy, d/dx, d/dz) in the property table)
__global__ void particle_stats_kernel(const double* __restrict__ props, long long np, StatsPartial* __restrict__ part)
{
    __shared__ double red[6][32];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        auto P = [&](int slot) { return props[p * kPropCount + slot]; };
        const double U0 = P(4), U1 = P(5), U2 = P(6);
        const double dudx = P(8), dvdx = P(11), dwdx = P(14);
        const double dudy = P(7), dvdy = P(10), dwdy = P(13);
        const double dudz = P(9), dvdz = P(12), dwdz = P(15);
        acc[0] += U0 * U0 + U1 * U1 + U2 * U2;
        acc[1] += dudx * dudx + 0.5 * ((dudy + dvdx) * (dudy + dvdx)) + 0.5 * ((dudz + dwdx) * (dudz + dwdx)) +
                  0.5 * ((dwdy + dvdz) * (dwdy + dvdz)) + dvdy * dvdy + dwdz * dwdz;
        acc[2] += dudx * dudx;
        acc[3] += dudx * dudx * dudx;
        acc[4] += dwdz * dwdz;
        acc[5] += dwdz * dwdz * dwdz;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int s = 0; s < 6; s++) {
        double v = acc[s];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[s][wid] = v;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        double v = 0.0;
        if (threadIdx.x < 6)
            for (int w2 = 0; w2 < (int)(blockDim.x >> 5); w2++) v += red[threadIdx.x][w2];
        part[blockIdx.x].v[threadIdx.x] = v;
    }
}

// moment s (one warp each) over the blocks' partials: strided lane sums, then a fixed shuffle tree, so
// the result does not depend on timing.  Bound by the latency of its loads: one thread per moment summing
// all 592 partials in turn took 40 us.
__device__ __forceinline__ double sum_partials(const StatsPartial* __restrict__ part, int nblocks, int s)
{
    double v = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x & 31; b < nblocks; b += 32) v += part[b].v[s];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__global__ void particle_stats_finish(const StatsPartial* __restrict__ part, int nblocks, double* __restrict__ out)
{
    const int s = threadIdx.x >> 5;
    const double v = sum_partials(part, nblocks, s);
    if ((threadIdx.x & 31) == 0) out[s] = v;
}

template <class CT>
__global__ void particles_eval_kernel(Coefs3T<CT> cf, SplineGrid g, long long np, const double* __restrict__ py,
                                      const double* __restrict__ px, const double* __restrict__ pz,
                                      double* __restrict__ Uu, double* __restrict__ Uv, double* __restrict__ Uw)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        double U[3];
        eval3<false, CT>(cf.c, g, py[p], px[p], pz[p], U);
        Uu[p] = U[0];
        Uv[p] = U[1];
        Uw[p] = U[2];
    }
}

// Heun step (src/ParticleTrack.cpp:48-73): U from the previous evaluation,
// U2 from the new spline at pos + U dt (pos is (y, x, z), U is (u, v, w)),
// pos += (U + U2) dt / 2, periodic wrap, then U at the new position for the
// next step's predictor (the reference's getParticleProp at loop start).
// particle p read from src and written to dst (the same arrays, or the sorted copy and the
// particle arrays); arrays y, x, z, u, v, w
template <class CT>
__device__ __forceinline__ void heun_particle(const Coefs3T<CT>& cf, const SplineGrid& g, double dt, long long p,
                                              const ParticleArrays& src, const ParticleArrays& dst)
{
    const double twopi = 2.0 * 3.14159265358979311600;   // 2 * atan(1)*4 in double
    double pos[3] = {src.a[0][p], src.a[1][p], src.a[2][p]};
    const double U[3] = {src.a[3][p], src.a[4][p], src.a[5][p]};
    double U2[3];
    eval3<sizeof(CT) == 8, CT>(cf.c, g, add(pos[0], mul(U[1], dt)), add(pos[1], mul(U[0], dt)), add(pos[2], mul(U[2], dt)), U2);
    pos[0] = add(pos[0], mul(mul(0.5, add(U[1], U2[1])), dt));
    pos[1] = add(pos[1], mul(mul(0.5, add(U[0], U2[0])), dt));
    pos[2] = add(pos[2], mul(mul(0.5, add(U[2], U2[2])), dt));
#pragma unroll
    for (int q = 0; q < 3; q++) {
        if (pos[q] > twopi) pos[q] = fmod(pos[q], twopi);
        if (pos[q] < 0) pos[q] = sub(twopi, fmod(-pos[q], twopi));
    }
    double Un[3];
    eval3<sizeof(CT) == 8, CT>(cf.c, g, pos[0], pos[1], pos[2], Un);
    dst.a[0][p] = pos[0];
    dst.a[1][p] = pos[1];
    dst.a[2][p] = pos[2];
    dst.a[3][p] = Un[0];
    dst.a[4][p] = Un[1];
    dst.a[5][p] = Un[2];
}

// Heun step (src/ParticleTrack.cpp:48-73): U from the previous evaluation,
// U2 from the new spline at pos + U dt (pos is (y, x, z), U is (u, v, w)),
// pos += (U + U2) dt / 2, periodic wrap, then U at the new position for the
// next step's predictor (the reference's getParticleProp at loop start).
// With tag_src the particles come from the sorted copy and their tags move with them.
template <class CT>
__global__ void particles_heun_kernel(Coefs3T<CT> cf, SplineGrid g, const DevClock* __restrict__ clock, long long np,
                                      ParticleArrays src, ParticleArrays dst, const long long* __restrict__ tag_src,
                                      long long* __restrict__ tag_dst)
{
    const double dt = clock->dt;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        heun_particle<CT>(cf, g, dt, p, src, dst);
        if (tag_src) tag_dst[p] = tag_src[p];
    }
}

// ------------------------------------------------------- particle ordering --
// Particles are kept ordered by blocks of 8^3 spline cells (y-major, z fastest,
// the coefficient layout), so the 4x4x4 windows that a warp gathers overlap
// in L1/L2.  A counting sort: keys and counts, an exclusive scan of the
// counts, a scatter into the second particle arrays.  Each particle's
// arithmetic is independent of the order.
__global__ void particle_keys_kernel(SplineGrid g, int nb, long long np, ParticleArrays P, unsigned* __restrict__ keys,
                                     unsigned* __restrict__ counts)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        double t;
        const int a = locate(g, P.a[0][p], t) >> 3, b = locate(g, P.a[1][p], t) >> 3, c = locate(g, P.a[2][p], t) >> 3;
        const unsigned key = ((unsigned)a * nb + b) * nb + c;
        keys[p] = key;
        atomicAdd(&counts[key], 1u);
    }
}

constexpr int kScanChunk = 1024;   // elements per CTA of the scan (256 threads x 4)

// exclusive scan of data[0, n) in chunks of kScanChunk; chunk totals to sums (if given)
__global__ void __launch_bounds__(256) scan_chunks_kernel(unsigned* __restrict__ data, long long n,
                                                          unsigned* __restrict__ sums)
{
    __shared__ unsigned warp_tot[8];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const long long base = (long long)blockIdx.x * kScanChunk + 4LL * tid;
    unsigned v[4], run = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
        v[e] = (base + e < n) ? data[base + e] : 0u;
        run += v[e];
    }
    unsigned x = run;   // inclusive scan of the threads' totals within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
        unsigned t = lane < 8 ? warp_tot[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < 8) warp_tot[lane] = t;
    }
    __syncthreads();
    unsigned excl = x - run + (wid ? warp_tot[wid - 1] : 0u);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        if (base + e < n) data[base + e] = excl;
        excl += v[e];
    }
    if (sums && tid == 0) sums[blockIdx.x] = warp_tot[7];
}

__global__ void scan_add_kernel(unsigned* __restrict__ data, long long n, const unsigned* __restrict__ sums)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        data[i] += sums[i / kScanChunk];
}

// Transfers in upload order.  A host array of np x 3 values passes through three device arrays of np
// (the sorted copy's, free between steps): element e of it lies in array e / np.  Export: slot p's
// triple (positions or velocities) to its upload index; import: the triples into the particle arrays,
// tags in order.  Scattered 24-byte stores, bound by their sectors; the host then copies whole arrays.
// With the reordering on the host, a step of 1M particles and their download took 37 ms, then 8.7 (0.5 of it
// from the spline solves).
struct Triple {
    double* a[3];
};
__device__ __forceinline__ double& triple_at(const Triple& s, long long np, long long e)
{
    const int b = (e >= np) + (e >= 2 * np);
    return s.a[b][e - b * np];
}
__global__ void particle_export_kernel(long long np, const long long* __restrict__ tag, Triple src, Triple dst,
                                       DevClock* clock)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        const long long t = tag[p];
        if (t < 0 || t >= np) {
            atomicOr(&clock->status, kStatusTags);
            continue;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) triple_at(dst, np, 3 * t + c) = src.a[c][p];
    }
}
// With tags, a report of damaged ones ends: these are new.
__global__ void particle_import_kernel(long long np, Triple src, Triple dst, long long* __restrict__ tag, DevClock* clock)
{
    if (tag && blockIdx.x == 0 && threadIdx.x == 0) atomicAnd(&clock->status, ~kStatusTags);
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
#pragma unroll
        for (int c = 0; c < 3; c++) dst.a[c][p] = triple_at(src, np, 3 * p + c);
        if (tag) tag[p] = p;
    }
}

__global__ void particle_scatter_kernel(long long np, const unsigned* __restrict__ keys, unsigned* __restrict__ offsets,
                                        ParticleArrays src, ParticleArrays dst, const long long* __restrict__ tag_src,
                                        long long* __restrict__ tag_dst)
{
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        const unsigned d = atomicAdd(&offsets[keys[p]], 1u);
#pragma unroll
        for (int c = 0; c < 6; c++) dst.a[c][d] = src.a[c][p];
        tag_dst[d] = tag_src[p];
    }
}

// ---------------------------------------------------------------- stats --
// PrintStats (src/update.cpp:688-842) on the device.  At a node the spline
// value equals the data (interpolation), so rho and u come from the cell; the
// gradients come from the coefficients: per axis the node weights are
// (1, 4, 1)/6 for values and (-1, 0, 1)/2 * dinv for the derivative.
template <class CT>
__device__ __forceinline__ void node_grad(const CT* __restrict__ C, long long M, int a, int b, int c, double dinv,
                                          double g[3])
{
    const double w[3] = {1.0 / 6.0, 4.0 / 6.0, 1.0 / 6.0};
    const double d[3] = {-0.5 * dinv, 0.0, 0.5 * dinv};
    double g0 = 0, g1 = 0, g2 = 0;
#pragma unroll
    for (int x = 0; x < 3; x++)
#pragma unroll
        for (int y = 0; y < 3; y++) {
            const CT* row = C + ((long long)(a + x) * M + (b + y)) * M + c;
            const double r0 = (double)row[0], r1 = (double)row[1], r2 = (double)row[2];
            const double cw = w[0] * r0 + w[1] * r1 + w[2] * r2;
            const double cd = d[0] * r0 + d[2] * r2;
            g0 += d[x] * w[y] * cw;
            g1 += w[x] * d[y] * cw;
            g2 += w[x] * w[y] * cd;
        }
    g[0] = g0;
    g[1] = g1;
    g[2] = g2;
}

__device__ __forceinline__ double visc(const FieldConst& fc, double T)
{
    double x = T / fc.T0;
    if (fc.visc == 1) return fc.mu0 * pow(x, 0.76);
    return fc.mu0 * pow(x, 1.5) * (fc.T0 + 110.4) / (T + 110.4);
}

__device__ __forceinline__ void cell_c2p(const double* W, long long comp, long long idx, double gm1, double& d, double& u,
                                         double& v, double& w, double& P, double& T)
{
    d = W[idx];
    u = W[comp + idx] / d;
    v = W[2 * comp + idx] / d;
    w = W[3 * comp + idx] / d;
    const double vs = u * u + v * v + w * w;
    P = (d * gm1) * (W[4 * comp + idx] / d - 0.5 * vs);
    T = P / (287.0 * d);
}

template <int PASS, class CT>
__global__ void stats_kernel(const double* __restrict__ W, FieldConst fc, SplineGrid g, Coefs3T<CT> cf,
                             const double* __restrict__ means, StatsPartial* __restrict__ part)
{
    __shared__ double red[16][32];
    const int n = fc.n, nt = fc.nt;
    const long long comp = fc.comp, total = (long long)n * n * n;
    const long long M = g.npts + g.pad;
    const int off = g.periodic ? 0 : 3;   // coefficient window start of interior cell m
    double acc[16];
#pragma unroll
    for (int s = 0; s < 16; s++) acc[s] = 0.0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(e / ((long long)n * n)), i = (int)((e / n) % n), k = (int)(e % n);
        const long long idx = ((long long)(j + 3) * nt + (i + 3)) * fc.pitch + (k + 3);
        double d, u, v, w, P, T;
        cell_c2p(W, comp, idx, fc.gm1, d, u, v, w, P, T);
        if (PASS == 0) {
            double gu[3], gv[3], gw[3];
            node_grad<CT>(cf.c[0], M, j + off, i + off, k + off, g.dinv, gu);
            node_grad<CT>(cf.c[1], M, j + off, i + off, k + off, g.dinv, gv);
            node_grad<CT>(cf.c[2], M, j + off, i + off, k + off, g.dinv, gw);
            const double dudx = gu[1], dudy = gu[0], dudz = gu[2];
            const double dvdx = gv[1], dvdy = gv[0], dvdz = gv[2];
            const double dwdx = gw[1], dwdy = gw[0], dwdz = gw[2];
            const double a2 = dudx * dudx + dudy * dudy + dudz * dudz + dvdx * dvdx + dvdy * dvdy + dvdz * dvdz +
                              dwdx * dwdx + dwdy * dwdy + dwdz * dwdz;
            acc[0] += d * (u * u + v * v + w * w);                      // TKE
            acc[1] += visc(fc, T) * a2;                                 // Diss
            acc[2] += dudx * dudx + 0.5 * (dudy + dvdx) * (dudy + dvdx) + 0.5 * (dudz + dwdx) * (dudz + dwdx) +
                      0.5 * (dwdy + dvdz) * (dwdy + dvdz) + dvdy * dvdy + dwdz * dwdz;   // SijSij
            acc[3] += dudx * dudx;
            acc[4] += dudx * dudx * dudx;
            acc[5] += dudx * dudx * dudx * dudx;
            acc[6] += dvdy * dvdy;
            acc[7] += dvdy * dvdy * dvdy;
            acc[8] += dvdy * dvdy * dvdy * dvdy;
            acc[9] += dwdz * dwdz;
            acc[10] += dwdz * dwdz * dwdz;
            acc[11] += dwdz * dwdz * dwdz * dwdz;
            acc[12] += P;
            acc[13] += T;
            acc[14] += 1.0 / d;
        } else {
            acc[0] += (means[0] - P) * (means[0] - P);
            acc[1] += (means[1] - T) * (means[1] - T);
            acc[2] += (means[2] - 1.0 / d) * (means[2] - 1.0 / d);
        }
    }
    // deterministic block reduction: warp shuffles, then warp partials in fixed order
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int s = 0; s < 16; s++) {
        double v = acc[s];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[s][wid] = v;
    }
    __syncthreads();
    if (threadIdx.x < 16) {
        double v = 0.0;
        for (int w2 = 0; w2 < (int)(blockDim.x >> 5); w2++) v += red[threadIdx.x][w2];
        part[blockIdx.x].v[threadIdx.x] = v;
    }
}

// sums the partials (16 warps); PASS 0 also forms the means for pass 1
__global__ void stats_finish(const StatsPartial* __restrict__ part, int nblocks, double ncells, int pass,
                             double* __restrict__ out)
{
    const int s = threadIdx.x >> 5;
    const double v = sum_partials(part, nblocks, s);
    if (threadIdx.x & 31) return;
    if (pass == 0) out[s] = v / ncells;
    else if (s < 3) out[16 + s] = sqrt(v / ncells);
}

template <class K, class... Args>
cudaError_t grid_launch(K kernel, long long work, int threads, cudaStream_t s, Args... args)
{
    long long b = (work + threads - 1) / threads;
    if (b < 1) b = 1;
    if (b > 148 * 16) b = 148 * 16;
    kernel<<<(unsigned)b, threads, 0, s>>>(args...);
    return cudaGetLastError();
}

// ---- ensemble forms: one launch per pass over every member's lines / particles; the lines in groups of
// 32, one warp each, off[] the members' work items of all three components: groups, or with resident lines
// blocks of them (spline_items)
__device__ __forceinline__ const MemberDev& ensemble_group(const MemberDev* __restrict__ mem,
                                                           const long long* __restrict__ off, int nm, long long w,
                                                           int pass, int& q, long long& group)
{
    const int m = find_member(off, nm, w);
    const MemberDev& md = mem[m];
    const long long local = w - off[m], groups = spline_groups(pass, md.grid.npts, md.grid.pad);
    q = (int)(local / groups);
    group = local - q * groups;
    return md;
}

// Resident lines of members of several sizes: a block has the shared memory of the largest member's group, rounded up as
// far as no block per SM is lost, and takes as many groups of one component of a member as fit it (a warp each),
// so small members' lines fill the SMs as well.  With one group per block whatever its size, 64 members of
// 48^3 beside one of 194^3 took 1.75 ms (four warps per SM for all lines) against 1.39 streamed; so 1.18.
constexpr int kEnsembleWarps = 4;
__host__ __device__ inline int resident_per_block(int npts, int warps, int smem)
{
    const int fit = smem / resident_bytes(npts);
    return fit < warps ? fit : warps;
}
// this warp's group of component q of a member and its part of the shared memory; false without one
template <int WARPS>
__device__ __forceinline__ bool ensemble_resident(const MemberDev* __restrict__ mem, const long long* __restrict__ off,
                                                  int nm, int pass, int bytes, const MemberDev*& md, int& q,
                                                  long long& group, double*& smem)
{
    extern __shared__ double line_smem[];
    const int m = find_member(off, nm, blockIdx.x);
    md = mem + m;
    const int N = md->grid.npts;
    if constexpr (WARPS == 1) {
        const long long local = blockIdx.x - off[m], groups = spline_groups(pass, N, md->grid.pad);
        q = (int)(local / groups);
        group = local - q * groups;
        smem = line_smem;
        return true;
    }
    const int warp = threadIdx.x >> 5, per = resident_per_block(N, blockDim.x >> 5, bytes);
    const long long groups = spline_groups(pass, N, md->grid.pad), blocks = (groups + per - 1) / per;
    const long long local = blockIdx.x - off[m];
    q = (int)(local / blocks);
    group = (local - q * blocks) * per + warp;
    smem = line_smem + warp * (resident_bytes(N) / (int)sizeof(double));
    return warp < per && group < groups;
}

template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) ensemble_resident0(const MemberDev* __restrict__ mem,
                                                                  const long long* __restrict__ off, int nm,
                                                                  int buf, int bytes)
{
    const MemberDev* md;
    int q;
    long long group;
    double* smem;
    if (!ensemble_resident<WARPS>(mem, off, nm, 0, bytes, md, q, group, smem)) return;
    resident_pass0<true>(md->buf[buf], md->fc, md->grid, md->tb, q + 1, md->coef[q],
                         (long long)md->grid.npts * md->grid.npts, group, smem);
}
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) ensemble_resident1(const MemberDev* __restrict__ mem,
                                                                  const long long* __restrict__ off, int nm,
                                                                  int bytes)
{
    const MemberDev* md;
    int q;
    long long group;
    double* smem;
    if (!ensemble_resident<WARPS>(mem, off, nm, 1, bytes, md, q, group, smem)) return;
    resident_pass1(md->coef[q], md->grid.npts, md->grid, md->tb, md->scratch[q], group, smem);
}
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS) ensemble_resident2(const MemberDev* __restrict__ mem,
                                                                  const long long* __restrict__ off, int nm,
                                                                  int bytes)
{
    const MemberDev* md;
    int q;
    long long group;
    double* smem;
    if (!ensemble_resident<WARPS>(mem, off, nm, 2, bytes, md, q, group, smem)) return;
    resident_pass2<double>(md->scratch[q], md->grid, md->tb, md->coef[q], group, smem);
}

__global__ void __launch_bounds__(128, kPassCtasPerSm) ensemble_pass0_kernel(const MemberDev* __restrict__ mem, const long long* __restrict__ off, int nm,
                                      int buf)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = off[nm];
    for (long long w = (long long)blockIdx.x * 4 + warp; w < total; w += (long long)gridDim.x * 4) {
        int q;
        long long group;
        const MemberDev& md = ensemble_group(mem, off, nm, w, 0, q, group);
        const long long L = group * 32 + lane;
        if (L < (long long)md.grid.npts * md.grid.npts)
            pass0_line<kLineBatch0, true>(md.buf[buf], md.fc, md.grid, md.tb, q + 1, md.coef[q], L);
    }
}

__global__ void __launch_bounds__(128, kPassCtasPerSm) ensemble_pass1_kernel(const MemberDev* __restrict__ mem, const long long* __restrict__ off, int nm)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long total = off[nm];
    for (long long w = (long long)blockIdx.x * 4 + warp; w < total; w += (long long)gridDim.x * 4) {
        int q;
        long long group;
        const MemberDev& md = ensemble_group(mem, off, nm, w, 1, q, group);
        const long long L = group * 32 + lane;
        if (L < (long long)(md.grid.npts + md.grid.pad) * md.grid.npts)
            pass1_line<kLineBatch1Batched>(md.coef[q], md.grid, md.tb, md.scratch[q], L);
    }
}

__global__ void __launch_bounds__(32 * kPass2Warps, kPassCtasPerSm)
    ensemble_pass2_kernel(const MemberDev* __restrict__ mem, const long long* __restrict__ off, int nm)
{
    __shared__ double stage[kPass2Warps][32][kLineChunk + 1];
    const int warp = threadIdx.x >> 5;
    const long long total = off[nm];
    for (long long w = (long long)blockIdx.x * kPass2Warps + warp; w < total; w += (long long)gridDim.x * kPass2Warps) {
        int q;
        long long group;
        const MemberDev& md = ensemble_group(mem, off, nm, w, 2, q, group);
        const long long M = md.grid.npts + md.grid.pad;
        pass2_group(md.scratch[q], md.grid, md.tb, md.coef[q], group * 32, M * M, stage[warp]);
    }
}

__global__ void ensemble_heun_kernel(const MemberDev* __restrict__ mem, const long long* __restrict__ off, int nm)
{
    const long long total = off[nm];
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < total; x += (long long)gridDim.x * blockDim.x) {
        const int m = find_member(off, nm, x);
        const MemberDev& md = mem[m];
        const Coefs3 cf{{md.coef[0], md.coef[1], md.coef[2]}};
        const ParticleArrays P{{md.P[0], md.P[1], md.P[2], md.P[3], md.P[4], md.P[5]}};
        heun_particle<double>(cf, md.grid, md.clock->dt, x - off[m], P, P);
    }
}

// the line kernels' shared-memory limit, on the current device
cudaError_t resident_prepare()
{
    const int bytes = resident_bytes(kResidentSingle > kResidentBatched ? kResidentSingle : kResidentBatched);
    const void* kernels[] = {(const void*)spline_resident0<true>,    (const void*)spline_resident0<false>,
                             (const void*)spline_resident1,          (const void*)spline_resident2<double>,
                             (const void*)spline_resident2<float>,   (const void*)ensemble_resident0<1>,
                             (const void*)ensemble_resident1<1>,     (const void*)ensemble_resident2<1>,
                             (const void*)ensemble_resident0<kEnsembleWarps>,
                             (const void*)ensemble_resident1<kEnsembleWarps>,
                             (const void*)ensemble_resident2<kEnsembleWarps>};
    for (const void* k : kernels) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// one component (kind q) through resident lines: pass 0 to `mid` (stride0 along axis 0), pass 1 to `buf`
// (from in_rows rows per plane), pass 2 to out
template <class OutT>
cudaError_t resident_component(const double* W, const FieldConst& fc, const SplineGrid& g, const SplineTables& tb, int q,
                               double* mid, long long stride0, int in_rows, double* buf, OutT* out, cudaStream_t s)
{
    const int smem = resident_bytes(g.npts);
    const unsigned g0 = (unsigned)spline_groups(0, g.npts, g.pad), g1 = (unsigned)spline_groups(1, g.npts, g.pad),
                   g2 = (unsigned)spline_groups(2, g.npts, g.pad);
    if (q >= 1 && q <= 3) spline_resident0<true><<<g0, 32, smem, s>>>(W, fc, g, tb, q, mid, stride0);
    else spline_resident0<false><<<g0, 32, smem, s>>>(W, fc, g, tb, q, mid, stride0);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    spline_resident1<<<g1, 32, smem, s>>>(mid, in_rows, g, tb, buf);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    spline_resident2<OutT><<<g2, 32, smem, s>>>(buf, g, tb, out);
    return cudaGetLastError();
}

cudaError_t launch_pass2(const double* in, const SplineGrid& g, const SplineTables& tb, double* out, cudaStream_t s)
{
    const long long M = g.npts + g.pad;
    long long b = (M * M + 32 * kPass2Warps - 1) / (32 * kPass2Warps);
    if (b < 1) b = 1;
    if (b > 148 * 16) b = 148 * 16;
    spline_pass2<<<(unsigned)b, 32 * kPass2Warps, 0, s>>>(in, g, tb, out);
    return cudaGetLastError();
}

}  // namespace

cudaError_t spline_prepare() { return resident_prepare(); }

cudaError_t launch_spline_build(const double* W, const FieldConst& fc, const SplineGrid& g, const SplineTables& tb,
                                double* coef_u, double* coef_v, double* coef_w, double* scratch, cudaStream_t s)
{
    double* outs[3] = {coef_u, coef_v, coef_w};
    for (int f = 0; f < 3; f++) {
        cudaError_t e = launch_spline_component(W, fc, g, tb, f + 1, outs[f], scratch, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// one velocity component (1 = u, 2 = v, 3 = w) with caller-provided scratch and tables
cudaError_t launch_spline_component(const double* W, const FieldConst& fc, const SplineGrid& g, const SplineTables& tb,
                                    int component, double* coef, double* scratch, cudaStream_t s)
{
    const long long N = g.npts, M = N + g.pad;
    if (N <= kResidentSingle) return resident_component(W, fc, g, tb, component, coef, N * N, (int)N, scratch, coef, s);
    const bool vel = component >= 1 && component <= 3;
    cudaError_t e = vel ? grid_launch(spline_pass0<true>, N * N, 128, s, W, fc, g, tb, component, coef)
                        : grid_launch(spline_pass0<false>, N * N, 128, s, W, fc, g, tb, component, coef);
    if (e != cudaSuccess) return e;
    e = grid_launch(spline_pass1, M * N, 128, s, (const double*)coef, g, tb, scratch);
    if (e != cudaSuccess) return e;
    return launch_pass2((const double*)scratch, g, tb, coef, s);
}

SplineLaunch spline_launch(const int* npts, int count)
{
    const int most = *std::max_element(npts, npts + count), least = *std::min_element(npts, npts + count);
    if (most > kResidentBatched) return {0, 0};
    constexpr int kPerSm = 228 * 1024, kReserved = 1024;   // an SM's shared memory, and what it keeps of it per block
    const int bytes = resident_bytes(most), ctas = kPerSm / (bytes + kReserved);
    const int smem = (kPerSm / (ctas < 32 ? ctas : 32) - kReserved) & ~15;
    const int warps = resident_per_block(least, kEnsembleWarps, smem);
    // Blocks of several groups where they save a tenth of the groups' time, taken as points over groups per SM: below
    // that their longer code decides (16 members of 32^3 to 2 of 96^3, 7 % by this count: 0.432 -> 0.446 ms; 30 of
    // 32^3 and 2 of 96^3, 22 %: 0.282 -> 0.260; 31 of 32^3 and one of 194^3, 13 %: 0.847 -> 0.728).
    double single = 0.0, packed = 0.0;
    for (int k = 0; k < count; k++) {
        const double points = (double)npts[k] * npts[k] * npts[k];
        single += points;
        packed += points / resident_per_block(npts[k], warps, smem);
    }
    if (packed > 0.9 * single) return {1, bytes};
    return {warps, smem};
}
long long spline_items(int pass, int npts, int pad, const SplineLaunch& l)
{
    const long long groups = spline_groups(pass, npts, pad), per = l.warps ? resident_per_block(npts, l.warps, l.smem) : 1;
    return 3 * ((groups + per - 1) / per);
}

template <int WARPS>
static cudaError_t ensemble_resident_t(const MemberDev* mem, const EnsembleWork& w, const long long totals[3], int nm,
                                       const SplineLaunch& l, int buf, cudaStream_t s)
{
    const int threads = 32 * l.warps;
    ensemble_resident0<WARPS><<<(unsigned)totals[0], threads, l.smem, s>>>(mem, w.group0, nm, buf, l.smem);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ensemble_resident1<WARPS><<<(unsigned)totals[1], threads, l.smem, s>>>(mem, w.group1, nm, l.smem);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ensemble_resident2<WARPS><<<(unsigned)totals[2], threads, l.smem, s>>>(mem, w.group2, nm, l.smem);
    return cudaGetLastError();
}

cudaError_t launch_ensemble_splines(const MemberDev* mem, const EnsembleWork& w, const long long totals[3], int nm,
                                    const SplineLaunch& l, int buf, cudaStream_t s)
{
    if (l.warps == 1) return ensemble_resident_t<1>(mem, w, totals, nm, l, buf, s);
    if (l.warps > 1) return ensemble_resident_t<kEnsembleWarps>(mem, w, totals, nm, l, buf, s);
    cudaError_t e = grid_launch(ensemble_pass0_kernel, totals[0] * 32, 128, s, mem, w.group0, nm, buf);
    if (e != cudaSuccess) return e;
    e = grid_launch(ensemble_pass1_kernel, totals[1] * 32, 128, s, mem, w.group1, nm);
    if (e != cudaSuccess) return e;
    long long b = (totals[2] + kPass2Warps - 1) / kPass2Warps;
    if (b < 1) b = 1;
    if (b > 148 * 16) b = 148 * 16;
    ensemble_pass2_kernel<<<(unsigned)b, 32 * kPass2Warps, 0, s>>>(mem, w.group2, nm);
    return cudaGetLastError();
}

cudaError_t launch_ensemble_heun(const MemberDev* mem, const long long* off, int nm, long long total, cudaStream_t s)
{
    if (total <= 0) return cudaSuccess;
    return grid_launch(ensemble_heun_kernel, total, 128, s, mem, off, nm);
}

// spline of an arbitrary source (spline_source kinds) with caller scratch
cudaError_t launch_spline_source(const double* src, const FieldConst& fc, const SplineGrid& g, const SplineTables& tb,
                                 int kind, double* coef, double* scratch, cudaStream_t s)
{
    return launch_spline_component(src, fc, g, tb, kind, coef, scratch, s);
}

cudaError_t launch_lap_nodes(const double* coef, const SplineGrid& g, const FieldConst& fc, double* out, cudaStream_t s)
{
    const long long N = g.npts;
    return grid_launch(lap_nodes_kernel, N * N * N, 128, s, coef, g, fc, out);
}

cudaError_t launch_particle_export(long long np, const long long* tag, double* const src[3], double* const dst[3],
                                   DevClock* clock, cudaStream_t s)
{
    if (np <= 0) return cudaSuccess;
    return grid_launch(particle_export_kernel, np, 256, s, np, tag, Triple{{src[0], src[1], src[2]}},
                       Triple{{dst[0], dst[1], dst[2]}}, clock);
}

cudaError_t launch_particle_import(long long np, double* const src[3], double* const dst[3], long long* tag,
                                   DevClock* clock, cudaStream_t s)
{
    return grid_launch(particle_import_kernel, np, 256, s, np, Triple{{src[0], src[1], src[2]}},
                       Triple{{dst[0], dst[1], dst[2]}}, tag, clock);
}

cudaError_t launch_particle_props(const double* const coefs[8], const SplineGrid& g, long long np, const double* py,
                                  const double* px, const double* pz, const long long* tag, double* props,
                                  DevClock* clock, cudaStream_t s)
{
    if (np <= 0) return cudaSuccess;
    Coefs8 cf;
    for (int q = 0; q < 8; q++) cf.c[q] = coefs[q];
    return grid_launch(particle_props_kernel, np, 128, s, cf, g, np, py, px, pz, tag, props, clock);
}

cudaError_t launch_particle_stats(const double* props, long long np, StatsPartial* partials, int nblocks, double* out6,
                                  cudaStream_t s)
{
    particle_stats_kernel<<<nblocks, 256, 0, s>>>(props, np, partials);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    particle_stats_finish<<<1, 6 * 32, 0, s>>>(partials, nblocks, out6);
    return cudaGetLastError();
}

template <class CT>
static cudaError_t particles_eval_t(const CT* const coefs[3], const SplineGrid& g, long long np, const double* py,
                                    const double* px, const double* pz, double* Uu, double* Uv, double* Uw,
                                    cudaStream_t s)
{
    if (np <= 0) return cudaSuccess;
    Coefs3T<CT> cf{{coefs[0], coefs[1], coefs[2]}};
    return grid_launch(particles_eval_kernel<CT>, np, 128, s, cf, g, np, py, px, pz, Uu, Uv, Uw);
}

cudaError_t launch_particles_eval(const double* const coefs[3], const SplineGrid& g, long long np, const double* py,
                                  const double* px, const double* pz, double* Uu, double* Uv, double* Uw,
                                  cudaStream_t s)
{
    return particles_eval_t<double>(coefs, g, np, py, px, pz, Uu, Uv, Uw, s);
}

cudaError_t launch_particles_eval(const float* const coefs[3], const SplineGrid& g, long long np, const double* py,
                                  const double* px, const double* pz, double* Uu, double* Uv, double* Uw,
                                  cudaStream_t s)
{
    return particles_eval_t<float>(coefs, g, np, py, px, pz, Uu, Uv, Uw, s);
}

template <class CT>
static cudaError_t particles_heun_t(const CT* const coefs[3], const SplineGrid& g, const DevClock* clock, long long np,
                                    const ParticleArrays& src, const ParticleArrays& dst, const long long* tag_src,
                                    long long* tag_dst, cudaStream_t s)
{
    if (np <= 0) return cudaSuccess;
    Coefs3T<CT> cf{{coefs[0], coefs[1], coefs[2]}};
    return grid_launch(particles_heun_kernel<CT>, np, 128, s, cf, g, clock, np, src, dst, tag_src, tag_dst);
}

cudaError_t launch_particles_heun(const double* const coefs[3], const SplineGrid& g, const DevClock* clock, long long np,
                                  const ParticleArrays& src, const ParticleArrays& dst, const long long* tag_src,
                                  long long* tag_dst, cudaStream_t s)
{
    return particles_heun_t<double>(coefs, g, clock, np, src, dst, tag_src, tag_dst, s);
}

cudaError_t launch_particles_heun(const float* const coefs[3], const SplineGrid& g, const DevClock* clock, long long np,
                                  const ParticleArrays& src, const ParticleArrays& dst, const long long* tag_src,
                                  long long* tag_dst, cudaStream_t s)
{
    return particles_heun_t<float>(coefs, g, clock, np, src, dst, tag_src, tag_dst, s);
}

int scan_temp_size(long long n)
{
    long long total = 0;
    for (long long m = (n + kScanChunk - 1) / kScanChunk; m > 1; m = (m + kScanChunk - 1) / kScanChunk) total += m;
    return (int)(total + 1);
}

// exclusive scan of data[0, n) in place; temp holds scan_temp_size(n) values
static cudaError_t scan_exclusive(unsigned* data, long long n, unsigned* temp, int* launches, cudaStream_t s)
{
    const long long chunks = (n + kScanChunk - 1) / kScanChunk;
    if (chunks <= 1) {
        scan_chunks_kernel<<<1, 256, 0, s>>>(data, n, nullptr);
        *launches += 1;
        return cudaGetLastError();
    }
    scan_chunks_kernel<<<(unsigned)chunks, 256, 0, s>>>(data, n, temp);
    *launches += 1;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = scan_exclusive(temp, chunks, temp + chunks, launches, s);
    if (e != cudaSuccess) return e;
    long long b = (n + 255) / 256;
    if (b > 148 * 16) b = 148 * 16;
    scan_add_kernel<<<(unsigned)b, 256, 0, s>>>(data, n, temp);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_particle_sort(const SplineGrid& g, long long np, const ParticleArrays& src, const ParticleArrays& dst,
                                 const long long* tag_src, long long* tag_dst, unsigned* keys, unsigned* counts,
                                 unsigned* temp, int* launches, cudaStream_t s)
{
    if (np <= 0) return cudaSuccess;
    const int nb = (g.npts + 7) / 8;
    const long long nkeys = (long long)nb * nb * nb;
    cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(unsigned) * (size_t)nkeys, s);
    if (e != cudaSuccess) return e;
    e = grid_launch(particle_keys_kernel, np, 256, s, g, nb, np, src, keys, counts);
    if (e != cudaSuccess) return e;
    *launches += 1;   // the memset is a copy-engine operation, not a kernel
    e = scan_exclusive(counts, nkeys, temp, launches, s);
    if (e != cudaSuccess) return e;
    return grid_launch(particle_scatter_kernel, np, 256, s, np, (const unsigned*)keys, counts, src, dst, tag_src, tag_dst);
}

template <class CT>
static cudaError_t stats_t(const double* W, const FieldConst& fc, const SplineGrid& g, const CT* const coefs[3],
                           StatsPartial* partials, int nblocks, double* out, cudaStream_t s)
{
    Coefs3T<CT> cf{{coefs[0], coefs[1], coefs[2]}};
    const double ncells = (double)fc.n * fc.n * fc.n;
    stats_kernel<0, CT><<<nblocks, 256, 0, s>>>(W, fc, g, cf, nullptr, partials);
    stats_finish<<<1, 16 * 32, 0, s>>>(partials, nblocks, ncells, 0, out);
    // means of p, T, 1/rho sit in out[12..14]
    stats_kernel<1, CT><<<nblocks, 256, 0, s>>>(W, fc, g, cf, out + 12, partials);
    stats_finish<<<1, 16 * 32, 0, s>>>(partials, nblocks, ncells, 1, out);
    return cudaGetLastError();
}

cudaError_t launch_stats(const double* W, const FieldConst& fc, const SplineGrid& g, const double* const coefs[3],
                         StatsPartial* partials, int nblocks, double* out, cudaStream_t s)
{
    return stats_t<double>(W, fc, g, coefs, partials, nblocks, out, s);
}

cudaError_t launch_stats(const double* W, const FieldConst& fc, const SplineGrid& g, const float* const coefs[3],
                         StatsPartial* partials, int nblocks, double* out, cudaStream_t s)
{
    return stats_t<float>(W, fc, g, coefs, partials, nblocks, out, s);
}

cudaError_t launch_spline_build_f32(const double* W, const FieldConst& fc, const SplineGrid& g, const SplineTables& tb,
                                    float* coef_u, float* coef_v, float* coef_w, double* buf, cudaStream_t s)
{
    float* outs[3] = {coef_u, coef_v, coef_w};
    const long long N = g.npts, M = N + g.pad;
    for (int f = 0; f < 3; f++) {
        if (N <= kResidentSingle) {
            cudaError_t e = resident_component(W, fc, g, tb, f + 1, buf, M * N, (int)M, buf, outs[f], s);
            if (e != cudaSuccess) return e;
            continue;
        }
        cudaError_t e = grid_launch(spline_pass0_room, N * N, 128, s, W, fc, g, tb, f + 1, buf);
        if (e != cudaSuccess) return e;
        e = grid_launch(spline_pass1_inplace, M * N, 128, s, buf, g, tb);
        if (e != cudaSuccess) return e;
        long long b = (M * M + 32 * kPass2Warps - 1) / (32 * kPass2Warps);
        if (b < 1) b = 1;
        if (b > 148 * 16) b = 148 * 16;
        spline_pass2_f32<<<(unsigned)b, 32 * kPass2Warps, 0, s>>>(buf, g, tb, outs[f]);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace gkm
