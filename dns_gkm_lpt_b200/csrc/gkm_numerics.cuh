// Device numerics of the gas-kinetic step: WENO-SYMOO reconstruction and the
// BGK flux integrated over one time step.  Templated on the arithmetic type T
// (double for the FP64 drop-in, float for the mixed-precision form).
//
// Mathematics follow the reference CPU path:
//   WENO-SYMOO        src/update.cpp:556-680
//   flux              src/GKMflux.cpp:11-229
//   moment products   src/GKMflux.cpp:238-278 (MCal)
//   slope solve       src/GKMflux.cpp:283-297
//   c2p               src/GKMflux.cpp:302-309
//
// Two forms of the flux.  gks_flux_mcal keeps the reference's moment algebra
// (one MCal per table, weight and slope vector) and is what the operation
// counter measures.  gks_flux_peculiar, the one the kernels run, takes the same
// moments of the same slope vectors in the velocity frame of each state, where
// most of them are closed forms, and forms each reciprocal once (grouped
// divisions, one reciprocal square root per state).  The two forms and the
// reference differ only by rounding.
#pragma once

#include <math.h>

#include <type_traits>
#include <utility>

#ifdef __CUDACC__
#include <cuda_runtime.h>
#define GKM_HD __host__ __device__ __forceinline__
#include "f32x2.cuh"
#else
// host-only compilation (op counting, CPU checks of the device numerics)
#include <algorithm>
#include <cmath>
#define GKM_HD inline
#endif

// GKM_REFERENCE_FORM 1 keeps the reference's arithmetic in the shared helpers
// (two divisions per WENO scalar, the divisions of temperature and face energy)
// and its MCal moment algebra; the operation counter compiles that form.  The
// kernels (0) form each reciprocal once and take the moments in the peculiar frames.
#ifndef GKM_REFERENCE_FORM
#define GKM_REFERENCE_FORM 0
#endif

namespace gkm {

// single-precision arithmetic: float, and the packed pair F2 (f32x2.cuh)
template <class T>
struct single_t {
    static constexpr bool value = sizeof(T) == 4;
};
#ifdef __CUDACC__
template <>
struct single_t<F2> {
    static constexpr bool value = true;
};
#endif

constexpr double kR = 287.0;        // gas constant, src/param.h:21
constexpr double kPrandtl = 0.70;   // src/param.h:19
constexpr double kWenoEps = 1e-10;  // pow(10,-10), src/param.h:18

// 1/x.  In double precision on the device the hardware's approximate reciprocal (20 bits) with one
// third-order step in fused multiply-adds, r + r (e + e^2), e = 1 - x r (Newton's iteration carried one
// term further): within an ulp for normal x and 1/x (0.505 measured), four dependent instructions and no
// branch, where a division takes about ten and a branch.  Zero, infinite and subnormal x give NaN, a
// subnormal 1/x is 0.  The sweeps wait on these
// chains (256^3 FP64 step 11.99 -> 11.08 ms, with the reciprocal square roots and the constants of K
// taken from the launch).
template <class T>
GKM_HD T recip(T x)
{
    return T(1) / x;
}
#ifdef __CUDACC__
template <>
GKM_HD double recip<double>(double x)
{
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
#else
    return 1.0 / x;
#endif
}
#endif

template <class T>
struct Phys {
    T gam;        // ratio of specific heats
    T gm1;        // gam - 1
    T Rg;         // gas constant in the working units
    int K;        // internal degrees of freedom (int((5-3g)/(g-1)))
    // K + 2 .. K + 7 and 1 / (Pr (K + 3)) as the flux uses them (the sweeps take them from the launch's
    // constants, so they occupy no registers)
    T k2 = T(K + 2), k3 = T(K + 3), k4 = T(K + 4), k5 = T(K + 5), k7 = T(K + 7);
    T iK3 = T(1) / T(K + 3), iPrK3 = T(1.0 / kPrandtl) * (T(1) / T(K + 3));
    // twice what the energy of a Maxwellian with K internal degrees of freedom exceeds p / (gam - 1) by,
    // over p: zero but for rounding where (5-3g)/(g-1) is whole
    T dK2 = T(K + 3) - T(2) / gm1;
};

// ---------------------------------------------------------------- WENO ----
// One scalar, both sides of the face between cells L (=a1) and R (=b1).
// a3, a2, a1 = cells L-2, L-1, L ; b1, b2, b3 = cells R, R+1, R+2.
// Linear weights 1/20, 9/20, 9/20, 1/20; IS_3 replaced by max(IS_0..IS_3);
// alpha_k = g_k / (eps + IS_k).
#if GKM_REFERENCE_FORM
// the reference's arithmetic, the normalised weights formed with one division per side:
// w_k = g_k prod_{m!=k}(eps+IS_m) / sum_m g_m prod_{m'!=m}(eps+IS_m')
template <class T>
GKM_HD void weno_scalar(T a3, T a2, T a1, T b1, T b2, T b3, T eps, T& fl, T& fr)
{
    const T c13 = T(1.0 / 3.0), c76 = T(7.0 / 6.0), c116 = T(11.0 / 6.0), c16 = T(1.0 / 6.0), c56 = T(5.0 / 6.0);
    const T c1312 = T(13.0 / 12.0), c14 = T(0.25);
    // candidate polynomials (left-biased "p", right-biased "n")
    T P0p = a3 * c13 - a2 * c76 + a1 * c116;
    T P0n = b3 * c13 - b2 * c76 + b1 * c116;
    T P1p = -a2 * c16 + a1 * c56 + b1 * c13;
    T P1n = -b2 * c16 + b1 * c56 + a1 * c13;
    T P2p = a1 * c13 + b1 * c56 - b2 * c16;
    T P2n = b1 * c13 + a1 * c56 - a2 * c16;
    T P3p = b1 * c116 - b2 * c76 + b3 * c13;
    T P3n = a1 * c116 - a2 * c76 + a3 * c13;
    // smoothness indicators
    T d;
    T e;
    d = a3 - T(2) * a2 + a1; e = a3 - T(4) * a2 + T(3) * a1; T I0p = c1312 * d * d + c14 * e * e;
    d = b3 - T(2) * b2 + b1; e = b3 - T(4) * b2 + T(3) * b1; T I0n = c1312 * d * d + c14 * e * e;
    d = a2 - T(2) * a1 + b1; e = b1 - a2;                    T I1p = c1312 * d * d + c14 * e * e;
    d = b2 - T(2) * b1 + a1; e = a1 - b2;                    T I1n = c1312 * d * d + c14 * e * e;
    d = a1 - T(2) * b1 + b2; e = -T(3) * a1 + T(4) * b1 - b2; T I2p = c1312 * d * d + c14 * e * e;
    d = b1 - T(2) * a1 + a2; e = -T(3) * b1 + T(4) * a1 - a2; T I2n = c1312 * d * d + c14 * e * e;
    d = b1 - T(2) * b2 + b3; e = -T(5) * b1 + T(8) * b2 - T(3) * b3; T I3p = c1312 * d * d + c14 * e * e;
    d = a1 - T(2) * a2 + a3; e = -T(5) * a1 + T(8) * a2 - T(3) * a3; T I3n = c1312 * d * d + c14 * e * e;
    I3p = fmax(fmax(fmax(I0p, I1p), I2p), I3p);
    I3n = fmax(fmax(fmax(I0n, I1n), I2n), I3n);
    {
        T e0 = eps + I0p, e1 = eps + I1p, e2 = eps + I2p, e3 = eps + I3p;
        T p01 = e0 * e1, p23 = e2 * e3;
        T n0 = e1 * p23, n1 = T(9) * e0 * p23, n2 = T(9) * p01 * e3, n3 = p01 * e2;
        fl = (n0 * P0p + n1 * P1p + n2 * P2p + n3 * P3p) / (n0 + n1 + n2 + n3);
    }
    {
        T e0 = eps + I0n, e1 = eps + I1n, e2 = eps + I2n, e3 = eps + I3n;
        T p01 = e0 * e1, p23 = e2 * e3;
        T n0 = e1 * p23, n1 = T(9) * e0 * p23, n2 = T(9) * p01 * e3, n3 = p01 * e2;
        fr = (n0 * P0n + n1 * P1n + n2 * P2n + n3 * P3n) / (n0 + n1 + n2 + n3);
    }
}
#else
// The kernels' form works on the five differences of neighbouring cells.  The left-biased
// candidate k and the right-biased candidate 3-k are the same polynomial of the same three
// cells, and so are the second differences of their indicators, so four of each serve both
// sides; a candidate is a1 + delta/6.  The indicators are taken four times over, 4 (eps + IS) =
// (13/3 d^2 + 4 eps) + e^2, which leaves the weights as they are: 64 operations for both sides
// where candidates and indicators of the cell values took 112.
// Measured at 256^3 (a step, default shapes): FP64 13.97 -> 13.00 ms, mixed 8.26 -> 8.05 ms; the
// reconstructed values' error against extended precision is a tenth (FP64) and a third (FP32) of
// that of the candidates formed from cell values.

// the larger of two indicators (positive): on the device by their bit patterns, which keeps the
// comparison off the FP64 pipe
template <class T>
GKM_HD T imax(T a, T b)
{
    return fmax(a, b);
}
#ifdef __CUDACC__
template <>
GKM_HD double imax<double>(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
#else
    return a < b ? b : a;
#endif
}
#endif

template <class T>
struct WenoParts {
    T d0, d1, d2, d3;        // six times (candidate - a1), 9 times that for the middle two (their linear
                             // weight against the outer two's): the left side's 0..3, the right side's 3..0
    T l0, l1, l2, l3;        // 4 (eps + IS) of the left side
    T r0, r1, r2, r3;        // and of the right side
};

template <class T>
GKM_HD WenoParts<T> weno_parts(T a3, T a2, T a1, T b1, T b2, T b3, T eps)
{
    const T f1 = a2 - a3, f2 = a1 - a2, f3 = b1 - a1, f4 = b2 - b1, f5 = b3 - b2;
    const T c = T(13.0 / 3.0), e4 = T(4) * eps;
    const T dA = f2 - f1, dB = f3 - f2, dC = f4 - f3, dD = f5 - f4;
    const T qA = c * dA * dA + e4, qB = c * dB * dB + e4, qC = c * dC * dC + e4, qD = c * dD * dD + e4;
    WenoParts<T> w;
    const T el = T(3) * f2 - f1, er = T(3) * f4 - f5;
    T e;
    w.l0 = qA + el * el;
    e = f2 + f3;                 w.l1 = qB + e * e;
    e = T(3) * f3 - f4;          w.l2 = qC + e * e;
    e = er - T(2) * dD;          w.l3 = qD + e * e;   // 5 f4 - 3 f5
    w.r0 = qD + er * er;
    e = f3 + f4;                 w.r1 = qC + e * e;
    e = T(3) * f3 - f2;          w.r2 = qB + e * e;
    e = el + T(2) * dA;          w.r3 = qA + e * e;   // 5 f2 - 3 f1
    w.l3 = imax<T>(imax<T>(w.l0, w.l1), imax<T>(w.l2, w.l3));
    w.r3 = imax<T>(imax<T>(w.r0, w.r1), imax<T>(w.r2, w.r3));
    w.d0 = T(2) * el - f2;                       // 5 f2 - 2 f1
    w.d1 = T(18) * f3 + T(9) * f2;
    w.d2 = T(36) * f3 - T(9) * f4;
    w.d3 = T(6) * f3 - T(T(2) * er - f4);        // 6 f3 - 5 f4 + 2 f5
    return w;
}

// double precision: fl = a1 + Nl / (6 Dl), fr = a1 + Nr / (6 Dr), so a caller can share one division
// among several scalars
template <class T>
GKM_HD void weno_nd(T a3, T a2, T a1, T b1, T b2, T b3, T eps, T& Nl, T& Dl, T& Nr, T& Dr)
{
    const WenoParts<T> w = weno_parts<T>(a3, a2, a1, b1, b2, b3, eps);
    const T n = T(9);
    {
        const T p01 = w.l0 * w.l1, p23 = w.l2 * w.l3;
        Nl = p23 * (w.l1 * w.d0 + w.l0 * w.d1) + p01 * (w.l3 * w.d2 + w.l2 * w.d3);
        Dl = p23 * (n * w.l0 + w.l1) + p01 * (n * w.l3 + w.l2);
    }
    {
        const T p01 = w.r0 * w.r1, p23 = w.r2 * w.r3;
        Nr = p23 * (w.r1 * w.d3 + w.r0 * w.d2) + p01 * (w.r3 * w.d1 + w.r2 * w.d0);
        Dr = p23 * (n * w.r0 + w.r1) + p01 * (n * w.r3 + w.r2);
    }
}

template <class T>
GKM_HD void weno_scalar(T a3, T a2, T a1, T b1, T b2, T b3, T eps, T& fl, T& fr)
{
    if constexpr (single_t<T>::value) {
        // single precision: products of three (eps + IS) underflow on flat stencils, so the
        // candidates 2 and 3 enter with the ratio (IS_0 IS_1) / (IS_2 IS_3), at most IS_0 / IS_2
        // because IS_3 is the largest; eps is such that a product of two is a normal number
        const WenoParts<T> w = weno_parts<T>(a3, a2, a1, b1, b2, b3, eps);
        const T n = T(9), c16 = T(1.0 / 6.0);
        {
            const T t = (w.l0 * w.l1) / (w.l2 * w.l3);
            const T x = w.l1 * w.d0 + w.l0 * w.d1, y = w.l3 * w.d2 + w.l2 * w.d3;
            const T u = n * w.l0 + w.l1, v = n * w.l3 + w.l2;
            fl = a1 + c16 * T((x + t * y) / (u + t * v));
        }
        {
            const T t = (w.r0 * w.r1) / (w.r2 * w.r3);
            const T x = w.r1 * w.d3 + w.r0 * w.d2, y = w.r3 * w.d1 + w.r2 * w.d0;
            const T u = n * w.r0 + w.r1, v = n * w.r3 + w.r2;
            fr = a1 + c16 * T((x + t * y) / (u + t * v));
        }
    } else {
        T Nl, Dl, Nr, Dr;
        weno_nd<T>(a3, a2, a1, b1, b2, b3, eps, Nl, Dl, Nr, Dr);
        // both sides with one division: D ranges from about 80 (4 eps)^3 (flat stencil) to about
        // 64 IS_max^3, so Dl Dr stays far inside the double range for any physical state
        const T inv = T(1.0 / 6.0) * recip<T>(Dl * Dr);
        fl = a1 + Nl * (Dr * inv);
        fr = a1 + Nr * (Dl * inv);
    }
}
#endif

// temperature of a conserved state, src/update.cpp:615-620
template <class T>
GKM_HD T temperature(T r, T m1, T m2, T m3, T E, const Phys<T>& ph)
{
#if GKM_REFERENCE_FORM
    T ir = T(1) / r;
    return ph.gm1 * (E * ir - T(0.5) * (m1 * m1 + m2 * m2 + m3 * m3) * ir * ir) / ph.Rg;
#else
    const T ir = recip<T>(r);
    return (E - (T(0.5) * (m1 * m1 + m2 * m2 + m3 * m3)) * ir) * (ir * (ph.gm1 / ph.Rg));
#endif
}

// face energy from reconstructed rho, momentum and temperature, src/update.cpp:673-674
template <class T>
GKM_HD T face_energy(T r, T m1, T m2, T m3, T Tf, const Phys<T>& ph)
{
#if GKM_REFERENCE_FORM
    return r * ph.Rg * Tf / ph.gm1 + T(0.5) * (m1 * m1 + m2 * m2 + m3 * m3) / r;
#else
    return r * Tf * (ph.Rg / ph.gm1) + T(0.5) * (m1 * m1 + m2 * m2 + m3 * m3) * recip<T>(r);
#endif
}

// face energy with 1/r given (the sweeps form the two sides' reciprocals together)
template <class T>
GKM_HD T face_energy_ir(T r, T ir, T m1, T m2, T m3, T Tf, const Phys<T>& ph)
{
    return r * Tf * (ph.Rg / ph.gm1) + T(0.5) * (m1 * m1 + m2 * m2 + m3 * m3) * ir;
}

// ------------------------------------------------------ moment tables ----
// Maxwellian moments of one state: x half-space table H (and H2 for the
// equilibrium state's other half), full tables X (x), Y (y), Z (z).
// src/GKMflux.cpp:45-68 (l, r) and :85-103 (e).

template <class T>
struct Moments {
    T H[7];
    T X[7];
    T Y[6], Z[6];
    T Ie2, Ie4;
};

template <class T>
GKM_HD T erfc_t(T x);
template <>
GKM_HD double erfc_t<double>(double x) { return ::erfc(x); }
template <>
GKM_HD float erfc_t<float>(float x) { return erfcf(x); }
template <class T>
GKM_HD T exp_t(T x);
template <>
GKM_HD double exp_t<double>(double x) { return exp(x); }
template <>
GKM_HD float exp_t<float>(float x) { return expf(x); }
template <class T>
GKM_HD T sqrt_t(T x);
template <>
GKM_HD double sqrt_t<double>(double x) { return sqrt(x); }
template <>
GKM_HD float sqrt_t<float>(float x) { return sqrtf(x); }
// 1 / sqrt(x) for normal x > 0, within 2 ulp (0.99 measured, 0.51 with CUDA's rsqrt); zero, infinite and negative
// x give NaN, subnormal x infinity; on the host 1 / sqrt
template <class T>
GKM_HD T rsqrt_t(T x);
template <>
GKM_HD double rsqrt_t<double>(double x)
{
#ifdef __CUDA_ARCH__
    // as recip: r + r (e/2 + 3 e^2/8), e = 1 - x r^2
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x * r, r, 1.0);
    return fma(r * e, fma(0.375, e, 0.5), r);
#else
    return 1.0 / sqrt(x);
#endif
}
template <>
GKM_HD float rsqrt_t<float>(float x)
{
#ifdef __CUDA_ARCH__
    return rsqrtf(x);
#else
    return 1.0f / sqrtf(x);
#endif
}

// half: +1 positive-u half space (erfc(-sqrt(lam) u)/2), -1 negative half
template <class T>
GKM_HD void half_table(T* H, T U0, T lam, T inv2lam, int half)
{
    const T pi = T(3.14159265358979323846);
    T sl = sqrt_t<T>(lam);
    T g = T(0.5) * exp_t<T>(-lam * U0 * U0) / sqrt_t<T>(lam * pi);
    if (half > 0) {
        H[0] = T(0.5) * erfc_t<T>(-sl * U0);
        H[1] = U0 * H[0] + g;
    } else {
        H[0] = T(0.5) * erfc_t<T>(sl * U0);
        H[1] = U0 * H[0] - g;
    }
#pragma unroll
    for (int i = 2; i < 7; i++) H[i] = U0 * H[i - 1] + H[i - 2] * (T(i - 1) * inv2lam);
}

template <class T, int N>
GKM_HD void full_table(T* F, T U, T inv2lam)
{
    F[0] = T(1);
    F[1] = U;
#pragma unroll
    for (int i = 2; i < N; i++) F[i] = U * F[i - 1] + F[i - 2] * (T(i - 1) * inv2lam);
}

template <class T>
GKM_HD void build_moments(Moments<T>& M, const T U[3], T lam, int K, int half)
{
    T inv2lam = T(1) / (T(2) * lam);
    M.Ie2 = T(K) * inv2lam;
    M.Ie4 = T(3 * K + K * (K - 1)) * inv2lam * inv2lam;
    half_table<T>(M.H, U[0], lam, inv2lam, half);
    full_table<T, 7>(M.X, U[0], inv2lam);
    full_table<T, 6>(M.Y, U[1], inv2lam);
    full_table<T, 6>(M.Z, U[2], inv2lam);
}

#define GKM_TABLES(S) S.Y, S.Z
#define TM(A, B, C) (I[k + (A)] * Y[l + (B)] * Z[m + (C)])
#define GKM_YZ_PARAM const T* Y, const T* Z

// ----------------------------------------------------------- MCal -----
// <psi (u^k v^l w^m) (a0 + a1 u + a2 v + a3 w + a4 psi4)> with psi = (1,u,v,w,psi4),
// psi4 = (u^2+v^2+w^2+xi^2)/2; I = normal table (full or half), Y, Z tangential.
template <int k, int l, int m, class T>
GKM_HD void mcal(T M[5], const T* I, GKM_YZ_PARAM, T Ie2, T Ie4, const T a[5])
{
    T t000 = TM(0, 0, 0), t100 = TM(1, 0, 0), t010 = TM(0, 1, 0), t001 = TM(0, 0, 1);
    T t200 = TM(2, 0, 0), t020 = TM(0, 2, 0), t002 = TM(0, 0, 2);
    T t110 = TM(1, 1, 0), t101 = TM(1, 0, 1), t011 = TM(0, 1, 1);
    T v0 = T(0.5) * (t200 + t020 + t002 + t000 * Ie2);
    T v1 = T(0.5) * (TM(3, 0, 0) + TM(1, 2, 0) + TM(1, 0, 2) + t100 * Ie2);
    T v2 = T(0.5) * (TM(2, 1, 0) + TM(0, 3, 0) + TM(0, 1, 2) + t010 * Ie2);
    T v3 = T(0.5) * (TM(2, 0, 1) + TM(0, 2, 1) + TM(0, 0, 3) + t001 * Ie2);
    M[0] = a[0] * t000 + a[1] * t100 + a[2] * t010 + a[3] * t001 + a[4] * v0;
    M[1] = a[0] * t100 + a[1] * t200 + a[2] * t110 + a[3] * t101 + a[4] * v1;
    M[2] = a[0] * t010 + a[1] * t110 + a[2] * t020 + a[3] * t011 + a[4] * v2;
    M[3] = a[0] * t001 + a[1] * t101 + a[2] * t011 + a[3] * t002 + a[4] * v3;
    M[4] = T(0.25) * a[4] *
               (TM(4, 0, 0) + TM(0, 4, 0) + TM(0, 0, 4) + t000 * Ie4 +
                T(2) * (TM(2, 2, 0) + TM(2, 0, 2) + t200 * Ie2 + TM(0, 2, 2) + t020 * Ie2 + t002 * Ie2)) +
           a[0] * v0 + a[1] * v1 + a[2] * v2 + a[3] * v3;
}

template <int k, int l, int m, class T>
GKM_HD void mcal0(T M[5], const T* I, GKM_YZ_PARAM, T Ie2)
{
    M[0] = TM(0, 0, 0);
    M[1] = TM(1, 0, 0);
    M[2] = TM(0, 1, 0);
    M[3] = TM(0, 0, 1);
    M[4] = T(0.5) * (TM(2, 0, 0) + TM(0, 2, 0) + TM(0, 0, 2) + TM(0, 0, 0) * Ie2);
}

template <class T>
GKM_HD void axpy5(T* acc, T s, const T* M)
{
#pragma unroll
    for (int q = 0; q < 5; q++) acc[q] += s * M[q];
}

// ----------------------------------------------------- slope solver ---
// Solve the 5x5 moment system for the Maxwellian slope coefficients, with the
// Prandtl-number correction on the energy component (src/GKMflux.cpp:283-297).
template <class T>
struct SlopeState {
    T U[3];
    T lam2;     // 2 lam
    T usqc;     // u.u + (K+3)/(2 lam)
    T a4fac;    // (1/Pr) (4 lam^2) / (K+3)
};

template <class T>
GKM_HD SlopeState<T> slope_state(const T U[3], T lam, int K)
{
    SlopeState<T> s;
    s.U[0] = U[0];
    s.U[1] = U[1];
    s.U[2] = U[2];
    s.lam2 = T(2) * lam;
    s.usqc = U[0] * U[0] + U[1] * U[1] + U[2] * U[2] + T(K + 3) / s.lam2;
    s.a4fac = T(1.0 / kPrandtl) * (T(4) * lam * lam) / T(K + 3);
    return s;
}

template <class T>
GKM_HD void slope_solve(const T b[5], const SlopeState<T>& s, T a[5])
{
    T r2 = b[1] - s.U[0] * b[0];
    T r3 = b[2] - s.U[1] * b[0];
    T r4 = b[3] - s.U[2] * b[0];
    T r5 = T(2) * b[4] - b[0] * s.usqc;
    a[4] = s.a4fac * (r5 - T(2) * (s.U[0] * r2 + s.U[1] * r3 + s.U[2] * r4));
    a[3] = s.lam2 * r4 - s.U[2] * a[4];
    a[2] = s.lam2 * r3 - s.U[1] * a[4];
    a[1] = s.lam2 * r2 - s.U[0] * a[4];
    a[0] = b[0] - a[1] * s.U[0] - a[2] * s.U[1] - a[3] * s.U[2] - T(0.5) * a[4] * s.usqc;
}

template <class T>
GKM_HD void c2p(const T W[5], T gm1, T& den, T U[3], T& P)
{
    den = W[0];
    T ir = T(1) / den;
    U[0] = W[1] * ir;
    U[1] = W[2] * ir;
    U[2] = W[3] * ir;
    P = (den * gm1) * (W[4] * ir - T(0.5) * (U[0] * U[0] + U[1] * U[1] + U[2] * U[2]));
}

// ------------------------------------------------- time coefficients ----
// Integrals over [0, dt] of the BGK relaxation, src/GKMflux.cpp:162-167,197-204.
// With e = exp(-dt/tau) the coefficients are differences of nearly equal terms
// when dt/tau is small, so they are always formed in double precision
// (wide_t), whatever type the flux itself runs in.
template <class T>
struct Wide {
    using type = double;
};
template <class T>
using wide_t = typename Wide<T>::type;

template <class D>
struct TimeCoefs {
    D gm1, gm2, gm3, gm4, gm5, p0, p1, p2, p3, p4, p5;
};

// BGK time integrals over [0, dt] with e = exp(-dt/tau) (src/GKMflux.cpp:162-167,197-204).
template <class D>
GKM_HD TimeCoefs<D> time_coefs(D tau, D dt)
{
    TimeCoefs<D> c;
    D ex = exp_t<D>(-dt / tau);
    D omx = D(1) - ex;
    D gm0 = dt - tau * omx;
    D igm0 = D(1) / gm0;
    c.gm1 = -omx * igm0;
    c.gm2 = (-dt + D(2) * tau * omx - dt * ex) * igm0;
    c.gm3 = -c.gm1;
    c.gm4 = (dt * ex - tau * omx) * igm0;
    c.gm5 = tau * c.gm3;
    D Pc = tau * omx;                               // -tau (e - 1)
    D Qc = -tau * dt * ex + tau * tau * omx;        // -tau dt e - tau^2 (e - 1)
    c.p0 = dt - Pc;
    c.p1 = D(0.5) * dt * dt - tau * c.p0;
    c.p2 = -tau * c.p0 + Qc;
    c.p3 = Pc;
    c.p4 = -Qc - tau * Pc;
    c.p5 = -tau * Pc;
    return c;
}

// --------------------------------------------------------- the flux ----
// The face inputs come from a provider so that the 30 slope values are formed
// where they are consumed instead of being held in registers.  A provider has
//   T WL(int q), WR(int q)   cell averages left/right of the face
//   T Wl(int q), Wr(int q)   reconstructed face states
//   T DW(int v, int q)       slope vectors v = 0..5: DWxl, DWxr, DWyl, DWyr, DWzl, DWzr
// all in the face frame (slot 1 = normal momentum).  tau0 = mu(T_L)/p_L of the
// left cell.  Output F[5] = flux integrated over [0, dt] (not divided by dt).
template <class T>
struct FaceInput {
    T WL_[5], WR_[5], Wl_[5], Wr_[5];
    T DW_[6][5];
    GKM_HD T WL(int q) const { return WL_[q]; }
    GKM_HD T WR(int q) const { return WR_[q]; }
    GKM_HD T Wl(int q) const { return Wl_[q]; }
    GKM_HD T Wr(int q) const { return Wr_[q]; }
    GKM_HD T DW(int v, int q) const { return DW_[v][q]; }
};

// The flux with the reference's moment algebra: one MCal (25 triple products
// and their sums) per table, weight and slope vector.  The operation counter
// instantiates this form; the kernels run gks_flux_peculiar below.
template <class T, class Prov>
GKM_HD void gks_flux_mcal(const Prov& in, T tau0, T dt, T dx, const Phys<T>& ph, T F[5])
{
    const int K = ph.K;
    T denl, Ul[3], Pl, denr, Ur[3], Pr;
    {
        T wl[5], wr[5];
#pragma unroll
        for (int q = 0; q < 5; q++) {
            wl[q] = in.Wl(q);
            wr[q] = in.Wr(q);
        }
        c2p<T>(wl, ph.gm1, denl, Ul, Pl);
        c2p<T>(wr, ph.gm1, denr, Ur, Pr);
    }
    T laml = T(0.5) * denl / Pl;
    T lamr = T(0.5) * denr / Pr;

    // collision time with the pressure-jump correction, src/GKMflux.cpp:156-157
    T ql = denl / laml, qr = denr / lamr;
    const TimeCoefs<wide_t<T>> tc = time_coefs<wide_t<T>>(
        wide_t<T>(tau0) + wide_t<T>(dt) * wide_t<T>(fabs(ql - qr) / fabs(ql + qr)), wide_t<T>(dt));
    const T gm1 = T(tc.gm1), gm2 = T(tc.gm2), gm3 = T(tc.gm3), gm4 = T(tc.gm4), gm5 = T(tc.gm5);
    const T p0 = T(tc.p0), p1 = T(tc.p1), p2 = T(tc.p2), p3 = T(tc.p3), p4 = T(tc.p4), p5 = T(tc.p5);

    T We[5] = {0, 0, 0, 0, 0};      // equilibrium state at the face, src/GKMflux.cpp:73-77
    T by_[5] = {0, 0, 0, 0, 0}, bz_[5] = {0, 0, 0, 0, 0};
    T Bacc[5] = {0, 0, 0, 0, 0};   // B_ * dene, without the gm1/gm3 terms
    T Facc[5] = {0, 0, 0, 0, 0};
    T M[5];

    const T cB = gm4 + gm5;
    // ---------------- one side (l: positive half with left state, r: negative half with right state)
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const T den = side == 0 ? denl : denr;
        const T* Us = side == 0 ? Ul : Ur;
        const T lam = side == 0 ? laml : lamr;
        Moments<T> S;
        build_moments<T>(S, Us, lam, K, side == 0 ? +1 : -1);
        SlopeState<T> ss = slope_state<T>(Us, lam, K);
        T iden = T(1) / den;
        mcal0<0, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2);
        axpy5<T>(We, den, M);
        T Bs[5] = {0, 0, 0, 0, 0};   // -(Mf100 ax + Mf010 ay + Mf001 az)
        T b[5], a[5];
        // normal slope
#pragma unroll
        for (int q = 0; q < 5; q++) b[q] = in.DW(0 + side, q) * iden;
        slope_solve<T>(b, ss, a);
        mcal<1, 0, 0, T>(M, S.X, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bs, T(-1), M);
        mcal<1, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bacc, cB * den, M);
        mcal<2, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Facc, p4 * den, M);
        // first tangential slope
#pragma unroll
        for (int q = 0; q < 5; q++) b[q] = in.DW(2 + side, q) * iden;
        slope_solve<T>(b, ss, a);
        mcal<0, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(by_, T(1), M);
        mcal<0, 1, 0, T>(M, S.X, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bs, T(-1), M);
        mcal<0, 1, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bacc, cB * den, M);
        mcal<1, 1, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Facc, p4 * den, M);
        // second tangential slope
#pragma unroll
        for (int q = 0; q < 5; q++) b[q] = in.DW(4 + side, q) * iden;
        slope_solve<T>(b, ss, a);
        mcal<0, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(bz_, T(1), M);
        mcal<0, 0, 1, T>(M, S.X, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bs, T(-1), M);
        mcal<0, 0, 1, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bacc, cB * den, M);
        mcal<1, 0, 1, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Facc, p4 * den, M);
        // time slope of this side, src/GKMflux.cpp:145-151
        slope_solve<T>(Bs, ss, a);
        mcal<0, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Bacc, gm5 * den, M);
        mcal<1, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2, S.Ie4, a);
        axpy5<T>(Facc, p5 * den, M);
        // free transport of the initial half-Maxwellian
        mcal0<1, 0, 0, T>(M, S.H, GKM_TABLES(S), S.Ie2);
        axpy5<T>(Facc, p3 * den, M);
    }

    // ---------------- equilibrium part
    T dene, Ue[3], Pe;
    c2p<T>(We, ph.gm1, dene, Ue, Pe);
    T lame = T(0.5) * dene / Pe;
    Moments<T> E;
    build_moments<T>(E, Ue, lame, K, +1);
    T H2[7];
    {
        T inv2lam = T(1) / (T(2) * lame);
        half_table<T>(H2, Ue[0], lame, inv2lam, -1);
    }
    SlopeState<T> se = slope_state<T>(Ue, lame, K);
    T b[5], a[5];
    const T idx2 = T(2) / (dene * dx);
    // normal equilibrium slopes from the cell averages, src/GKMflux.cpp:115-116
#pragma unroll
    for (int q = 0; q < 5; q++) b[q] = (We[q] - in.WL(q)) * idx2;
    slope_solve<T>(b, se, a);
    mcal<1, 0, 0, T>(M, E.H, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Bacc, gm2 * dene, M);
    mcal<2, 0, 0, T>(M, E.H, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Facc, p2 * dene, M);
#pragma unroll
    for (int q = 0; q < 5; q++) b[q] = (in.WR(q) - We[q]) * idx2;
    slope_solve<T>(b, se, a);
    mcal<1, 0, 0, T>(M, H2, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Bacc, gm2 * dene, M);
    mcal<2, 0, 0, T>(M, H2, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Facc, p2 * dene, M);
    // tangential equilibrium slopes
    slope_solve<T>(by_, se, a);
    mcal<0, 1, 0, T>(M, E.X, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Bacc, gm2 * dene, M);
    mcal<1, 1, 0, T>(M, E.X, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Facc, p2 * dene, M);
    slope_solve<T>(bz_, se, a);
    mcal<0, 0, 1, T>(M, E.X, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Bacc, gm2 * dene, M);
    mcal<1, 0, 1, T>(M, E.X, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Facc, p2 * dene, M);
    // time derivative of the equilibrium, src/GKMflux.cpp:183-191
    mcal0<0, 0, 0, T>(M, E.X, GKM_TABLES(E), E.Ie2);
    T idene = T(1) / dene;
#pragma unroll
    for (int q = 0; q < 5; q++) b[q] = (gm1 * dene * M[q] + Bacc[q] + gm3 * We[q]) * idene;
    slope_solve<T>(b, se, a);
    mcal<1, 0, 0, T>(M, E.X, GKM_TABLES(E), E.Ie2, E.Ie4, a);
    axpy5<T>(Facc, p1 * dene, M);
    mcal0<1, 0, 0, T>(M, E.X, GKM_TABLES(E), E.Ie2);
    axpy5<T>(Facc, p0 * dene, M);
#pragma unroll
    for (int q = 0; q < 5; q++) F[q] = Facc[q];
}

// ---------------------------------------------- the peculiar-frame flux ----
// The moments of a Maxwellian are Gaussian in the peculiar velocity
// (c, v', w') = (u, v, w) - U: over the full space the odd ones vanish and the even ones are
// products of s = 1/(2 lam); over a half space only the normal direction keeps a table,
// J_k = <c^k>_{u>0}.  Written in psi'' = (1, c, v', w', (c^2 + v'^2 + w'^2 + xi^2)/2),
//   * the slope solve is diagonal (SlopeP, solve_lab / solve_pec);
//   * the full-space moments of G = u (psi.a_n) + v (psi.a_y) + w (psi.a_z) are closed forms
//     of a few products: with A = U a_n + V a_y + W a_z and D = c P_n + v' P_y + w' P_z,
//     G = psi''.A + D;
//   * the half-space moments of G and of psi.a are sums of four or three J_k per component,
//     because the tangential average of zeta = v'^2 + w'^2 + xi^2 against a polynomial differs
//     from <zeta> times its average by one product with s (half_poly, half_P).
// Every moment, slope and time coefficient is the reference's (src/GKMflux.cpp:11-229); the
// frames, and so the order of the sums, are not.  Each side's moments go from its own frame to
// the equilibrium state's by psi_e = T(U - U_e) psi'' (add_in_frame), where the equilibrium's slopes
// are solved, and the summed flux to the laboratory frame at the end.  The reference's
// gamma_1 (moments of the equilibrium) + gamma_3 (its conserved state), gamma_3 = -gamma_1, has
// an energy component only, gamma_1 p dK2 / 2 (Phys).  About 900 operations per face beside the divisions and
// the special functions, where the moments in the laboratory frame took about 2,000; the sweeps
// are bound by the FP64 (mixed: FP32) arithmetic: the FP64 pipe takes a warp instruction every 2.2
// cycles from independent streams and every 2.5 to 3 from chains of one or two, however many warps
// there are, so the count of operations decides.  Measured at 256^3 with the default shapes: a step
// 18.00 -> 13.97 ms in FP64, 10.62 -> 8.26 ms in the mixed form; with the polynomials of a side combined
// before one contraction per weight, single reciprocals and the shorter WENO sums the x/y/z sweeps went
// from 2.67/2.74/3.14 to 2.57/2.63/3.02 ms (64- and 48-face segments).  Errors against extended precision
// are smaller in every component than with the laboratory-frame moments.

// Primitive values of a state: 1/rho, p, s = 1 / (2 lam) = p / rho and 1 / s.
template <class T>
struct Prim {
    T den, ir, U[3], P, s, is;
};

// 1/rho and 1/p each by a reciprocal of its own (grouping them under one costs more products than the
// short reciprocal has steps)
template <class T>
GKM_HD Prim<T> prim(const T W[5], T gm1)
{
    Prim<T> p;
    p.den = W[0];
    p.ir = recip<T>(W[0]);
    p.U[0] = W[1] * p.ir;
    p.U[1] = W[2] * p.ir;
    p.U[2] = W[3] * p.ir;
    p.P = gm1 * (W[4] - T(0.5) * (W[1] * p.U[0] + W[2] * p.U[1] + W[3] * p.U[2]));
    p.s = p.P * p.ir;
    p.is = p.den * recip<T>(p.P);
    return p;
}

// Horner's rule, c[0] + c[1] t + ..
template <class T, int N>
GKM_HD T horner(const double (&c)[N], T t)
{
    T r = T(c[N - 1]);
#pragma unroll
    for (int k = N - 2; k >= 0; k--) r = r * t + T(c[k]);
    return r;
}

// exp(-x^2/2) and erf(x/sqrt(2))/2 for x^2 <= 2 as polynomials in t = x^2: the interpolants of
// exp(-t/2) and erf(sqrt(t/2)) / (2 sqrt(t)) at the Chebyshev points of [0, 2] (degrees 12 and 11: the
// interpolants within 8e-18 of the functions, relative, with their coefficients rounded to double within
// 9.8e-17 and 1.3e-16; erf of degree 6 in single precision: 1.4e-9).  As evaluated, largest relative errors
// measured: 4.0 and 2.9 units of 2^-53, single precision 2.6 and 2.2 of 2^-24.
template <class T>
GKM_HD void gauss_small(T x, T t, T& ex, T& herf)
{
    if constexpr (single_t<T>::value) {
        const double q[7] = {0.39894227996049447, -0.066490358435689789, 0.0099733829240630997, -0.001186799713508448,
                            0.00011466371578999978, -8.8574673457925686e-06, 4.3508473942210419e-07};
        ex = exp_t<T>(T(-0.5) * t);
        herf = x * horner<T>(q, t);
    } else {
        const double p[13] = {1, -0.4999999999999995, 0.12499999999998568, -0.020833333333175521,
                            0.0026041666657620841, -0.00026041666357754114, 2.1701382107946786e-05, -1.5500892124483604e-06,
                            9.6871088514534077e-08, -5.3752300794789401e-09, 2.657581414044206e-10, -1.1184386854931272e-11,
                            3.1052342897486384e-13};
        const double q[12] = {0.3989422804014327, -0.066490380066905067, 0.0099735570100268726, -0.0011873282153967736,
                            0.00011543468721120926, -9.444655101548686e-06, 6.659672481574838e-07, -4.1224151072896811e-08,
                            2.271501082181806e-09, -1.1192508602593551e-10, 4.7370852926482607e-12, -1.3458332338909829e-13};
        ex = horner<T>(p, t);
        herf = x * horner<T>(q, t);
    }
}

// <1> and <c> over the half space u > 0 (half > 0) or u < 0: J_0 = erfc(-+ x/sqrt(2))/2 and
// J_1 = +- sqrt(s / (2 pi)) exp(-x^2/2), x = U / sqrt(s), with sqrt(s) from one reciprocal square
// root.  Normal velocities up to sqrt(2 s) (Mach 1.2) take the polynomials: erfc and exp of the
// library cost 105 and 28 FP64 issue slots each, the two polynomials 24 together (256^3 step,
// default shapes: FP64 13.00 -> 12.06 ms, mixed 8.05 -> 7.91 ms).
template <class T>
GKM_HD void half_space(const Prim<T>& p, int half, T& J0, T& g)
{
    const T rs = rsqrt_t<T>(p.is);   // sqrt(s)
    const T x = p.U[0] * (p.is * rs), t = x * x;
    T ex;
    if (t <= T(2)) {
        T herf;
        gauss_small<T>(x, t, ex, herf);
        J0 = half > 0 ? T(0.5) + herf : T(0.5) - herf;
    } else {
        const T y = x * T(0.70710678118654752440);
        ex = exp_t<T>(-y * y);
        J0 = T(0.5) * erfc_t<T>(half > 0 ? -y : y);
    }
    const T e = (T(0.39894228040143267794) * rs) * ex;
    g = half > 0 ? e : -e;
}

// J_k = <c^k> over that half space: J_k = (k - 1) s J_{k-2} + (-U)^{k-1} g
template <class T, int N>
GKM_HD void half_moments(T* J, T J0, T g, T U, T s)
{
    J[0] = J0;
    J[1] = g;
    T q = g;
#pragma unroll
    for (int k = 2; k < N; k++) {
        q = -U * q;
        J[k] = (T(k - 1) * s) * J[k - 2] + q;
    }
}

// Below, psi'' is taken with its last component doubled, c^2 + v'^2 + w'^2 + xi^2, which spares the
// halves; its moments are halved once, in the flux.

// one slope vector in the peculiar frame of its state:
// psi.a = a0 + a1 c + a2 v' + a3 w' + h (c^2 + v'^2 + w'^2 + xi^2)
template <class T>
struct SlopeP {
    T a0, a1, a2, a3, h;
};

// what the solves of one state share: uq = (|U|^2 + (K+3) s)/2, z3 = (K+3) s, hf = 1/(Pr (K+3) s^2)
template <class T>
struct SolveP {
    T uq, z3, hf;
};
template <class T>
GKM_HD SolveP<T> solve_consts(const Prim<T>& p, const Phys<T>& ph)
{
    SolveP<T> c;
    c.z3 = ph.k3 * p.s;
    c.uq = T(0.5) * (p.U[0] * p.U[0] + p.U[1] * p.U[1] + p.U[2] * p.U[2] + c.z3);
    c.hf = ph.iPrK3 * (p.is * p.is);
    return c;
}

// the slope solver (src/GKMflux.cpp:283-297) of sc * b, b the moments in the laboratory frame
template <class T>
GKM_HD SlopeP<T> solve_lab(T b0, T b1, T b2, T b3, T b4, T sc, const Prim<T>& p, const SolveP<T>& c)
{
    const T r1 = b1 - p.U[0] * b0, r2 = b2 - p.U[1] * b0, r3 = b3 - p.U[2] * b0;
    const T e = b4 - p.U[0] * r1 - p.U[1] * r2 - p.U[2] * r3 - c.uq * b0;
    const T l = sc * p.is;
    SlopeP<T> a;
    a.h = (sc * c.hf) * e;
    a.a1 = l * r1;
    a.a2 = l * r2;
    a.a3 = l * r3;
    a.a0 = sc * b0 - a.h * c.z3;
    return a;
}
// the same of moments already in the state's peculiar frame
template <class T>
GKM_HD SlopeP<T> solve_pec(const T b[5], const Prim<T>& p, const SolveP<T>& c)
{
    SlopeP<T> a;
    a.h = (T(0.5) * c.hf) * (b[4] - c.z3 * b[0]);
    a.a1 = p.is * b[1];
    a.a2 = p.is * b[2];
    a.a3 = p.is * b[3];
    a.a0 = b[0] - a.h * c.z3;
    return a;
}

// acc += w o with o taken from a frame moving with U to the frame moving with U - d:
// psi -> T(d) psi, d2 = 2 d, dd = |d|^2
template <class T>
GKM_HD void add_in_frame(T acc[5], T w, const T o[5], const T d[3], const T d2[3], T dd)
{
    acc[0] += w * o[0];
    acc[1] += w * (o[1] + d[0] * o[0]);
    acc[2] += w * (o[2] + d[1] * o[0]);
    acc[3] += w * (o[3] + d[2] * o[0]);
    acc[4] += w * (o[4] + d2[0] * o[1] + d2[1] * o[2] + d2[2] * o[3] + dd * o[0]);
}
template <class T>
GKM_HD void add_in_frame(T acc[5], const T o[5], const T d[3], const T d2[3], T dd)
{
    acc[0] += o[0];
    acc[1] = (acc[1] + o[1]) + d[0] * o[0];
    acc[2] = (acc[2] + o[2]) + d[1] * o[0];
    acc[3] = (acc[3] + o[3]) + d[2] * o[0];
    acc[4] = (acc[4] + o[4]) + (d2[0] * o[1] + d2[1] * o[2] + d2[2] * o[3] + dd * o[0]);
}

// <psi'' (psi.a)> with the normal weight N_k (N = J: weight 1; N = L: weight u); z1 = (K+2) s = <zeta>
template <class T>
GKM_HD void half_P(T o[5], const T* N, const SlopeP<T>& a, T s, T z1)
{
    const T hz = a.h * z1;
    const T t = a.a0 + hz;
    const T s0 = t * N[0] + a.a1 * N[1] + a.h * N[2];
    const T s1 = t * N[1] + a.a1 * N[2] + a.h * N[3];
    const T s2 = t * N[2] + a.a1 * N[3] + a.h * N[4];
    const T sn = s * N[0];
    o[0] = s0;
    o[1] = s1;
    o[2] = sn * a.a2;
    o[3] = sn * a.a3;
    o[4] = z1 * s0 + (s2 + (sn + sn) * hz);
}

// the same with weights 1 and u (o and p) over one table
template <class T>
GKM_HD void half_P2(T o[5], T p[5], const T* N, const SlopeP<T>& a, T s, T U, T z1)
{
    const T hz = a.h * z1;
    const T t = a.a0 + hz;
    const T s0 = t * N[0] + a.a1 * N[1] + a.h * N[2];
    const T s1 = t * N[1] + a.a1 * N[2] + a.h * N[3];
    const T s2 = t * N[2] + a.a1 * N[3] + a.h * N[4];
    const T s3 = t * N[3] + a.a1 * N[4] + a.h * N[5];
    const T sn = s * N[0], sm = s * N[1] + U * sn;
    o[0] = s0;
    o[1] = s1;
    o[2] = sn * a.a2;
    o[3] = sn * a.a3;
    o[4] = z1 * s0 + (s2 + (sn + sn) * hz);
    p[0] = s1 + U * s0;
    p[1] = s2 + U * s1;
    p[2] = sm * a.a2;
    p[3] = sm * a.a3;
    p[4] = z1 * p[0] + ((s3 + U * s2) + (sm + sm) * hz);
}

// the convective part of G: A = U a_n + V a_y + W a_z
template <class T>
GKM_HD SlopeP<T> convect(const T U[3], const SlopeP<T>& n, const SlopeP<T>& y, const SlopeP<T>& z)
{
    SlopeP<T> A;
    A.a0 = U[0] * n.a0 + U[1] * y.a0 + U[2] * z.a0;
    A.a1 = U[0] * n.a1 + U[1] * y.a1 + U[2] * z.a1;
    A.a2 = U[0] * n.a2 + U[1] * y.a2 + U[2] * z.a2;
    A.a3 = U[0] * n.a3 + U[1] * y.a3 + U[2] * z.a3;
    A.h = U[0] * n.h + U[1] * y.h + U[2] * z.h;
    return A;
}

// A polynomial Q = k G + l P_t (+ m) of the half-space moments, by its tangential averages:
// <Q> = c0 + c1 c + c2 c^2 + c3 c^3, <zeta Q> = z1 <Q> + 2 s (y0 + y1 c), <v' Q> = s (v0 + v1 c + v2 c^2),
// <w' Q> likewise
template <class T>
struct HalfPoly {
    T c0, c1, c2, c3, y0, y1, v0, v1, v2, w0, w1, w2;
};
// <psi'' Q> with the normal weight N_k (J: 1; L: u)
template <class T>
GKM_HD void half_poly(T o[5], const T* N, const HalfPoly<T>& Q, T s, T z1)
{
    const T s0 = Q.c0 * N[0] + Q.c1 * N[1] + Q.c2 * N[2] + Q.c3 * N[3];
    const T s1 = Q.c0 * N[1] + Q.c1 * N[2] + Q.c2 * N[3] + Q.c3 * N[4];
    const T s2 = Q.c0 * N[2] + Q.c1 * N[3] + Q.c2 * N[4] + Q.c3 * N[5];
    o[0] = s0;
    o[1] = s1;
    o[2] = s * (Q.v0 * N[0] + Q.v1 * N[1] + Q.v2 * N[2]);
    o[3] = s * (Q.w0 * N[0] + Q.w1 * N[1] + Q.w2 * N[2]);
    o[4] = z1 * s0 + (s2 + (s + s) * (Q.y0 * N[0] + Q.y1 * N[1]));
}

// a face provider may give raw differences and their common factors instead of slopes:
//   T dW(int v, int q), the difference; T scale(int v), the factor (slope = scale * dW)
template <class Prov, class = void>
struct has_raw : std::false_type {};
template <class Prov>
struct has_raw<Prov, std::void_t<decltype(std::declval<const Prov&>().scale(0))>> : std::true_type {};

template <class T, class Prov>
GKM_HD SlopeP<T> face_slope(const Prov& in, int v, const Prim<T>& p, const SolveP<T>& c)
{
    if constexpr (has_raw<Prov>::value)
        return solve_lab<T>(in.dW(v, 0), in.dW(v, 1), in.dW(v, 2), in.dW(v, 3), in.dW(v, 4), in.scale(v), p, c);
    else
        return solve_lab<T>(in.DW(v, 0), in.DW(v, 1), in.DW(v, 2), in.DW(v, 3), in.DW(v, 4), T(1), p, c);
}

// the factor of a one-sided difference over half a cell, 2 / dx
template <class T, class Prov>
GKM_HD T normal_scale(const Prov& in, T dx)
{
    if constexpr (has_raw<Prov>::value) return in.scale(0);
    else return T(2) / dx;
}

// The time integrals the peculiar form needs, from src/GKMflux.cpp:162-167,197-204 with
// gm0 = dt - tau (1 - e), e = exp(-dt/tau), multiplied out: the slope of the equilibrium is solved
// from gm0 B_, so the coefficients are
//   of the sides  gm0 (gm4 + gm5) = dt e, gm0 gm5 = P, p3 = P, p4 = tau (dt e - 2 P), p5 = -tau P,
//   of the rest   gm0 gm1 = -(1 - e), gm0 gm2 = h = 2 P - dt - dt e, p2 = tau h, p0 = gm0,
//                 p1 / gm0 = dt^2 / (2 gm0) - tau,
// with P = tau (1 - e).  They are formed in double precision whatever the flux runs in, as
// differences of nearly equal terms where dt / tau is small.  EXPM1: 1 - e as -expm1(-dt/tau),
// exact there (the mixed form); otherwise the reference's 1 - e.  Fewer values stay live across the
// moments than with the reference's eleven coefficients, and the mixed form needs no FP64 exp: 256^3
// step FP64 12.06 -> 11.99 ms, mixed 7.91 -> 7.78 ms.
template <class T>
struct RelaxCoefs {
    T tau, omx, P, dte, h, p0, p1g;
};
template <class T, bool EXPM1>
GKM_HD RelaxCoefs<T> relax_coefs(wide_t<T> tau, wide_t<T> dt)
{
    using D = wide_t<T>;
    D e = D(0), omx = D(1);
    // beyond x = dt / tau = 40, e (under 2^-57) is below the rounding of every term it enters
    const D x = dt / tau;
    if (!(x > D(40))) {
        if constexpr (EXPM1) {
            omx = -expm1(-x);
            e = D(1) - omx;
        } else {
            e = exp_t<D>(-x);
            omx = D(1) - e;
        }
    }
    const D P = tau * omx, dte = dt * e, gm0 = dt - P;
    RelaxCoefs<T> c;
    c.tau = T(tau);
    c.omx = T(omx);
    c.P = T(P);
    c.dte = T(dte);
    c.h = T((P - dt) + (P - dte));
    c.p0 = T(gm0);
    c.p1g = T((D(0.5) * dt) * (dt * recip<D>(gm0)) - tau);
    return c;
}

// The flux of gks_flux_mcal with every moment taken in the peculiar frames.  The slopes of a side
// are kept times its density (and the equilibrium's times its own), which is the factor their
// moments enter the flux with.
template <class T, class Prov>
GKM_HD void gks_flux_peculiar(const Prov& in, T tau0, T dt, T dx, const Phys<T>& ph, T F[5])
{
    Prim<T> st[2];
    {
        T wl[5], wr[5];
#pragma unroll
        for (int q = 0; q < 5; q++) {
            wl[q] = in.Wl(q);
            wr[q] = in.Wr(q);
        }
        st[0] = prim<T>(wl, ph.gm1);
        st[1] = prim<T>(wr, ph.gm1);
    }
    // collision time with the pressure-jump correction, src/GKMflux.cpp:156-157:
    // |rho_l/lam_l - rho_r/lam_r| / |rho_l/lam_l + rho_r/lam_r| with rho/lam = 2 p (p > 0)
    const RelaxCoefs<T> rc = relax_coefs<T, (sizeof(T) < sizeof(wide_t<T>))>(
        wide_t<T>(tau0) + wide_t<T>(dt) * wide_t<T>(fabs(st[0].P - st[1].P) * recip<T>(st[0].P + st[1].P)), wide_t<T>(dt));

    // the equilibrium state at the face (src/GKMflux.cpp:73-77), from both half-Maxwellians
    T We[5], J0[2], g[2];
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const Prim<T>& p = st[j];
        half_space<T>(p, j == 0 ? +1 : -1, J0[j], g[j]);
        const T m = p.den * J0[j], mu = p.den * (p.U[0] * J0[j] + g[j]);   // rho <1>, rho <u>
        const T o2 = m * p.U[1], o3 = m * p.U[2];
        const T o4 = T(0.5) * (mu * p.U[0] + o2 * p.U[1] + o3 * p.U[2] + ph.k3 * (p.P * J0[j]));
        if (j == 0) {
            We[0] = m; We[1] = mu; We[2] = o2; We[3] = o3; We[4] = o4;
        } else {
            We[0] += m; We[1] += mu; We[2] += o2; We[3] += o3; We[4] += o4;
        }
    }
    const Prim<T> e = prim<T>(We, ph.gm1);

    // sums over the sides, in the equilibrium's frame: the tangential slopes of the equilibrium
    // (times its density), gm0 rho_e B_ and the flux
    T by[5] = {0, 0, 0, 0, 0}, bz[5] = {0, 0, 0, 0, 0}, B[5] = {0, 0, 0, 0, 0}, Fe[5] = {0, 0, 0, 0, 0};
    // ---------------- one side (l: positive half with left state, r: negative half with right state)
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const Prim<T> p = side == 0 ? st[0] : st[1];
        const T s = p.s, U = p.U[0];
        const T z1 = ph.k2 * s, k4 = ph.k4 * s;
        const SolveP<T> sv = solve_consts<T>(p, ph);
        const T d[3] = {U - e.U[0], p.U[1] - e.U[1], p.U[2] - e.U[2]};
        const T d2[3] = {d[0] + d[0], d[1] + d[1], d[2] + d[2]};
        const T dd = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
        T J[7];
        half_moments<T, 7>(J, side == 0 ? J0[0] : J0[1], side == 0 ? g[0] : g[1], U, s);
        const T wy = e.den * p.ir;
        T o[5], q[5];
        const SlopeP<T> ay = face_slope<T>(in, 2 + side, p, sv);
        half_P<T>(o, J, ay, s, z1);
        add_in_frame<T>(by, wy, o, d, d2, dd);
        const SlopeP<T> az = face_slope<T>(in, 4 + side, p, sv);
        half_P<T>(o, J, az, s, z1);
        add_in_frame<T>(bz, wy, o, d, d2, dd);
        const SlopeP<T> an = face_slope<T>(in, side, p, sv);
        const SlopeP<T> A = convect<T>(p.U, an, ay, az);
        // <psi G>, averaged over the tangential velocities
        HalfPoly<T> G;
        G.y0 = A.h * z1 + s * (ay.a2 + az.a3);
        G.y1 = an.h * z1;
        G.c0 = A.a0 + G.y0;
        G.c1 = (A.a1 + an.a0) + G.y1;
        G.c2 = A.h + an.a1;
        G.c3 = an.h;
        G.v0 = (A.a2 + ay.a0) + ay.h * k4;
        G.v1 = an.a2 + ay.a1;
        G.v2 = ay.h;
        G.w0 = (A.a3 + az.a0) + az.h * k4;
        G.w1 = an.a3 + az.a1;
        G.w2 = az.h;
        // this side's time slope (src/GKMflux.cpp:145-151) with its sign changed: the slopes of
        // <psi G> over the full space; averaged likewise (its v' and w' parts are t2, t3 alone)
        const T S = an.a1 + ay.a2 + az.a3, k5 = ph.k5 * s;
        const T th = T(1.0 / kPrandtl) * A.h + ph.iPrK3 * S, ty = th * z1;
        const T t1 = (A.a1 + an.a0) + an.h * k5;
        const T t2 = (A.a2 + ay.a0) + ay.h * k5;
        const T t3 = (A.a3 + az.a0) + az.h * k5;
        const T t0 = ((A.a0 + s * S) + (A.h - th) * sv.z3) + ty;
        // gm0 B_ takes dt e G - P P_t, the flux p4 u G + p5 u P_t (the time slope's sign is in both) and
        // the free transport of the initial half-Maxwellian, P rho u
        const T dte = rc.dte, P = rc.P, p5 = rc.tau * P, p4 = rc.tau * dte - (p5 + p5);
        HalfPoly<T> Q;
        Q.c0 = dte * G.c0 - P * t0;
        Q.c1 = dte * G.c1 - P * t1;
        Q.c2 = dte * G.c2 - P * th;
        Q.c3 = dte * G.c3;
        Q.y0 = dte * G.y0 - P * ty;
        Q.y1 = dte * G.y1;
        Q.v0 = dte * G.v0 - P * t2;
        Q.v1 = dte * G.v1;
        Q.v2 = dte * G.v2;
        Q.w0 = dte * G.w0 - P * t3;
        Q.w1 = dte * G.w1;
        Q.w2 = dte * G.w2;
        half_poly<T>(o, J, Q, s, z1);
        Q.c0 = p4 * G.c0 + p5 * t0 + P * p.den;
        Q.c1 = p4 * G.c1 + p5 * t1;
        Q.c2 = p4 * G.c2 + p5 * th;
        Q.c3 = p4 * G.c3;
        Q.y0 = p4 * G.y0 + p5 * ty;
        Q.y1 = p4 * G.y1;
        Q.v0 = p4 * G.v0 + p5 * t2;
        Q.v1 = p4 * G.v1;
        Q.v2 = p4 * G.v2;
        Q.w0 = p4 * G.w0 + p5 * t3;
        Q.w1 = p4 * G.w1;
        Q.w2 = p4 * G.w2;
        T L[6];
#pragma unroll
        for (int k = 0; k < 6; k++) L[k] = J[k + 1] + U * J[k];   // <u c^k>
        half_poly<T>(q, L, Q, s, z1);
        add_in_frame<T>(B, o, d, d2, dd);
        add_in_frame<T>(Fe, q, d, d2, dd);
    }

    // ---------------- equilibrium part, in its own frame
    const T s = e.s, U = e.U[0];
    const T z1 = ph.k2 * s, k5 = ph.k5 * s, k7 = ph.k7 * s;
    const SolveP<T> sv = solve_consts<T>(e, ph);
    const T h = rc.h, p2 = rc.tau * h;
    // normal slopes from the cell averages (src/GKMflux.cpp:115-116), left minus right and right:
    // <P_l>_{u>0} + <P_r>_{u<0} = <P_l - P_r>_{u>0} + <P_r>
    const T idx2 = normal_scale<T>(in, dx);
    T br[5], bd[5];
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const T WL = in.WL(i), WR = in.WR(i);
        br[i] = WR - We[i];
        bd[i] = (We[i] - WL) - br[i];
    }
    {
        T J0e, ge, J[7], L[6], o[5], q[5];
        half_space<T>(e, +1, J0e, ge);
        half_moments<T, 7>(J, J0e, ge, U, s);
#pragma unroll
        for (int k = 0; k < 6; k++) L[k] = J[k + 1] + U * J[k];   // <u c^k>
        const SlopeP<T> ad = solve_lab<T>(bd[0], bd[1], bd[2], bd[3], bd[4], idx2, e, sv);
        half_P2<T>(o, q, L, ad, s, U, z1);
        axpy5<T>(B, h, o);
        axpy5<T>(Fe, p2, q);
    }
    {
        // G with the right normal slope and the tangential slopes, over the full space
        const SlopeP<T> an = solve_lab<T>(br[0], br[1], br[2], br[3], br[4], idx2, e, sv);
        const SlopeP<T> ay = solve_pec<T>(by, e, sv), az = solve_pec<T>(bz, e, sv);
        const SlopeP<T> A = convect<T>(e.U, an, ay, az);
        const T S = an.a1 + ay.a2 + az.a3, sS = s * S, w = A.a0 + A.h * k5;
        const T x0 = (A.a0 + sS) + A.h * sv.z3;
        const T x1 = s * ((A.a1 + an.a0) + an.h * k5);
        const T x2 = s * ((A.a2 + ay.a0) + ay.h * k5);
        const T x3 = s * ((A.a3 + az.a0) + az.h * k5);
        const T x4 = sv.z3 * w + k5 * sS;
        const T ss = s * s;
        const T c1 = s * ((w + sS) + (s + s) * an.a1);
        const T c4 = k5 * (s * ((A.a1 + an.a0) + an.h * k7));
        B[0] += h * x0;
        B[1] += h * x1;
        B[2] += h * x2;
        B[3] += h * x3;
        B[4] += h * x4 - (rc.omx * ph.dK2) * e.P;
        Fe[0] += p2 * (x1 + U * x0);
        Fe[1] += p2 * (c1 + U * x1);
        Fe[2] += p2 * (ss * (an.a2 + ay.a1) + U * x2);
        Fe[3] += p2 * (ss * (an.a3 + az.a1) + U * x3);
        Fe[4] += p2 * (c4 + U * x4);
    }
    {
        // the equilibrium's time slope (src/GKMflux.cpp:183-191): <psi'' (psi.a)> of the slopes of B is B
        // itself but for the Prandtl-corrected energy component
        const SlopeP<T> a = solve_pec<T>(B, e, sv);
        const T w = a.a0 + a.h * k5, p1 = rc.p1g;
        Fe[0] += p1 * (B[1] + U * B[0]);
        Fe[1] += p1 * (s * w + U * B[1]);
        Fe[2] += p1 * (U * B[2]);
        Fe[3] += p1 * (U * B[3]);
        Fe[4] += p1 * (k5 * B[1] + U * (sv.z3 * w));
        const T r = rc.p0 * e.P;
        Fe[0] += rc.p0 * We[1];
        Fe[1] += r;
        Fe[4] += (ph.k3 * U) * r;
    }
    // to the laboratory frame
    F[0] = Fe[0];
    F[1] = Fe[1] + U * Fe[0];
    F[2] = Fe[2] + e.U[1] * Fe[0];
    F[3] = Fe[3] + e.U[2] * Fe[0];
    F[4] = T(0.5) * Fe[4] + U * Fe[1] + e.U[1] * Fe[2] + e.U[2] * Fe[3] +
           (T(0.5) * (U * U + e.U[1] * e.U[1] + e.U[2] * e.U[2])) * Fe[0];
}

// The flux the kernels run; the operation counter takes the reference's MCal form.
template <class T, class Prov>
GKM_HD void gks_flux(const Prov& in, T tau0, T dt, T dx, const Phys<T>& ph, T F[5])
{
#if GKM_REFERENCE_FORM
    gks_flux_mcal<T>(in, tau0, dt, dx, ph, F);
#else
    gks_flux_peculiar<T>(in, tau0, dt, dx, ph, F);
#endif
}

}  // namespace gkm
