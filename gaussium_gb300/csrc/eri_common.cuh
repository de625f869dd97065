// Shared device/host code of the ERI engine: record layouts, the Boys function, the
// per-shell-quartet driver (primitive loops -> generated VRR -> contraction -> HRR) and
// the class kernels.  Compiled by nvcc for sm_103a; the record layouts, Boys function and
// quartet driver also compile as plain C++ (GS_HOST_ONLY) for CPU checks of the generated
// recursions.
#pragma once
#include <cmath>
#include <cstdint>

#if defined(__CUDACC__)
#define GS_HD __host__ __device__
#define GS_INLINE __forceinline__
#define GS_UNROLL _Pragma("unroll")
#else
#define GS_HD
#define GS_INLINE inline
#define GS_UNROLL
#endif

#include "boys_table.h"

namespace gs {

// ------------------------------------------------------------------ records
// One primitive pair of a shell pair (a,b), la >= lb:
//   p = alpha+beta, i2p = 1/(2p), P = (alpha A + beta B)/p, PA = P - A,
//   Kp = sqrt(2 pi^(5/2)) * c_a c_b exp(-alpha beta/p |AB|^2) / p
// so that [00|00]^(m) = Kp_bra Kp_ket (p+q)^(-1/2) F_m(T).
template <typename T> struct PrimRec;
template <> struct alignas(16) PrimRec<double> {
    double p, i2p, Px, Py, Pz, PAx, PAy, PAz, Kp, pad;
};
template <> struct alignas(16) PrimRec<float> {
    float p, i2p, Px, Py, Pz, PAx, PAy, PAz, Kp, pad0, pad1, pad2;
};

// One shell pair: AB = A - B, its primitive pairs [prim_off, prim_off + nprim), and the
// two shells (sa has the larger angular momentum).
struct alignas(16) PairRec {
    double ABx, ABy, ABz;
    int prim_off, nprim, sa, sb;
    float qmax;   // Schwarz bound sqrt(max |(ab|ab)|) of the pair (0 until computed)
    int pad;
};

// Microbench / dense-block task: canonical bra and ket pair, 3-bit permutation code
// (bit0: bra shells swapped, bit1: ket shells swapped, bit2: bra<->ket swapped) and the
// offset of the block in the caller's original (a,b,c,d) order.
struct alignas(8) WriteTask {
    int bra, ket;
    int code, pad;
    long long off;
};

template <typename T> struct VrrCoef {
    T PAx, PAy, PAz, WPx, WPy, WPz, QCx, QCy, QCz, WQx, WQy, WQz, i2p, rp2, i2q, rq2, i2pq;
};

template <int LA, int LB, int LC, int LD> struct ClassGen;

// ------------------------------------------------------------------ math helpers
// FP64 sums and products as fused multiply-adds.  On this part a DADD or a DMUL holds the FP64
// pipe 19 % longer than a DFMA (79.5 against 67 cycles a warp instruction, eight independent
// chains), so a + b is fma(a, 1, b) and a b is fma(a, b, 0), the same roundings (only the sign
// of an exact zero product is lost).  The one and the zero come from constant memory, which
// the compiler cannot fold back and the instruction takes as an operand.
#if defined(__CUDACC__)
static __constant__ double gs_one_zero[2] = {1.0, 0.0};
#endif
GS_HD GS_INLINE double gs_fma(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
    return fma(a, b, c);
#else
    return a * b + c;
#endif
}
GS_HD GS_INLINE double gs_add(double a, double b) {
#if defined(__CUDA_ARCH__)
    return fma(a, gs_one_zero[0], b);
#else
    return a + b;
#endif
}
GS_HD GS_INLINE double gs_sub(double a, double b) {
#if defined(__CUDA_ARCH__)
    return fma(-b, gs_one_zero[0], a);
#else
    return a - b;
#endif
}
GS_HD GS_INLINE double gs_mul(double a, double b) {
#if defined(__CUDA_ARCH__)
    return fma(a, b, gs_one_zero[1]);
#else
    return a * b;
#endif
}
GS_HD GS_INLINE float gs_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return fmaf(a, b, c);
#else
    return a * b + c;
#endif
}
GS_HD GS_INLINE float gs_add(float a, float b) { return a + b; }
GS_HD GS_INLINE float gs_sub(float a, float b) { return a - b; }
GS_HD GS_INLINE float gs_mul(float a, float b) { return a * b; }
GS_HD GS_INLINE double norm2(double x, double y, double z) {
    return gs_fma(z, z, gs_fma(y, y, gs_mul(x, x)));
}
GS_HD GS_INLINE float norm2(float x, float y, float z) { return x * x + y * y + z * z; }

// 1 / sqrt(x): the hardware's 20-bit approximation y and one step of Householder's method of
// second order, y (1 + r/2 + 3/8 r^2) with r = 1 - x y^2, whose error is 5/16 r^3 < 2^-58
// before rounding; five FP64 instructions.  The approximation's low word is zero (PTX ISA,
// rsqrt.approx.ftz.f64), so y^2 is exact in double and r is rounded once, at its own size: 0.52
// units in the last place at most and 0.289 rms, as the library's function (with r from
// (x y) y it was 1.0 and 0.334).  Zero, subnormal and non-finite x, and negative ones, go to the
// library's function.
GS_HD GS_INLINE double gs_rsqrt(double x) {
#if defined(__CUDA_ARCH__)
    if ((unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u) {
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
        const double r = fma(-x, gs_mul(y, y), 1.0);
        return fma(gs_mul(y, r), fma(0.375, r, 0.5), y);
    }
    return rsqrt(x);
#else
    return 1.0 / std::sqrt(x);
#endif
}
GS_HD GS_INLINE float gs_rsqrt(float x) {
#if defined(__CUDA_ARCH__)
    return rsqrtf(x);
#else
    return 1.0f / std::sqrt(x);
#endif
}

// 1 / x: the hardware's approximation y and y (1 + e + e^2) with e = 1 - x y, whose error is
// e^3 < 2^-57 before rounding; three FP64 instructions.  Zero, subnormal, non-finite and
// negative x, and those whose reciprocal is subnormal, go to the division.
GS_HD GS_INLINE double gs_rcp(double x) {
#if defined(__CUDA_ARCH__)
    if ((unsigned)__double2hiint(x) - 0x00100000u < 0x7fc00000u) {
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
        const double e = fma(-x, y, 1.0);
        return fma(y, fma(e, e, e), y);
    }
#endif
    return 1.0 / x;
}

// ------------------------------------------------------------------ Boys function
// F_m(T_k) and e^{-T_k} on the grid T_k = k / BOYS_INV_H, for the orders that a translation unit
// has no rows of (GS_BOYS_ORDER)
#if defined(__CUDACC__)
__device__ const double g_boys_d[BOYS_ROWS * BOYS_NCOL] = {GS_BOYS_TABLE_VALUES};
#endif
static const double h_boys_d[BOYS_ROWS * BOYS_NCOL] = {GS_BOYS_TABLE_VALUES};

GS_HD GS_INLINE const double* boys_table() {
#if defined(__CUDA_ARCH__)
    return g_boys_d;
#else
    return h_boys_d;
#endif
}

// Start of the asymptotic branch for orders 0..M: the smallest T (rounded up) at which
// F_m(T) ~ (2m-1)!! / (2T)^m * sqrt(pi/T) / 2 is within 2^-54 (FP64) or 2^-26 (FP32) of
// F_m for every m <= M.  Its relative error is the regularised upper incomplete gamma
// function Q(m + 1/2, T), which grows with m, so the threshold depends on M only.
constexpr unsigned kBoysAsym64[17] = {36, 40, 43, 46, 49, 52, 54, 57, 59, 61, 64, 66, 68, 70, 72, 74, 76};
constexpr unsigned kBoysAsym32[17] = {17, 20, 23, 25, 28, 30, 32, 34, 36, 38, 40, 42, 43, 45, 47, 48, 50};

// Taylor rows of the one Boys order the kernels of a translation unit evaluate most
// (GS_BOYS_ORDER, defined by the generated class and gradient units): see boys_table_gen.c.
// Other orders use the grid.
struct alignas(32) BoysRow64 {
    double c[4], e[4];      // F_{M+j}(T_k) / j! and exp(-T_k) / j!, j = 0..3
    float f[4], x[4];       // the same, j = 4..6
};
template <int M> constexpr int kBoysRows64 = (int)(kBoysAsym64[M] + 1) * BOYS_INV_H64 + 1;
#if defined(__CUDACC__) && defined(GS_BOYS_ORDER)
#define GS_BOYS_CAT2(a, b) a##b
#define GS_BOYS_CAT(a, b) GS_BOYS_CAT2(a, b)
__device__ const BoysRow64 g_boys_row64[] = {GS_BOYS_CAT(GS_BOYS_ROW64_, GS_BOYS_ORDER)};
__device__ __align__(16) const float g_boys_f32[BOYS_ROWS32 * 12] = {
    GS_BOYS_CAT(GS_BOYS_F32_, GS_BOYS_ORDER)};
constexpr int kBoysOrder = GS_BOYS_ORDER;
static_assert(kBoysOrder >= 0 && kBoysOrder <= BOYS_TAYLOR_MMAX, "Boys order without rows");
static_assert(sizeof(g_boys_row64) == kBoysRows64<kBoysOrder> * sizeof(BoysRow64),
              "rows of another threshold");
#else
constexpr int kBoysOrder = -1;
#endif

template <typename T> GS_HD GS_INLINE T ldg(const T* p) {
#if defined(__CUDA_ARCH__)
    return __ldg(p);
#else
    return *p;
#endif
}

// ------------------------------------------------------------------ work moved off the FP64 pipe
// A warp-wide FP64 instruction takes 64 cycles of its scheduler's pipe here (measured: 0.5
// lanes per clock, the same for one warp and for four), a conversion to or from double 82, a
// DSETP 64; an integer or FP32 instruction takes one.  These helpers do with a few integer
// operations on the IEEE words what would otherwise take such an instruction.

// (float)x, rounded to nearest even; the conversion itself outside the normal floats.
GS_HD GS_INLINE float narrow(double x) {
#if defined(__CUDA_ARCH__)
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned e = (hi >> 20) & 0x7ffu;
    if (e - 897u < 253u) {                    // 2^-126 <= |x| < 2^127
        const unsigned f = ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
        const unsigned rest = lo & 0x1fffffffu;
        const unsigned up = rest > 0x10000000u - (f & 1u) ? 1u : 0u;
        return __uint_as_float((hi & 0x80000000u) | (f + up));
    }
    if (((hi << 1) | lo) == 0) return __uint_as_float(hi);
#endif
    return (float)x;
}
GS_HD GS_INLINE double narrow_to(double, double x) { return x; }
GS_HD GS_INLINE float narrow_to(float, double x) { return narrow(x); }

// (double)x, exact; the conversion itself for zero, subnormals, infinities and NaN.
GS_HD GS_INLINE double widen(float x) {
#if defined(__CUDA_ARCH__)
    const unsigned b = __float_as_uint(x);
    if (((b >> 23) & 0xffu) - 1u < 254u)
        return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)),
                                (int)(b << 29));
#endif
    return (double)x;
}
GS_HD GS_INLINE double widen(double x) { return x; }

// 2 x, exact.
GS_HD GS_INLINE double twice(double x) {
#if defined(__CUDA_ARCH__)
    const int hi = __double2hiint(x);
    if ((((unsigned)hi >> 20) & 0x7ffu) - 1u < 0x7fdu)
        return __hiloint2double(hi + 0x00100000, __double2loint(x));
#endif
    return 2.0 * x;
}
GS_HD GS_INLINE float twice(float x) { return 2.0f * x; }

// The larger of two values that are not negative (densities' magnitudes): as integers.
GS_HD GS_INLINE double max_nonneg(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
#else
    return a > b ? a : b;
#endif
}

// a >= b for values that are not negative.
GS_HD GS_INLINE bool not_less(double a, double b) {
#if defined(__CUDA_ARCH__)
    return __double_as_longlong(a) >= __double_as_longlong(b);
#else
    return a >= b;
#endif
}

// High word of a whole number n, 1 <= n < 2^20, as a double.
GS_HD constexpr unsigned whole_hiword(unsigned n) {
    unsigned e = 0;
    for (unsigned m = n; m > 1; m >>= 1) ++e;
    return ((1023u + e) << 20) | ((n << (20 - e)) & 0xfffffu);
}

// t < n for t >= 0 and a whole number n: false for NaN.
template <unsigned N> GS_HD GS_INLINE bool below(double t) {
#if defined(__CUDA_ARCH__)
    return (unsigned)__double2hiint(t) < whole_hiword(N);
#else
    return t < (double)N;
#endif
}
template <unsigned N> GS_HD GS_INLINE bool below(float t) { return t < (float)N; }

// x / 2 for normal x with a normal half.
GS_HD GS_INLINE double halve(double x) {
#if defined(__CUDA_ARCH__)
    const int hi = __double2hiint(x);
    if ((((unsigned)hi >> 20) & 0x7ffu) - 2u < 0x7fdu)
        return __hiloint2double(hi - 0x00100000, __double2loint(x));
#endif
    return 0.5 * x;
}

// exp(x): x = k ln 2 + r by Cody and Waite's two-part ln 2, the Taylor sum of exp(r) to r^13
// (|r| <= ln 2 / 2: the rest is below 2^-57) with its terms from r^9 on, under 2^-32 of the sum,
// in float, and k added to the exponent; thirteen FP64 instructions where the library's function
// takes the time of 19.  |x| >= 700 and NaN go to the library's.
GS_HD GS_INLINE double gs_exp(double x) {
#if defined(__CUDA_ARCH__)
    if (((unsigned)__double2hiint(x) & 0x7fffffffu) < 0x4085e000u) {
        const double magic = 6755399441055744.0;
        const double kf = gs_fma(x, 1.4426950408889634074, magic);
        const double kd = gs_sub(kf, magic);
        const double r = gs_fma(kd, -2.3190468138462996e-17, gs_fma(kd, -0.69314718055994530942, x));
        const float f = narrow(r);
        float t = fmaf(f, 1.0f / 6227020800.0f, 1.0f / 479001600.0f);
        t = fmaf(f, t, 1.0f / 39916800.0f);
        t = fmaf(f, t, 1.0f / 3628800.0f);
        t = fmaf(f, t, 1.0f / 362880.0f);
        double y = gs_fma(widen(t), r, 1.0 / 40320.0);
        y = gs_fma(y, r, 1.0 / 5040.0);
        y = gs_fma(y, r, 1.0 / 720.0);
        y = gs_fma(y, r, 1.0 / 120.0);
        y = gs_fma(y, r, 1.0 / 24.0);
        y = gs_fma(y, r, 1.0 / 6.0);
        y = gs_fma(y, r, 0.5);
        y = gs_fma(y, r, 1.0);
        y = gs_fma(y, r, 1.0);
        return __hiloint2double(__double2hiint(y) + (__double2loint(kf) << 20), __double2loint(y));
    }
    return exp(x);
#else
    return std::exp(x);
#endif
}

// Nearest row k of the half-step grid of t >= 0 and T_k - t (exact), the rounding by the sum
// with 1.5 2^52, whose last bit is worth one.  k is held to the table whatever t is.
template <int M> GS_HD GS_INLINE int boys_row(double t, double& d) {
    const double magic = 6755399441055744.0;
    const double kf = gs_fma(t, BOYS_INV_H64, magic);
    const double kd = gs_sub(kf, magic);
    d = gs_fma(kd, 1.0 / BOYS_INV_H64, -t);
#if defined(__CUDA_ARCH__)
    return min((unsigned)__double2loint(kf), (unsigned)(kBoysRows64<M> - 1));
#else
    return kd >= 0 && kd < kBoysRows64<M> ? (int)kd : kBoysRows64<M> - 1;
#endif
}

// The seven-term expansion about a row, |d| <= 1/64: the three smallest terms, under 2^-28 of
// the sum, in float (df = d), four multiply-adds in FP64 instead of six.  (ss|ss) to (pp|ss)
// spend a quarter of a primitive quartet's FP64 instructions here.  With the downward recursion
// F_0..F_M, M = 0..9, are off by 2 to 9 x 2^-53 at most and 0.5 to 1.3 rms; seven terms in FP64 on
// the grid of twice the step by 4 to 55 and 0.6 to 7.5, most of it the terms left out.
GS_HD GS_INLINE double boys_horner(const double* c, const float* f, double d, float df) {
    const float tail = gs_fma(df, gs_fma(df, f[2], f[1]), f[0]);
    return gs_fma(gs_fma(gs_fma(gs_fma(widen(tail), d, c[3]), d, c[2]), d, c[1]), d, c[0]);
}

// F[m] = pref F_m(t), m = 0..M, from row r of order M: F_M and exp(-t) expanded about T_k,
// then the downward recursion of boys_small.
template <int M>
GS_HD GS_INLINE void boys_from_row(const BoysRow64& r, double t, double d, double pref,
                                   double* __restrict__ F) {
    const float df = narrow(d);
    F[M] = gs_mul(boys_horner(r.c, r.f, d, df), pref);
    if (M > 0) {
        const double et = gs_mul(boys_horner(r.e, r.x, d, df), pref);
        const double t2 = twice(t);
        GS_UNROLL for (int m = M; m >= 1; --m) {
            const double x = gs_fma(t2, F[m], et);
            F[m - 1] = m == 1 ? x : gs_mul(x, 1.0 / (2 * m - 1));
        }
    }
}

// Boys function of an FP64 quartet below BOYS_TMAX: Taylor expansion of F_M about the
// nearest grid point, then downward recursion
//   F_{m-1}(t) = (2t F_m(t) + e^{-t}) / (2m - 1),
// stable downwards; e^{-t} comes from the tabulated e^{-t_k} times the Taylor series of
// e^{-(t - t_k)}.  F[m] = pref * F_m(t).  Orders without rows expand 7 terms on the grid of
// step 1/BOYS_INV_H.
template <int M>
GS_HD GS_INLINE void boys_small(double t, double pref, double* __restrict__ F) {
#if defined(__CUDA_ARCH__) && defined(GS_BOYS_ORDER)
    if constexpr (M == kBoysOrder) {
        double d;
        const int k = boys_row<M>(t, d);
        boys_from_row<M>(g_boys_row64[k], t, d, pref, F);
        return;
    }
#endif
    const int k = (int)(t * BOYS_INV_H + 0.5);
    const double d = k * (1.0 / BOYS_INV_H) - t;
    const double* row = boys_table() + k * BOYS_NCOL;
    const double d2 = d * (1.0 / 2), d3 = d * (1.0 / 3), d4 = d * (1.0 / 4);
    const double d5 = d * (1.0 / 5), d6 = d * (1.0 / 6);
    double f = ldg(row + M + 6);
    f = f * d6 + ldg(row + M + 5);
    f = f * d5 + ldg(row + M + 4);
    f = f * d4 + ldg(row + M + 3);
    f = f * d3 + ldg(row + M + 2);
    f = f * d2 + ldg(row + M + 1);
    f = f * d + ldg(row + M);
    F[M] = f * pref;
    if (M > 0) {
        double e = d6 + 1.0;
        e = e * d5 + 1.0;
        e = e * d4 + 1.0;
        e = e * d3 + 1.0;
        e = e * d2 + 1.0;
        e = e * d + 1.0;
        const double et = e * ldg(row + BOYS_NCOL - 1) * pref;
        const double t2 = t + t;
        GS_UNROLL for (int m = M; m >= 1; --m) F[m - 1] = (t2 * F[m] + et) * (1.0 / (2 * m - 1));
    }
}

// The same below an FP32 quartet's threshold, without the FP64 pipe: F_M and exp(-t) as
// unevaluated sums of two floats.  row: twelve floats of grid point T_k (see
// boys_table_gen.c), d = T_k - t, exact in float (both are multiples of t's last place and
// |d| <= 1/32).  The leading term of each expansion and the linear one are pairs, so the float
// rounding of the rest, d^2 / 2 of it at most, is 2^-35 of the result; the downward recursion
// carries pairs with error-free sums and products (Dekker, Numer. Math. 18, 224 (1971)); each F_m
// is rounded to float once, as from FP64 (within 0.505 units in the last place, 0.2886 rms; with
// the linear term in one float 0.53 to 0.56 at most), and scaled.  About 17 FP32 instructions an
// order, against two FP64 ones and a conversion at 64 and 82 cycles a warp.
template <int M>
GS_HD GS_INLINE void boys_pair32(const float* __restrict__ r, float t, float d, float pref,
                                 float* __restrict__ F) {
    const float d2 = d * d;
    const float fp = d * r[2];                           // the linear term: fp + (fma + d lo)
    const float fr = fmaf(d, r[3], fmaf(d, r[2], -fp)) + d2 * fmaf(d, fmaf(d, r[6], r[5]), r[4]);
    float s0 = r[0] + fp;
    float z0 = (fp - (s0 - r[0])) + (r[1] + fr);         // |r[0]| >= |fp|
    float h = s0 + z0;
    float l = z0 - (h - s0);
    F[M] = h * pref;
    if (M > 0) {
        // exp(-t) = exp(-T_k) (1 + d + d^2 / 2 + ...)
        const float ep = r[8] * d;
        const float er = fmaf(r[9], d, fmaf(r[8], d, -ep)) +
                         r[8] * (d2 * fmaf(d, fmaf(d, 1.0f / 24, 1.0f / 6), 0.5f));
        s0 = r[8] + ep;
        z0 = (ep - (s0 - r[8])) + (r[9] + er);
        const float eh = s0 + z0;
        const float el = z0 - (eh - s0);
        const float t2 = t + t;
        GS_UNROLL for (int m = M; m >= 1; --m) {
            const float ph = t2 * h;
            const float pl = fmaf(t2, l, fmaf(t2, h, -ph));
            const float a = fmaxf(ph, eh), b = fminf(ph, eh);    // both positive
            float s = a + b;
            float z = (b - (s - a)) + (pl + el);
            if (m > 1) {                                  // times 1 / (2m - 1)
                const float ch = (float)(1.0 / (2 * m - 1));
                const float cl = (float)(1.0 / (2 * m - 1) - (double)ch);
                const float g = s * ch;
                z = fmaf(z, ch, fmaf(s, cl, fmaf(s, ch, -g)));
                s = g;
            }
            h = s + z;
            l = z - (h - s);
            F[m - 1] = h * pref;
        }
    }
}

// Boys function below the asymptotic threshold for an FP32 quartet: from the order's pair
// rows where the translation unit has them, else from the FP64 grid: the Taylor expansion
// cut after the d^4 term (its remainder, at most d^5/5! < 3e-10 of F_M for |d| <= 1/32, is
// far below FP32 rounding) and the downward recursion, all in FP64; each F_m is rounded to
// float once and then scaled by pref in float.  Per primitive quartet the FP64 form holds
// the FP64 pipe for 14 + 2.4 M instructions' time, the pair form not at all.
template <int M>
GS_HD GS_INLINE void boys_small32(float t, float pref, float* __restrict__ F) {
    static_assert(M + 4 <= BOYS_NCOL - 2, "Taylor terms beyond the tabulated orders");
#if defined(__CUDA_ARCH__) && defined(GS_BOYS_ORDER)
    if constexpr (M == kBoysOrder) {
        const float kf = fmaf(t, float(BOYS_INV_H), 12582912.0f);    // 1.5 2^23: rounds
        const unsigned k = min(__float_as_uint(kf) & 0x3fffffu, (unsigned)(BOYS_ROWS32 - 1));
        const float d = (kf - 12582912.0f) * (1.0f / BOYS_INV_H) - t;
        const float4* g = reinterpret_cast<const float4*>(g_boys_f32) + 3 * k;
        const float4 g0 = __ldg(g), g1 = __ldg(g + 1), g2 = __ldg(g + 2);
        const float r[10] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w, g2.x, g2.y};
        boys_pair32<M>(r, t, d, pref, F);
        return;
    }
#endif
    const int k = (int)(t * float(BOYS_INV_H) + 0.5f);
    const double d = (double)((float)k * (1.0f / BOYS_INV_H) - t);
    const double* row = boys_table() + k * BOYS_NCOL;
    const double d2 = d * (1.0 / 2), d3 = d * (1.0 / 3), d4 = d * (1.0 / 4);
    double Fd[M + 1];
    double f = ldg(row + M + 4);
    f = f * d4 + ldg(row + M + 3);
    f = f * d3 + ldg(row + M + 2);
    f = f * d2 + ldg(row + M + 1);
    Fd[M] = f * d + ldg(row + M);
    if (M > 0) {
        double e = d4 + 1.0;
        e = e * d3 + 1.0;
        e = e * d2 + 1.0;
        e = e * d + 1.0;
        const double et = e * ldg(row + BOYS_NCOL - 1);
        const double t2 = 2.0 * (double)t;
        GS_UNROLL for (int m = M; m >= 1; --m) Fd[m - 1] = (t2 * Fd[m] + et) * (1.0 / (2 * m - 1));
    }
    GS_UNROLL for (int m = 0; m <= M; ++m) F[m] = (float)Fd[m] * pref;
}

// F[m] = pref * F_m(t), m = 0..M.  Below the threshold: the expansion and the downward
// recursion in FP64 (boys_small), or for an FP32 quartet in pairs of floats, or FP64 for orders
// without rows, rounded to float once (boys_small32).  Above it: F_0 = sqrt(pi/t)/2 and the upward
// recursion F_{m+1} = (2m+1) F_m / (2t) in the quartet's precision, exact to its rounding
// there.  Neither branch needs an exponential: lanes of one warp that take different
// branches cost the sum of both.
template <int M, typename T>
GS_HD GS_INLINE void boys(T t, T pref, T* __restrict__ F) {
    static_assert(M <= 16, "Boys orders beyond the table");
    constexpr bool dbl = sizeof(T) == 8;
    constexpr unsigned thr = dbl ? kBoysAsym64[M] : kBoysAsym32[M];
    static_assert(thr <= (dbl ? BOYS_TMAX : BOYS_TMAX32), "asymptotic threshold beyond the grid");
    if (below<thr>(t)) {
        if constexpr (dbl) boys_small<M>(t, pref, F);
        else boys_small32<M>(t, pref, F);
    } else {
        const T rs = gs_rsqrt(t);
        F[0] = gs_mul(gs_mul(pref, T(0.88622692545275801365)), rs);   // sqrt(pi)/2
        if (M > 0) {
            const T hit = gs_mul(gs_mul(T(0.5), rs), rs);
            GS_UNROLL for (int m = 0; m < M; ++m)
                F[m + 1] = gs_mul(m == 0 ? hit : gs_mul(T(2 * m + 1), hit), F[m]);
        }
    }
}

// ------------------------------------------------------------------ one shell quartet
// Adds one primitive quartet's [e0|f0] targets to the contraction accumulators.
template <int LA, int LB, int LC, int LD, typename T>
GS_HD GS_INLINE void eri_primitive(const PrimRec<T>& P, const PrimRec<T>& Q,
                                   T* __restrict__ acc) {
    using G = ClassGen<LA, LB, LC, LD>;
    const T pq = gs_add(P.p, Q.p);
    const T PQx = gs_sub(Q.Px, P.Px), PQy = gs_sub(Q.Py, P.Py), PQz = gs_sub(Q.Pz, P.Pz);
    const T r2 = norm2(PQx, PQy, PQz);
#if defined(__CUDA_ARCH__) && defined(GS_BOYS_ORDER)
    if constexpr (G::L == 0 && sizeof(T) == 8 && kBoysOrder == 0) {
        // (ss|ss): with X = p q R^2, T = X / (p + q); far quartets (T >= threshold) need only
        // 1/sqrt(X), near ones only 1/sqrt(p + q), so one reciprocal square root serves a
        // warp that holds both, and the far lanes add nothing to the near lanes' work
        constexpr double thr = kBoysAsym64[0];
        const T X = gs_mul(gs_mul(P.p, Q.p), r2);
        const T u = fma(-thr, pq, X);
        const bool far = __double2hiint(u) >= 0;
        const T y = gs_rsqrt(far ? X : pq);
        T f = T(0.88622692545275801365);                 // sqrt(pi)/2
        if (!far) {
            double d;
            const int k = boys_row<0>(gs_mul(X, gs_mul(y, y)), d);
            f = boys_horner(g_boys_row64[k].c, g_boys_row64[k].f, d, narrow(d));
        }
        acc[0] = fma(gs_mul(gs_mul(P.Kp, Q.Kp), y), f, acc[0]);
        return;
    }
#endif
    const T rs = gs_rsqrt(pq);
    const T ipq = gs_mul(rs, rs);
    const T wq = gs_mul(Q.p, ipq), wp = gs_mul(P.p, ipq);
    const T t = gs_mul(gs_mul(P.p, wq), r2);
    T F[G::L + 1];
    boys<G::L, T>(t, gs_mul(gs_mul(P.Kp, Q.Kp), rs), F);
    VrrCoef<T> c;
    c.PAx = P.PAx; c.PAy = P.PAy; c.PAz = P.PAz;
    c.WPx = gs_mul(wq, PQx); c.WPy = gs_mul(wq, PQy); c.WPz = gs_mul(wq, PQz);
    c.QCx = Q.PAx; c.QCy = Q.PAy; c.QCz = Q.PAz;
    c.WQx = gs_mul(-wp, PQx); c.WQy = gs_mul(-wp, PQy); c.WQz = gs_mul(-wp, PQz);
    c.i2p = P.i2p; c.i2q = Q.i2p;
    c.rp2 = gs_mul(wq, P.i2p); c.rq2 = gs_mul(wp, Q.i2p);
    c.i2pq = gs_mul(T(0.5), ipq);
    G::vrr(F, c, acc);
}

// Contracted Cartesian block of the canonical quartet (bra | ket), in the component
// order of ClassGen (blk[((ia*NB+ib)*NC+ic)*ND+id]), without per-component scaling.  The
// ket's primitives are the outer loop: the lanes of a warp share the bra pair far more often
// than the ket pair, so the inner loop's loads fall on one line instead of 32.
template <int LA, int LB, int LC, int LD, typename T>
GS_HD GS_INLINE void eri_quartet(const PairRec& B, const PairRec& K,
                                 const PrimRec<T>* __restrict__ prims, T* __restrict__ blk) {
    using G = ClassGen<LA, LB, LC, LD>;
    T acc[G::NACC];
    GS_UNROLL for (int i = 0; i < G::NACC; ++i) acc[i] = T(0);
    for (int j = 0; j < K.nprim; ++j) {
        const PrimRec<T> Q = prims[K.prim_off + j];
        for (int i = 0; i < B.nprim; ++i)
            eri_primitive<LA, LB, LC, LD, T>(prims[B.prim_off + i], Q, acc);
    }
    G::hrr(acc, T(B.ABx), T(B.ABy), T(B.ABz), T(K.ABx), T(K.ABy), T(K.ABz), blk);
}

// Contraction accumulators of the quartet over primitive quartets start, start + stride,
// ... (flat index j * B.nprim + i, the order of eri_quartet): the lanes of a warp that shares one quartet's primitive
// quartets each call this with their own start and stride 32, then sum the accumulators.
template <int LA, int LB, int LC, int LD, typename T>
GS_HD GS_INLINE void eri_accumulate(const PairRec& B, const PairRec& K,
                                    const PrimRec<T>* __restrict__ prims, T* __restrict__ acc,
                                    int start, int stride) {
    const int nB = B.nprim, ntot = nB * K.nprim;
    for (int x = start; x < ntot; x += stride)
        eri_primitive<LA, LB, LC, LD, T>(prims[B.prim_off + x % nB], prims[K.prim_off + x / nB],
                                         acc);
}

// ------------------------------------------------------------------ shell-pair records
// Shells as the engine stores them: centre (bohr), angular momentum l, primitives
// [prim_off[s], prim_off[s+1]) with exponent and effective coefficient (contraction times
// primitive and contracted normalisation of the shell's first Cartesian component), and
// comp_scale[s*6 + i], the ratio of component i's normalisation to the first one's.
struct ShellView {
    const double* centre;
    const int* l;
    const int* prim_off;
    const double* expo;
    const double* coef;
};

constexpr double kSqrt2Pi52 = 5.914967172795613;  // sqrt(2 pi^(5/2))

// Record of the primitive pair (a at A, b at B, AB = A - B) with contraction coefficients ca, cb.
// P - A = -b/p AB is formed as such, not as a difference of centres (no cancellation), and P from
// the centre of the larger exponent, its nearer one: seven FP64 instructions for the six where
// (aA + bB)/p and P - A took twelve.  Over random shells (rms, units of 2^-53) P is off by 0.44,
// P - A by 0.88 and Kp by 31.3, most of it its exponent's rounding; the other way it was 0.90,
// 10^6 (from pairs of centres close to each other or of very different exponents) and 31.5.
GS_HD GS_INLINE PrimRec<double> prim_pair(const double* A, const double* B, double ABx, double ABy,
                                          double ABz, double a, double b, double ca, double cb) {
    PrimRec<double> r;
    const double p = gs_add(a, b);
    const double ip = gs_rcp(p);
    const double bp = gs_mul(b, ip);
    r.p = p;
    r.i2p = halve(ip);
    r.PAx = gs_mul(-bp, ABx); r.PAy = gs_mul(-bp, ABy); r.PAz = gs_mul(-bp, ABz);
    const double ap = gs_mul(a, ip);
    const bool near = not_less(a, b);
    const double w = near ? -bp : ap;
    const double* C = near ? A : B;
    r.Px = gs_fma(w, ABx, C[0]); r.Py = gs_fma(w, ABy, C[1]); r.Pz = gs_fma(w, ABz, C[2]);
    const double x = gs_mul(gs_mul(-a, bp), norm2(ABx, ABy, ABz));
    r.Kp = gs_mul(gs_mul(gs_mul(kSqrt2Pi52, ca), gs_mul(cb, ip)), gs_exp(x));
    r.pad = a;          // exponent of the first shell (derivative weights)
    return r;
}

GS_HD GS_INLINE PrimRec<float> prim_pair32(const PrimRec<double>& r) {
    PrimRec<float> f;
    f.p = narrow(r.p); f.i2p = narrow(r.i2p);
    f.Px = narrow(r.Px); f.Py = narrow(r.Py); f.Pz = narrow(r.Pz);
    f.PAx = narrow(r.PAx); f.PAy = narrow(r.PAy); f.PAz = narrow(r.PAz);
    f.Kp = narrow(r.Kp);
    f.pad0 = narrow(r.pad);      // exponent of the first shell (FP32 derivative weights)
    f.pad1 = f.pad2 = 0.0f;
    return f;
}

// Primitive-pair screen: drop the pair when its Gaussian-product factor exp(-ab/p |AB|^2)
// is below exp(-max_exp) (max_exp > 0).  Written without the division (ab |AB|^2 >
// max_exp p), which on this part costs more FP64 issue slots than the rest of the test.
GS_HD GS_INLINE bool prim_pair_kept(double a, double b, double ab2, double max_exp) {
    return !(max_exp > 0.0 && a * b * ab2 > max_exp * (a + b));
}

// The same decision from the centres' difference, in float where float's rounding (under 2e-6 of
// either side together) cannot change it, so that the test stays off the FP64 pipe.
GS_HD GS_INLINE bool prim_pair_kept(double a, double b, double ABx, double ABy, double ABz,
                                    double max_exp) {
#if defined(__CUDA_ARCH__)
    if (!(max_exp > 0.0)) return true;
    const float x = narrow(ABx), y = narrow(ABy), z = narrow(ABz), af = narrow(a), bf = narrow(b);
    const float t = af * bf * (x * x + y * y + z * z), lim = narrow(max_exp) * (af + bf);
    if (lim > 1e-30f && t < 1e38f) {              // no product beyond float's range
        if (t < lim * 0.99999f) return true;
        if (t > lim * 1.00001f) return false;
    }
#endif
    return prim_pair_kept(a, b, ABx * ABx + ABy * ABy + ABz * ABz, max_exp);
}

// Fill the PairRec and the primitive-pair records of shell pair (sa, sb); la >= lb.
// Primitive pairs whose Gaussian-product factor exp(-ab/p |AB|^2) is below exp(-max_exp)
// are dropped when max_exp > 0 (their contributions are below that factor times the
// normalised block's scale); pr.nprim is the number kept.  Host form (tests); the device
// builds the same records one warp per pair (capi.cu, k_pairs_build).
GS_HD GS_INLINE void make_pair(const ShellView& S, int sa, int sb, int prim_off, PairRec& pr,
                               PrimRec<double>* pd, PrimRec<float>* pf, double max_exp = 0.0) {
    const double* A = S.centre + 3 * sa;
    const double* B = S.centre + 3 * sb;
    const double ABx = A[0] - B[0], ABy = A[1] - B[1], ABz = A[2] - B[2];
    const double ab2 = ABx * ABx + ABy * ABy + ABz * ABz;
    const int a0 = S.prim_off[sa], a1 = S.prim_off[sa + 1];
    const int b0 = S.prim_off[sb], b1 = S.prim_off[sb + 1];
    pr.ABx = ABx; pr.ABy = ABy; pr.ABz = ABz;
    pr.prim_off = prim_off;
    pr.sa = sa; pr.sb = sb;
    pr.qmax = 0.0f; pr.pad = 0;
    int n = prim_off;
    for (int i = a0; i < a1; ++i) {
        for (int j = b0; j < b1; ++j) {
            const double a = S.expo[i], b = S.expo[j];
            if (!prim_pair_kept(a, b, ab2, max_exp)) continue;
            const PrimRec<double> r = prim_pair(A, B, ABx, ABy, ABz, a, b, S.coef[i], S.coef[j]);
            pd[n] = r;
            if (pf) pf[n] = prim_pair32(r);
            ++n;
        }
    }
    pr.nprim = n - prim_off;
}

// Original-order strides of a canonical block (see WriteTask::code).
GS_HD GS_INLINE void block_strides(int code, int nA, int nB, int nC, int nD, long long s[4]) {
    const bool b0 = code & 1, b1 = code & 2, b2 = code & 4;
    int n[4];
    int posA, posB, posC, posD;
    if (!b2) {
        n[0] = b0 ? nB : nA; n[1] = b0 ? nA : nB;
        n[2] = b1 ? nD : nC; n[3] = b1 ? nC : nD;
        posA = b0 ? 1 : 0; posB = 1 - posA;
        posC = b1 ? 3 : 2; posD = 5 - posC;
    } else {
        n[2] = b0 ? nB : nA; n[3] = b0 ? nA : nB;
        n[0] = b1 ? nD : nC; n[1] = b1 ? nC : nD;
        posA = b0 ? 3 : 2; posB = 5 - posA;
        posC = b1 ? 1 : 0; posD = 1 - posC;
    }
    long long st[4] = {(long long)n[1] * n[2] * n[3], (long long)n[2] * n[3], n[3], 1};
    s[0] = st[posA]; s[1] = st[posB]; s[2] = st[posC]; s[3] = st[posD];
}

}  // namespace gs
