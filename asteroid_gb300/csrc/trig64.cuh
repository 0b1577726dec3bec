// trig64.cuh -- FP64 sine and cosine from a table.
//
// The FP64 kernels take the number of their FP64 instructions times the unit's 64 cycles (a lone
// warp) or 19 (four warps on an SM), and most of an RK4 step's were the sine and cosine of two angles
// in each stage: sincos() issues 25.  With a point of a table of 1024 angles next to x, at most
// pi/1024 away, three terms of each series are enough and x's sine and cosine take 16; memory,
// integer and predicate instructions run beside them.  20 011 evaluations of 480 points 27.1 -> 22.6 ms, a
// curve of 20 000 points 153 -> 117 with each function on a lane of its own.
//
// The table holds the points' sine and cosine as unevaluated sums of two doubles: the results are
// within 0.6 ulp of 1 for one rounding of each sum, 1.2 ulp of themselves near the zeros
// (tests/test_trig64.py).  1024 points: with 512 each series needs one term more, with 4096 none less, and
// 32 KB stay in the L1.
#pragma once
#include <stdint.h>
#include <string.h>
#include "dfloat.cuh"

namespace ast {

constexpr int kTrig64 = 1024;

namespace trig64 {

// Double-double arithmetic for the table's constant initialiser (Dekker 1971, Knuth TAOCP 4.2.2).
struct dd {
    double hi, lo;
};
constexpr dd two_sum(double a, double b)
{
    const double s = a + b, bb = s - a;
    return dd{s, (a - (s - bb)) + (b - bb)};
}
constexpr dd fast_sum(double a, double b)
{
    const double s = a + b;
    return dd{s, b - (s - a)};
}
constexpr dd two_prod(double a, double b)
{
    const double ca = 134217729.0 * a, cb = 134217729.0 * b;  // 2^27 + 1
    const double ah = ca - (ca - a), bh = cb - (cb - b), al = a - ah, bl = b - bh;
    const double p = a * b;
    return dd{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr dd add(dd a, dd b)
{
    const dd s = two_sum(a.hi, b.hi), t = two_sum(a.lo, b.lo);
    const dd u = fast_sum(s.hi, s.lo + t.hi);
    return fast_sum(u.hi, u.lo + t.lo);
}
constexpr dd mul(dd a, dd b)
{
    const dd p = two_prod(a.hi, b.hi);
    return fast_sum(p.hi, p.lo + (a.hi * b.lo + a.lo * b.hi));
}
constexpr dd div(dd a, double b)
{
    const double q = a.hi / b;
    const dd p = two_prod(q, b);
    return fast_sum(q, ((a.hi - p.hi) - p.lo + a.lo) / b);
}

// A point's sine and cosine.
struct alignas(16) Point {
    double s, c, sl, cl;
};
struct Table {
    Point p[kTrig64];
};

// pi as two doubles (the binary expansion of pi cut after 53 and 106 bits).
constexpr dd kPi2{3.141592653589793116, 1.2246467991473532e-16};

constexpr Table make()
{
    Table T{};
    for (int k = 0; k <= kTrig64 / 8; k++) {
        // The Taylor series on [0, pi/4]; x^28 / 28! < 2^-107.
        const dd x = div(mul(kPi2, dd{2.0 * k, 0.0}), kTrig64);
        const dd x2 = mul(x, x);
        dd s = x, c{1.0, 0.0}, ts = x, tc{1.0, 0.0};
        for (int n = 1; n < 14; n++) {
            tc = div(mul(tc, x2), -(2.0 * n - 1.0) * (2.0 * n));
            ts = div(mul(ts, x2), -(2.0 * n) * (2.0 * n + 1.0));
            c = add(c, tc);
            s = add(s, ts);
        }
        // The other octants: sin(pi/2 - x) = cos x, and quarter turns.
        constexpr int Q = kTrig64 / 4;
        for (int m = 0; m < 2; m++) {
            const dd a = m ? c : s, b = m ? s : c;
            const int j = m ? Q - k : k;
            for (int q = 0; q < 4; q++) {
                const dd S = q == 0 ? a : q == 1 ? b : q == 2 ? dd{-a.hi, -a.lo} : dd{-b.hi, -b.lo};
                const dd C = q == 0 ? b : q == 1 ? dd{-a.hi, -a.lo} : q == 2 ? dd{-b.hi, -b.lo} : a;
                T.p[(j + q * Q) & (kTrig64 - 1)] = Point{S.hi, C.hi, S.lo, C.lo};
            }
        }
    }
    return T;
}

#ifdef __CUDACC__
static __device__ const Table kTable = make();
#endif
AST_HD Point point(int k)
{
#ifdef __CUDA_ARCH__
    const double2* row = reinterpret_cast<const double2*>(kTable.p + k);
    const double2 h = __ldg(row), l = __ldg(row + 1);
    return Point{h.x, h.y, l.x, l.y};
#else
    static const Table host = make();
    return host.p[k];
#endif
}

// Finite angles outside the reduction's range.  Cold: one copy.
static __host__ __device__ __noinline__ void beyond(double x, double* s, double* c) { sincos(x, s, c); }

}  // namespace trig64

// sin x and cos x.  x = k d + r with d = 2pi/T: x - k d is exact in one fma for d rounded to double
// (both terms are multiples of 2^-62 unless k = 0, and the difference is below 2^-8), and d's rest
// enters with another; k is within half a step and its own product's rounding, 2^-5 of one at |x| =
// 2^40.  Infinities and NaN give NaN.  Every rounding explicit: the same bits in every kernel.
//
// shift: added to the table point, kTrig64 / 4 for (cos x, -sin x); the points a quarter turn on are
// the same numbers, so the bits are, too.  Without c only the first is computed, in 13 instructions.
AST_HD void sincos_tab(double x, double* s, double* c, int shift = 0)
{
    constexpr double kStep = 2.0 * trig64::kPi2.hi / kTrig64, kStepLo = 2.0 * trig64::kPi2.lo / kTrig64;
    const double magic = 6755399441055744.0;  // 1.5 2^52
    const double kb = DD_FMA(x, kTrig64 / (2.0 * trig64::kPi2.hi), magic);
    const double k = DD_SUB(kb, magic);
    const double r = DD_FMA(-k, kStepLo, DD_FMA(-k, kStep, x));
    uint64_t xb, bits;
#ifdef __CUDA_ARCH__
    xb = (uint64_t)__double_as_longlong(x);
    bits = (uint64_t)__double_as_longlong(kb);
#else
    memcpy(&xb, &x, 8);
    memcpy(&bits, &kb, 8);
#endif
    if (((uint32_t)(xb >> 32) & 0x7fffffffu) - 0x42700000u < 0x3d800000u) {  // 2^40 <= |x| < infinity
        double sx, cx;
        trig64::beyond(x, &sx, &cx);
        *s = shift ? cx : sx;
        if (c) *c = shift ? -sx : cx;
        return;
    }
    const trig64::Point P = trig64::point((int)((bits + (uint32_t)shift) & (kTrig64 - 1)));
    const double r2 = DD_MUL(r, r);
    const double sr = DD_FMA(DD_MUL(r, r2), DD_FMA(r2, 1.0 / 120.0, -1.0 / 6.0), r);  // sin r
    const double v = DD_MUL(r2, DD_FMA(r2, 1.0 / 24.0, -0.5));                        // cos r - 1
    *s = DD_ADD(P.s, DD_FMA(P.c, sr, DD_FMA(P.s, v, P.sl)));
    if (c) *c = DD_ADD(P.c, DD_FMA(-P.s, sr, DD_FMA(P.c, v, P.cl)));
}

// 1/s and 1/sqrt(x) within 2^-20 (measured: 2^-20.02 and 2^-20.08; the instructions read and write the upper 32 bits
// of a double), by the special function unit: no FP64 instruction.
AST_HD double rcp_seed(double s)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    return y;
#else
    return (double)(1.0f / (float)s);
#endif
}
AST_HD double rsqrt_seed(double x)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
#else
    return (double)(1.0f / sqrtf((float)x));
#endif
}

// 1 / s in three instructions: one cubic step (Householder's method of order 2), y + y (e + e^2), e = 1 - s y, leaves
// e^3 < 2^-60; 0.51 ulp.
AST_HD double recip(double s)
{
    const double y = rcp_seed(s);
    const double e = DD_FMA(-s, y, 1.0);
    return DD_FMA(y, DD_FMA(e, e, e), y);
}
// u / s in six instructions, against ten of the division: the reciprocal and the quotient's remainder (Markstein 1990),
// whose correction leaves 0.5 ulp and a 2^-52th of one.  No zero, infinite or denormal s, where the quotient is infinite
// and this NaN: an evaluation's chi^2 is NaN either way.
AST_HD double quot(double u, double s)
{
    const double y = recip(s);
    const double q = DD_MUL(u, y);
    return DD_FMA(DD_FMA(-s, q, u), y, q);
}
// 1 / sqrt(x) in six instructions, against twenty of root and division: the same step for x^(-1/2),
// y + y e (1/2 + 3/8 e), e = 1 - x y^2 < 2^-19, leaves 5/16 e^3 < 2^-58; 1 ulp.
AST_HD double inv_sqrt(double x)
{
    const double y0 = rsqrt_seed(x);
    const double e = DD_FMA(-DD_MUL(x, y0), y0, 1.0);
    return DD_FMA(DD_MUL(y0, e), DD_FMA(e, 0.375, 0.5), y0);
}

// The sine and cosine of an FP64 evaluation.  Evaluations proper (ast_eval_batch, curves, the FP64 chi^2
// reported of a mixed search) take the table's.  The FP64 simplex search keeps the library's: it chooses
// between chi^2 of models from the prior that no step resolves, where a sine's last bit decides (one of
// 2048 such chains then takes another number of evaluations).
struct TrigTable {
    static constexpr bool kAlgebraic = true;  // and ls_algebraic (model.cuh)
    static __device__ __forceinline__ void sincos(double x, double* s, double* c) { sincos_tab(x, s, c); }
    static __device__ __forceinline__ double sin_or_cos(double x, bool cosine)
    {
        double r;
        sincos_tab(x, &r, nullptr, cosine ? kTrig64 / 4 : 0);
        return r;
    }
    static __device__ __forceinline__ double div(double u, double s) { return quot(u, s); }
};
struct TrigLibrary {
    static constexpr bool kAlgebraic = false;
    static __device__ __forceinline__ void sincos(double x, double* s, double* c) { ::sincos(x, s, c); }
    static __device__ __forceinline__ double sin_or_cos(double x, bool cosine)
    {
        double s, c;
        ::sincos(x, &s, &c);
        return cosine ? c : s;
    }
    static __device__ __forceinline__ double div(double u, double s) { return u / s; }
};
// The parity build (build_parity_engine) evaluates as the search does, in the reference's expressions.
#ifdef AST_LIBRARY_TRIG
using TrigEval = TrigLibrary;
#else
using TrigEval = TrigTable;
#endif

}  // namespace ast
