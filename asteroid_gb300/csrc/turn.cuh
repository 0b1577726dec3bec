// turn.cuh -- the RK4 step of the mixed path: compact angles, unnormalised double-floats.
//
// The step of rk4_step_df2 (mixed.cuh) with the same stages, K1..K4 and combination
// (cuda.c:319-372), and the same target -- a few u^2 (u = 2^-24) of the state per step -- in half
// the FP32 operations.  The kernels that run it are bound by the FP32 pipe, so its lane operations
// are its time.  What it does differently:
//
//  * An angle is k table steps plus a remainder, a = (k + e + t) 2pi/T with |e| <= 1/2 and t a small
//    correction (Turn).  Advancing it adds the increment to (e, t) and takes the nearest
//    whole number of steps out again: four operations that are at the same time the argument
//    reduction of the next sin and cos.  The rounding of an update is u^2 of the increment, not
//    of the accumulated angle.
//  * T = 4096: sin and cos of the remainder need e^3/6 and e^4/24 only, both far below u, so the
//    table point and the remainder combine in seven operations each (turn_sincos).  256 points
//    take double-float products of full length.
//  * Time is counted in steps: w = h omega, so a stage point is y + K/2 or y + K, a sum with an
//    exactly scaled operand, and the right-hand side's constants absorb h once an interval.
//  * Products and sums keep the low word as it comes (|lo| of a few ulp(hi)) where the next
//    operation takes it so; a quotient's divisor and the stored state are normalised.
//  * The angular velocity carries a third word, its own rounding of the last update, which is
//    what the accumulated phase depended on most.
//
// A stage costs 250 lane operations against 555 (torque), 120 against 310 (free rotation).
#pragma once
#include "dfloat.cuh"

namespace ast {

// A double-float as a pair that need not be normalised.
AST_HD df u_mul(df x, df y)
{
    const float p = DF_MUL(x.hi, y.hi);
    return df{p, DF_FMA(x.lo, y.hi, DF_FMA(x.hi, y.lo, DF_FMA(x.hi, y.hi, -p)))};
}
AST_HD df u_add(df x, df y)
{
    const df s = two_sum(x.hi, y.hi);
    return df{s.hi, DF_ADD(s.lo, DF_ADD(x.lo, y.lo))};
}
// x y + z w
AST_HD df u_dot(df x, df y, df z, df w)
{
    const float p = DF_MUL(x.hi, y.hi), q = DF_MUL(z.hi, w.hi);
    const float pe = DF_FMA(x.lo, y.hi, DF_FMA(x.hi, y.lo, DF_FMA(x.hi, y.hi, -p)));
    const float qe = DF_FMA(z.lo, w.hi, DF_FMA(z.hi, w.lo, DF_FMA(z.hi, w.hi, -q)));
    const df s = two_sum(p, q);
    return df{s.hi, DF_ADD(s.lo, DF_ADD(pe, qe))};
}
// y + c k, c a power of two: c k.hi is exact, so the two-sum takes it in fused form.
AST_HD df u_axpy(df y, float c, df k)
{
    const float s = DF_FMA(c, k.hi, y.hi);
    const float bb = DF_SUB(s, y.hi);
    const float e = DF_ADD(DF_SUB(y.hi, DF_SUB(s, bb)), DF_FMA(c, k.hi, -bb));
    return df{s, DF_ADD(DF_FMA(c, k.lo, y.lo), e)};
}
AST_HD df2 u_axpy2(df2 y, float2 c, df2 k)
{
    const float2 s = f2_fma(c, k.hi, y.hi);
    const float2 bb = f2_sub(s, y.hi);
    const float2 e = f2_add(f2_sub(y.hi, f2_sub(s, bb)), f2_fma(c, k.hi, f2_neg(bb)));
    return df2{s, f2_add(f2_fma(c, k.lo, y.lo), e)};
}

// ------------------------------------------------ compact angles

// The angle (k/4 + e + t) 2pi/T, |e| <= 1/2, k taken modulo a multiple of 4 T by its owner: k counts
// the bytes of the table, so that one mask gives the address of all four words of sin and cos.
struct Turn {
    uint32_t k;
    float e, t;
};
struct Turn2 {
    uint32_t k0, k1;
    float2 e, t;
};

constexpr double kTurnStep = 6.283185307179586477 / kTurn;  // radians
constexpr float kTurnStepHi = (float)kTurnStep, kTurnStepLo = (float)(kTurnStep - (double)kTurnStepHi);
// The largest sum of an angle's remainder and an increment whose number of steps the 1.5*2^23
// rounding takes exactly.
constexpr float kTurnMax = 4194304.0f;

// k0 steps + a -> Turn.  a.hi minus the nearest integer is exact.
AST_HD Turn turn_reduce(df a, uint32_t k0)
{
    const float magic = 12582912.0f;
    const float kb = DF_ADD(a.hi, magic);
    return Turn{k0 + 4u * (uint32_t)DF_BITS(kb), DF_SUB(a.hi, DF_SUB(kb, magic)), a.lo};
}
AST_HD Turn2 turn_reduce2(df2 a, uint32_t k0, uint32_t k1)
{
    const float2 magic = f2(12582912.0f);
    const float2 kb = f2_add(a.hi, magic);
    return Turn2{k0 + 4u * (uint32_t)DF_BITS(kb.x), k1 + 4u * (uint32_t)DF_BITS(kb.y),
                 f2_sub(a.hi, f2_sub(kb, magic)), a.lo};
}
AST_HD df2 turn_rest(const Turn2& a) { return df2{a.e, a.t}; }

// The value in radians of a compact angle whose k/4 counts modulo `turns` times T, in
// [-turns pi, turns pi].
AST_HD df turn_value(uint32_t k, float e, float t, int turns)
{
    const int half = turns * kTurn / 2;
    int m = (int)(((k >> 2) + (uint32_t)half) & (uint32_t)(turns * kTurn - 1)) - half;
    if (m == -half && e < 0.0f) m = half;
    const float n = (float)m;
    return df_mul(df_add_f(two_sum(n, e), t), df{kTurnStepHi, kTurnStepLo});
}

// An angle in radians as a compact one (turns = 1), or twice it (turns = 2, its k/4 modulo 2 T).
AST_HD Turn turn_from(df a, int turns = 1)
{
    const df one = df_from_double(1.0 / kTurnStep), two = df_from_double(2.0 / kTurnStep);
    const df r = df_mul(df_reduce_2pi(a), turns == 1 ? one : two);
    return turn_reduce(r, 0);
}

// sin and cos of two compact angles.  With x = (e + t) 2pi/T = xh + xl: sin x = xh + sl, cos x =
// 1 - v, and sin(a) = S + C (xh + sl) - S v, cos(a) = C - S (xh + sl) - C v from the table's S, C.
// The leading sum h = S + C.hi xh is one fma, its remainder C.hi xh - (h - S) another (h - S is
// exact: |C xh| <= |S| / 2, or S = 0).  The sums are normalised: their low words, up to 4e-7 from S v,
// would carry that much rounding through every product and sum that follows.
AST_HD void turn_sincos2(const Turn2& a, const float* __restrict__ tab, df2* s, df2* c)
{
    const float* t0 = reinterpret_cast<const float*>(reinterpret_cast<const char*>(tab) + (a.k0 & (4 * kTurn - 1)));
    const float* t1 = reinterpret_cast<const float*>(reinterpret_cast<const char*>(tab) + (a.k1 & (4 * kTurn - 1)));
    const float2 Sh = make_float2(t0[0], t1[0]), Sl = make_float2(t0[kTurnRow], t1[kTurnRow]);
    const float2 Ch = make_float2(t0[kTurn / 4], t1[kTurn / 4]);
    const float2 Cl = make_float2(t0[kTurnRow + kTurn / 4], t1[kTurnRow + kTurn / 4]);
    const float2 c1 = f2(kTurnStepHi);
    const float2 xh = f2_mul(c1, a.e);
    const float2 xl = f2_fma(c1, a.t, f2_fma(f2(kTurnStepLo), a.e, f2_fma(c1, a.e, f2_neg(xh))));
    const float2 x = f2_add(xh, xl);
    const float2 x2 = f2_mul(x, x);
    const float2 sl = f2_fma(f2_mul(x2, x), f2(-1.0f / 6.0f), xl);
    const float2 v = f2_mul(x2, f2_fma(x2, f2(-1.0f / 24.0f), f2(0.5f)));
    const float2 nS = f2_neg(Sh);
    {
        const float2 h = f2_fma(Ch, xh, Sh);
        const float2 z = f2_sub(Sh, h);
        const float2 r = f2_fma(nS, v, f2_fma(Ch, sl, f2_fma(Cl, xh, Sl)));
        *s = fast_two_sum2(h, f2_add(f2_fma(Ch, xh, z), r));
    }
    {
        const float2 h = f2_fma(nS, xh, Ch);
        const float2 z = f2_sub(Ch, h);
        const float2 r = f2_fma(f2_neg(Ch), v, f2_fma(nS, sl, f2_fma(f2_neg(Sl), xh, Cl)));
        *c = fast_two_sum2(h, f2_add(f2_fma(nS, xh, z), r));
    }
}

// ------------------------------------------------ the step

// (e, t) + a / 6.  The quotient's remainder a.hi - 6 p is exact in one fma: a product with 1/6 as
// a double-float would turn every increment by the same 1e-15 and the phase with them.
AST_HD df turn_sixth(float e, float t, df a)
{
    const float c = 1.0f / 6.0f;
    const float p = DF_MUL(c, a.hi);
    const float pe = DF_MUL(c, DF_ADD(DF_FMA(-6.0f, p, a.hi), a.lo));
    const df s = two_sum(e, p);
    return df{s.hi, DF_ADD(DF_ADD(t, pe), s.lo)};
}
AST_HD df2 turn_sixth2(df2 y, df2 a)
{
    const float2 c = f2(1.0f / 6.0f);
    const float2 p = f2_mul(c, a.hi);
    const float2 pe = f2_mul(c, f2_add(f2_fma(f2(-6.0f), p, a.hi), a.lo));
    const df2 s = two_sum2(y.hi, p);
    return df2{s.hi, f2_add(f2_add(y.lo, pe), s.lo)};
}

// Three words w = hi + lo + r: w + c a, the rounding of the low word kept in r.
AST_HD void word3_mad(df& w, float& r, df c, df a)
{
    const float p = DF_MUL(c.hi, a.hi);
    const float pe = DF_FMA(c.lo, a.hi, DF_FMA(c.hi, a.lo, DF_FMA(c.hi, a.hi, -p)));
    const df s = two_sum(w.hi, p);
    const df l = two_sum(w.lo, DF_ADD(DF_ADD(pe, r), s.lo));
    w = fast_two_sum(s.hi, l.hi);
    r = l.lo;
}

// The integrated state.  Torque (cuda.c:46-58): angular velocity w in rad/day (three words each),
// phi, and a = (psi, theta).  Free rotation (cuda.c:69-75): phi and a = (2 psi, theta), the first k/4
// modulo 2 T, so that psi is half of it modulo 2 pi.
struct Spin {
    df w[3];
    float r[3];
    Turn phi;
    Turn2 a;
};
// Constants of an interval.  Torque, q = h T/2pi: q, 1/(6q), q h (Ti, Ts, Tl).  Free rotation: k =
// q (L, L Ip, L Im).
struct SpinStep {
    df q, c6, k[3];
};

// One step of torqued rotation; mu = 2pi/T ((Is-1)/Ii, (1-Ii)/Is, Ii-Is).  Returns false and
// leaves the state alone where an angle advances too far for the reduction (a blown-up rotation).
AST_HD bool turn_step_torque(Spin& Y, const SpinStep& C, const df* mu, const float* __restrict__ tab)
{
    const df W0 = u_mul(Y.w[0], C.q), W1 = u_mul(Y.w[1], C.q), W2 = u_mul(Y.w[2], C.q);
    df2 w01 = df2_pack(W0, W1);
    const df2 W01 = w01;
    df w2 = W2;
    Turn2 a = Y.a;
    const df2 A = turn_rest(a);
    df2 K01, K23, KA;  // w0 w1, w2 phi, psi theta
    float big = 0.0f;
    auto rhs = [&]() {
        df2 s, c;
        turn_sincos2(a, tab, &s, &c);
        const df w0 = df2_x(w01), w1 = df2_y(w01);
        const df s5 = df2_x(s), c5 = df2_x(c), s4 = df2_y(s), c4 = df2_y(c);
        const df K0 = u_add(u_mul(mu[0], u_mul(w1, w2)), C.k[0]);
        const df K1 = u_add(u_mul(mu[1], u_mul(w2, w0)), C.k[1]);
        const df K2 = u_add(u_mul(mu[2], u_mul(w0, w1)), C.k[2]);
        const df u = u_dot(w0, s5, w1, c5);
        const df K4 = u_dot(w0, c5, df_neg(w1), s5);
        const float inv = DF_RCP_APPROX(s4.hi);
        const float q = DF_MUL(u.hi, inv);
        const df K3{q, DF_MUL(DF_FMA(-s4.lo, q, DF_ADD(DF_FMA(-s4.hi, q, u.hi), u.lo)), inv)};
        const float p = DF_MUL(q, c4.hi);
        const float pe = DF_FMA(K3.lo, c4.hi, DF_FMA(q, c4.lo, DF_FMA(q, c4.hi, -p)));
        const df d = two_sum(w2.hi, -p);
        K01 = df2_pack(K0, K1);
        K23 = df2_pack(K2, K3);
        KA = df2_pack(df{d.hi, DF_ADD(d.lo, DF_SUB(w2.lo, pe))}, K4);
    };
    auto next = [&](float h) {  // the next stage's point, y + h K
        w01 = u_axpy2(W01, f2(h), K01);
        w2 = u_axpy(W2, h, df2_x(K23));
        const df2 b = u_axpy2(A, f2(h), KA);
        big = fmaxf(big, fmaxf(fabsf(b.hi.x), fabsf(b.hi.y)));
        a = turn_reduce2(b, Y.a.k0, Y.a.k1);
    };
    // K1 + 2 K2 + 2 K3 + K4.  The ends apart: their sums and their next point need less, and the
    // middle stays one rolled copy for the instruction cache (33.0 ms against 35.1 rolled whole
    // and 34.9 unrolled whole, 58 368 evaluations of a 60-day light curve).
    rhs();
    df2 acc01 = K01, acc23 = K23, accA = KA;
    next(0.5f);
#pragma unroll 1
    for (int st = 1; st < 3; st++) {
        rhs();
        acc01 = u_axpy2(acc01, f2(2.0f), K01);
        acc23 = u_axpy2(acc23, f2(2.0f), K23);
        accA = u_axpy2(accA, f2(2.0f), KA);
        next(st == 1 ? 0.5f : 1.0f);
    }
    rhs();
    acc01 = u_axpy2(acc01, f2(1.0f), K01);
    acc23 = u_axpy2(acc23, f2(1.0f), K23);
    accA = u_axpy2(accA, f2(1.0f), KA);
    const df2 b = turn_sixth2(A, accA);
    const df f = turn_sixth(Y.phi.e, Y.phi.t, df2_y(acc23));
    big = fmaxf(fmaxf(big, fabsf(f.hi)), fmaxf(fabsf(b.hi.x), fabsf(b.hi.y)));
    if (big > kTurnMax) return false;
    Y.a = turn_reduce2(b, Y.a.k0, Y.a.k1);
    Y.phi = turn_reduce(f, Y.phi.k);
    word3_mad(Y.w[0], Y.r[0], C.c6, df2_x(acc01));
    word3_mad(Y.w[1], Y.r[1], C.c6, df2_y(acc01));
    word3_mad(Y.w[2], Y.r[2], C.c6, df2_x(acc23));
    return true;
}

AST_HD bool turn_step_free(Spin& Y, const SpinStep& C, const float* __restrict__ tab)
{
    Turn2 a = Y.a;
    const df2 A = turn_rest(a);
    df2 KA;
    df K0;
    float big = 0.0f;
    auto rhs = [&]() {
        df2 s, c;
        turn_sincos2(a, tab, &s, &c);
        K0 = u_add(C.k[1], df_neg(u_mul(C.k[2], df2_x(c))));
        const df K1 = u_mul(u_mul(C.k[2], df2_y(s)), df2_x(s));
        const df d = u_add(C.k[0], df_neg(K0));
        KA = df2_pack(u_mul(df2_y(c), df{DF_MUL(2.0f, d.hi), DF_MUL(2.0f, d.lo)}), K1);
    };
    auto next = [&](float h) {
        const df2 b = u_axpy2(A, f2(h), KA);
        big = fmaxf(big, fmaxf(fabsf(b.hi.x), fabsf(b.hi.y)));
        a = turn_reduce2(b, Y.a.k0, Y.a.k1);
    };
    rhs();
    df2 accA = KA;
    df accF = K0;
    next(0.5f);
#pragma unroll 1
    for (int st = 1; st < 3; st++) {
        rhs();
        accA = u_axpy2(accA, f2(2.0f), KA);
        accF = u_axpy(accF, 2.0f, K0);
        next(st == 1 ? 0.5f : 1.0f);
    }
    rhs();
    accA = u_axpy2(accA, f2(1.0f), KA);
    accF = u_axpy(accF, 1.0f, K0);
    const df2 b = turn_sixth2(A, accA);
    const df f = turn_sixth(Y.phi.e, Y.phi.t, accF);
    big = fmaxf(fmaxf(big, fabsf(f.hi)), fmaxf(fabsf(b.hi.x), fabsf(b.hi.y)));
    if (big > kTurnMax) return false;
    Y.a = turn_reduce2(b, Y.a.k0, Y.a.k1);
    Y.phi = turn_reduce(f, Y.phi.k);
    return true;
}

}  // namespace ast
