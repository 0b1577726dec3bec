// animate.cu -- frames of the ANIMATE build (compute_rgb, cuda.c:2394-2540 of the reference).
//
// The reference runs chi2_plot<<<ceil(SIZE_PIX^2 / BSIZE), BSIZE>>> in which every thread
// integrates the whole model over the plot grid (one RK4 recursion per pixel) and, at each
// snapshot, shades its own pixel: four lines of sight through the pixel's corners intersected with
// the triaxial ellipsoid, Lambert-like shading between terminator, shadow and sunlit colours, a
// red spot around the end of the b axis.  Here the recursion runs once (ast_model_geometry: one
// warp, the FP64 evaluation) and render_kernel shades every pixel of every frame from
// that geometry: one CTA per 32 x 8 tile of a frame, frames on the grid's y dimension, the frame's
// 20 doubles in shared memory, each line of sight through a pixel corner evaluated once and shared
// by the four pixels that meet there.  The bytes are those of the reference's FP64 arithmetic with
// every rounding explicit (no contracted multiply-adds), so that the CPU restatement reproduces
// each one: values are computed in double-float with a bound on their error, and again in that FP64
// arithmetic where a comparison or a byte's rounding lies within the bound.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>

#include "asteroid_gb300.h"
#include "dfloat.cuh"
#include "engine.cuh"

namespace ast {
namespace {

constexpr int kRenderTpb = 256;
// Colours (asteroid.h:300-313): deepest shadow, terminator, brightest sunlit element.
constexpr float kSminR = 6, kSminG = 8, kSminB = 10;
constexpr float kSmaxR = 30, kSmaxG = 41, kSmaxB = 53;
constexpr float kImaxR = 255, kImaxG = 191, kImaxB = 144;
constexpr float kSpotRad = 0.04f;  // SPOT_RAD (asteroid.h:315), a float: its square is rounded to float

#define M_(a, b) DD_MUL(a, b)
#define A_(a, b) DD_ADD(a, b)
#define S_(a, b) DD_SUB(a, b)

// Float pre-test of a corner line of sight.  Most lines of sight miss the ellipsoid; the
// reference settles them with the FP64 discriminant D = B^2 - 4AC < 0.  Here D is first formed in
// float together with a running bound on its error (each product x*y adds |x| e(y) + |y| e(x) +
// u|xy|, each sum e(x) + e(y) + u|x+y|, u = 2^-24, the inputs carrying one rounding each).  When
// D + 2 e(D) + 1e-12 M < 0 (M the sum of the magnitudes of D's terms, far above FP64's own
// rounding of them), the FP64 D is negative too and the corner is background; every other corner
// takes the reference's FP64 expressions, so the frame is the same byte for byte.
struct ScreenF {
    float Y1x, Y1y, Y1z, Z1x, Z1z;
    float ax[9];  // body axes b, c, a in inertial coordinates
    float Epb, Epc, Epa, ibb, icc, A;
};

__device__ __forceinline__ bool screen_background(const ScreenF& F, int cz, int cy, int S)
{
    constexpr float u = 5.9604645e-8f;  // 2^-24
    const float fS = (float)S;
    const float z1 = (2.4f * (float)(cz - S / 2)) / fS;
    const float y1 = (2.4f * (float)(cy - S / 2)) / fS;
    const float ez1 = 4.f * u * fabsf(z1), ey1 = 4.f * u * fabsf(y1);  // 2.4f, product, quotient
    // products and sums with their error bounds
#define PM(x, ex, y, ey, z, ez) \
    const float z = (x) * (y); \
    const float ez = fabsf(x) * (ey) + fabsf(y) * (ex) + u * fabsf(z);
#define PS(x, ex, y, ey, z, ez) \
    const float z = (x) + (y); \
    const float ez = (ex) + (ey) + u * fabsf(z);
    const float eY1x = u * fabsf(F.Y1x), eY1y = u * fabsf(F.Y1y), eY1z = u * fabsf(F.Y1z);
    const float eZ1x = u * fabsf(F.Z1x), eZ1z = u * fabsf(F.Z1z);
    PM(y1, ey1, F.Y1x, eY1x, yx, eyx) PM(z1, ez1, F.Z1x, eZ1x, zx, ezx) PS(yx, eyx, zx, ezx, px, epx)
    PM(y1, ey1, F.Y1y, eY1y, py, epy)
    PM(y1, ey1, F.Y1z, eY1z, yz, eyz) PM(z1, ez1, F.Z1z, eZ1z, zz, ezz) PS(yz, eyz, zz, ezz, pz, epz)
    float pbca[3], epbca[3];
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const float a0 = F.ax[3 * r], a1 = F.ax[3 * r + 1], a2 = F.ax[3 * r + 2];
        PM(a0, u * fabsf(a0), px, epx, t0, et0) PM(a1, u * fabsf(a1), py, epy, t1, et1)
        PM(a2, u * fabsf(a2), pz, epz, t2, et2) PS(t0, et0, t1, et1, s01, es01) PS(s01, es01, t2, et2, sr, esr)
        pbca[r] = sr;
        epbca[r] = esr;
    }
    const float pb = pbca[0], pc = pbca[1], pa = pbca[2], epb = epbca[0], epc = epbca[1], epa = epbca[2];
    const float eEpb = u * fabsf(F.Epb), eEpc = u * fabsf(F.Epc), eEpa = u * fabsf(F.Epa);
    const float eibb = u * F.ibb, eicc = u * F.icc, eA = u * fabsf(F.A);
    // B = 2 (pb Epb / b^2 + pc Epc / c^2 + pa Epa)
    PM(pb, epb, F.Epb, eEpb, b1, eb1) PM(b1, eb1, F.ibb, eibb, tb, etb)
    PM(pc, epc, F.Epc, eEpc, c1, ec1) PM(c1, ec1, F.icc, eicc, tc, etc_)
    PM(pa, epa, F.Epa, eEpa, ta, eta) PS(tb, etb, tc, etc_, s1, es1) PS(s1, es1, ta, eta, s2, es2)
    const float B = 2.f * s2, eB = 2.f * es2;
    const float Babs = 2.f * (fabsf(tb) + fabsf(tc) + fabsf(ta));
    // C = pb^2 / b^2 + pc^2 / c^2 + pa^2 - 1
    PM(pb, epb, pb, epb, q1, eq1) PM(q1, eq1, F.ibb, eibb, qb, eqb)
    PM(pc, epc, pc, epc, q2, eq2) PM(q2, eq2, F.icc, eicc, qc, eqc)
    PM(pa, epa, pa, epa, qa, eqa) PS(qb, eqb, qc, eqc, r1, er1) PS(r1, er1, qa, eqa, r2, er2)
    PS(r2, er2, -1.f, 0.f, C, eC)
    const float Cabs = qb + qc + qa + 1.f;
    // D = B^2 - 4 A C
    PM(B, eB, B, eB, BB, eBB) PM(F.A, eA, C, eC, AC, eAC) PS(BB, eBB, -4.f * AC, 4.f * eAC, D, eD)
#undef PM
#undef PS
    const float M = Babs * Babs + 4.f * fabsf(F.A) * Cabs;
    return D + 2.f * eD + 1e-12f * M < 0.f;
}

constexpr int kTileX = 32, kTileY = 8;
constexpr int kCorners = (kTileX + 1) * (kTileY + 1);
static_assert(kTileX * kTileY == kRenderTpb, "one thread per pixel of the tile");

// What the frame's geometry gives, once a frame: the reference's FP64 values, and the same quantities as
// double-floats for the corners.  A point of the image plane is p = y1 Y1 + z1 Z1, so p's body components,
// the quadratic's B and its discriminant D = B^2 - 4 A C are polynomials in (y1, z1).
struct FrameConst {
    double Z1x, Z1z, Y1x, Y1y, Y1z, A;
    ScreenF F;
    df al[3], be[3];         // p_k = y1 al_k + z1 be_k for the axes b, c, a
    df E[3], Sp[3];          // Earth and Sun in the body frame
    df ibb, icc, i2A, q;     // 1/b^2, 1/c^2, 1/(2A), 2.4/S
    df B1, B2;               // B = y1 B1 + z1 B2
    df d11, d12, d22, d0;    // D = d11 y1^2 + d12 y1 z1 + d22 z1^2 + d0
    float m11, m12, m22, m0; // the magnitudes of the terms that D is the difference of
    float imax, emax, pmax, smax;  // bounds of 1/b^2 and 1/c^2, |E|, |p|, |S| (components, at least 1)
};

__global__ void render_setup_kernel(const double* __restrict__ geo, int n_frames, int S, FrameConst* out)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_frames) return;
    const double* g = geo + (int64_t)kAstGeo * f;
    FrameConst K;
    // Image axes: X1 toward the observer (E), Z1 = [E x y], Y1 = [Z1 x X1] (cuda.c:2418-2427).
    const double Ex = g[2], Ey = g[3], Ez = g[4];
    const double scale = 1.0 / sqrt(A_(M_(Ex, Ex), M_(Ez, Ez)));
    K.Z1x = M_(-Ez, scale);
    K.Z1z = M_(Ex, scale);
    K.Y1x = M_(M_(-Ex, Ey), scale);
    K.Y1y = M_(A_(M_(Ex, Ex), M_(Ez, Ez)), scale);
    K.Y1z = M_(M_(-Ey, Ez), scale);
    // The quadratic's A depends on the frame only (cuda.c:2454).
    const double Epb = g[5], Epc = g[6], Epa = g[7], bb = M_(g[0], g[0]), cc = M_(g[1], g[1]);
    K.A = A_(A_(M_(Epb, Epb) / bb, M_(Epc, Epc) / cc), M_(Epa, Epa));
    ScreenF& F = K.F;
    F.Y1x = (float)K.Y1x; F.Y1y = (float)K.Y1y; F.Y1z = (float)K.Y1z; F.Z1x = (float)K.Z1x; F.Z1z = (float)K.Z1z;
    for (int r = 0; r < 9; r++) F.ax[r] = (float)g[11 + r];
    F.Epb = (float)Epb; F.Epc = (float)Epc; F.Epa = (float)Epa;
    F.ibb = (float)(1.0 / bb); F.icc = (float)(1.0 / cc); F.A = (float)K.A;
    double al[3], be[3], B1 = 0, B2 = 0, c11 = 0, c12 = 0, c22 = 0, a11 = 0, a12 = 0, a22 = 0, b1 = 0, b2 = 0;
    const double w[3] = {1.0 / bb, 1.0 / cc, 1.0}, E[3] = {Epb, Epc, Epa};
    for (int k = 0; k < 3; k++) {
        al[k] = g[11 + 3 * k] * K.Y1x + g[12 + 3 * k] * K.Y1y + g[13 + 3 * k] * K.Y1z;
        be[k] = g[11 + 3 * k] * K.Z1x + g[13 + 3 * k] * K.Z1z;
        K.al[k] = df_from_double(al[k]);
        K.be[k] = df_from_double(be[k]);
        K.E[k] = df_from_double(E[k]);
        K.Sp[k] = df_from_double(g[8 + k]);
        B1 += 2 * al[k] * E[k] * w[k];
        B2 += 2 * be[k] * E[k] * w[k];
        b1 += 2 * fabs(al[k] * E[k]) * w[k];
        b2 += 2 * fabs(be[k] * E[k]) * w[k];
        c11 += al[k] * al[k] * w[k];
        c12 += al[k] * be[k] * w[k];
        c22 += be[k] * be[k] * w[k];
        a12 += fabs(al[k] * be[k]) * w[k];
    }
    const double A4 = 4 * K.A;
    K.B1 = df_from_double(B1);
    K.B2 = df_from_double(B2);
    K.d11 = df_from_double(B1 * B1 - A4 * c11);
    K.d12 = df_from_double(2 * (B1 * B2 - A4 * c12));
    K.d22 = df_from_double(B2 * B2 - A4 * c22);
    K.d0 = df_from_double(A4);
    a11 = b1 * b1 + A4 * c11;
    a12 = 2 * (b1 * b2 + A4 * a12);
    a22 = b2 * b2 + A4 * c22;
    K.m11 = (float)a11;
    K.m12 = (float)a12;
    K.m22 = (float)a22;
    K.m0 = (float)A4;
    K.ibb = df_from_double(w[0]);
    K.icc = df_from_double(w[1]);
    K.i2A = df_from_double(0.5 / K.A);
    K.q = df_from_double(2.4 / S);
    K.imax = (float)fmax(fmax(w[0], w[1]), 1.0);
    K.emax = K.smax = 1.0f;
    double pa = 0, pb = 0;
    for (int k = 0; k < 3; k++) {
        K.emax = fmaxf(K.emax, (float)fabs(E[k]));
        K.smax = fmaxf(K.smax, (float)fabs(g[8 + k]));
        pa = fmax(pa, fabs(al[k]));
        pb = fmax(pb, fabs(be[k]));
    }
    K.pmax = fmaxf(1.0f, (float)(1.2 * (pa + pb)));
    out[f] = K;
}

// A corner's line of sight in double-float, on the FP32 pipe: bit 0 of *flags whether it hits, bit 1 the
// red spot, *I the cosine of the incidence and *e a bound on its distance from the reference's FP64
// value.  False where that value could fall on the other side of one of the reference's tests: D < 0, I <
// 0, the spot's edge, or where the bound is too wide for a colour (grazing lines of sight).  eD covers a
// dozen double-float operations on D's terms (2u^2 = 7e-15 each) and FP64's rounding of them nine times
// over; it passes through sqrt D and the division by 2 A into the point, by 1/b^2 or 1/c^2 into the normal,
// and by its length into I.
__device__ __forceinline__ bool corner_fast(const FrameConst& K, int cz, int cy, int S, df* I, float* e, unsigned* flags)
{
    const df y = df_mul_f(K.q, (float)(cy - S / 2)), z = df_mul_f(K.q, (float)(cz - S / 2));
    const df D = df_add(df_add(df_mul(df_add(df_mul(K.d11, y), df_mul(K.d12, z)), y), df_mul(df_mul(K.d22, z), z)), K.d0);
    const float eD = 1e-12f * (K.m11 * y.hi * y.hi + K.m12 * fabsf(y.hi * z.hi) + K.m22 * z.hi * z.hi + K.m0);
    *I = df{0.0f, 0.0f};
    *e = 0.0f;
    *flags = 0;
    if (D.hi < -4.0f * eD) return true;
    if (!(D.hi > 4.0f * eD)) return false;
    const df sD = df_sqrt(D);
    const df B = df_add(df_mul(K.B1, y), df_mul(K.B2, z));
    const df lam = df_mul(df_sub(sD, B), K.i2A);  // the larger root: A > 0
    df r[3];
#pragma unroll
    for (int k = 0; k < 3; k++)
        r[k] = df_add(df_add(df_mul(K.al[k], y), df_mul(K.be[k], z)), df_mul(lam, K.E[k]));
    const df nb = df_mul(r[0], K.ibb), nc = df_mul(r[1], K.icc), na = r[2];
    const df nn = df_add(df_add(df_mul(nb, nb), df_mul(nc, nc)), df_mul(na, na));
    const df num = df_add(df_add(df_mul(nb, K.Sp[0]), df_mul(nc, K.Sp[1])), df_mul(na, K.Sp[2]));
    const df len = df_sqrt(nn);
    *I = df_div(num, len);
    const float el = (eD / sD.hi + 1e-12f * (sD.hi + fabsf(B.hi))) * K.i2A.hi;
    const float er = el * K.emax + 1e-12f * (K.pmax + fabsf(lam.hi) * K.emax);
    *e = K.smax * (8.0f * er * K.imax / len.hi + 1e-12f);
    const float k2 = kSpotRad * kSpotRad;  // as a float, as the reference squares it
    const df v = df_add_f(df_add(df_mul(r[1], r[1]), df_mul(r[2], r[2])), -k2);
    const bool near_spot = v.hi < 1e-3f;
    if (near_spot && (fabsf(v.hi) < 1e-6f + 8.0f * er || fabsf(r[0].hi) < 1e-6f + 8.0f * er)) return false;
    *flags = v.hi < 0.0f && r[0].hi > 0.0f ? 3u : 1u;
    return *e < 1e-7f && fabsf(I->hi) > 2.0f * *e;
}

// The same in the reference's FP64 expressions (cuda.c:2453-2495).
__device__ __noinline__ double corner_exact(const double* g, const FrameConst& K, int cz, int cy, int S, unsigned* flags)
{
    const double bb = M_(g[0], g[0]), cc = M_(g[1], g[1]), A = K.A;
    const double Epb = g[5], Epc = g[6], Epa = g[7], Spb = g[8], Spc = g[9], Spa = g[10];
    const double z1 = 2.4 * (double)(cz - S / 2) / (double)S;
    const double y1 = 2.4 * (double)(cy - S / 2) / (double)S;
    const double p_x = A_(M_(y1, K.Y1x), M_(z1, K.Z1x));
    const double p_y = A_(M_(y1, K.Y1y), M_(z1, 0.0));
    const double p_z = A_(M_(y1, K.Y1z), M_(z1, K.Z1z));
    const double p_b = A_(A_(M_(g[11], p_x), M_(g[12], p_y)), M_(g[13], p_z));
    const double p_c = A_(A_(M_(g[14], p_x), M_(g[15], p_y)), M_(g[16], p_z));
    const double p_a = A_(A_(M_(g[17], p_x), M_(g[18], p_y)), M_(g[19], p_z));
    // Line of sight p + lambda E' against the ellipsoid (b, c, 1) (cuda.c:2453-2460).
    const double B = M_(2.0, A_(A_(M_(p_b, Epb) / bb, M_(p_c, Epc) / cc), M_(p_a, Epa)));
    const double C = S_(A_(A_(M_(p_b, p_b) / bb, M_(p_c, p_c) / cc), M_(p_a, p_a)), 1.0);
    const double D = S_(M_(B, B), M_(M_(4.0, A), C));
    *flags = 0;
    if (!(D >= 0.0)) return 0.0;
    const double sD = sqrt(D);
    double lambda = S_(-B, sD) / M_(2.0, A);
    const double lambda1 = A_(-B, sD) / M_(2.0, A);
    if (lambda1 > lambda) lambda = lambda1;
    const double ri_b = A_(p_b, M_(lambda, Epb));
    const double ri_c = A_(p_c, M_(lambda, Epc));
    const double ri_a = A_(p_a, M_(lambda, Epa));
    const bool red_spot = A_(M_(ri_c, ri_c), M_(ri_a, ri_a)) < (double)(kSpotRad * kSpotRad) && ri_b > 0.0;
    double ni_b = ri_b / bb, ni_c = ri_c / cc, ni_a = ri_a;
    const double scale = 1.0 / sqrt(A_(A_(M_(ni_b, ni_b), M_(ni_c, ni_c)), M_(ni_a, ni_a)));
    ni_b = M_(ni_b, scale);
    ni_c = M_(ni_c, scale);
    ni_a = M_(ni_a, scale);
    *flags = red_spot ? 3u : 1u;
    return A_(A_(M_(ni_b, Spb), M_(ni_c, Spc)), M_(ni_a, Spa));
}

// One corner's contribution to a channel: float + float + double * float, rounded back to float
// (cuda.c:2500-2525).
__device__ __forceinline__ float add_exact(float br, float base, double I, float range)
{
    return (float)A_((double)(br + base), M_(I, (double)range));
}
// The same from I as a double-float within e of it; *sure becomes false where the float it rounds to could
// be the next one.
__device__ __forceinline__ float add_fast(float br, float base, df I, float range, float e, bool* sure)
{
    const df s = df_add_f(df_mul_f(I, range), __fadd_rn(br, base));
    const float d = __fmaf_rn(e, fabsf(range), 1e-10f);
    if (__fadd_rn(s.hi, __fadd_rn(s.lo, d)) != s.hi || __fadd_rn(s.hi, __fadd_rn(s.lo, -d)) != s.hi) *sure = false;
    return s.hi;
}

__device__ __forceinline__ uint8_t channel(float br)
{
    const int v = (int)((double)br / 4.0);
    return (uint8_t)(v > 255 ? 255 : (v < 0 ? 0 : v));
}

// One CTA shades a kTileX x kTileY tile of one frame.  The four corners of a pixel are shared with its
// neighbours, so the CTA evaluates the (kTileX+1) x (kTileY+1) corner lines of sight of its tile once
// each (hit, red spot, I), then every thread accumulates its pixel's four corners in the reference's
// order (jz outer, jy inner) -- the same values, combined in the same float steps, as four evaluations
// per pixel would give.
//
// In the reference's FP64 a corner is 200 instructions and a lit pixel 70, at 16 cycles of the SM's FP64
// unit each; the frame's bytes need them only where a value falls within its error of a decision.  So the
// corners that the float pre-test leaves are evaluated in double-float with an error bound
// (corner_fast), the pixels from those, and what remains undecided -- grazing lines of sight, the edges
// of the shadow and of the spot within 1e-6, a channel within 5e-4 of the next byte whose float roundings
// are not certain -- is listed and takes the FP64 expressions.  24 frames of 1080^2: 4.86 ms in FP64.
__global__ void __launch_bounds__(kRenderTpb, 3) render_kernel(const double* __restrict__ geo,
                                                            const FrameConst* __restrict__ frames, int n_frames, int S,
                                                            uint8_t* __restrict__ rgb)
{
    __shared__ FrameConst K;
    __shared__ float cIh[kCorners], cIl[kCorners], cE[kCorners];
    __shared__ uint8_t cF[kCorners];  // bit 0: the line of sight hits the ellipsoid; bit 1: red spot
    __shared__ int16_t todo[kCorners], hard[kCorners];  // corners left by the pre-test, and by corner_fast
    __shared__ int n_todo, n_hard, n_pixels;
    const int f = blockIdx.y;
    const double* g = geo + (int64_t)kAstGeo * f;
    const int tiles_x = (S + kTileX - 1) / kTileX;
    const int y0 = (blockIdx.x % tiles_x) * kTileX;  // first pixel column (iy) of the tile
    const int z0 = (blockIdx.x / tiles_x) * kTileY;  // first pixel row (iz)
    for (int k = threadIdx.x; k < (int)(sizeof(FrameConst) / 4); k += kRenderTpb)
        reinterpret_cast<uint32_t*>(&K)[k] = reinterpret_cast<const uint32_t*>(&frames[f])[k];
    if (threadIdx.x == 0) n_todo = n_hard = n_pixels = 0;
    __syncthreads();
    // Pass 1: the float pre-test of every corner; the undecided ones are listed, so that the lines of sight
    // clustered on the asteroid's disc keep whole warps busy.
    for (int k = threadIdx.x; k < kCorners; k += kRenderTpb) {
        const int cz = z0 + k / (kTileX + 1), cy = y0 + k % (kTileX + 1);  // corner (iz + jz, iy + jy)
        if (screen_background(K.F, cz, cy, S)) cF[k] = 0;
        else todo[atomicAdd(&n_todo, 1)] = (int16_t)k;
    }
    __syncthreads();
    // Pass 2: the listed corners in double-float, what that leaves undecided in FP64.
    for (int i = threadIdx.x; i < n_todo; i += kRenderTpb) {
        const int k = todo[i];
        df I;
        float e;
        unsigned fl;
        if (!corner_fast(K, z0 + k / (kTileX + 1), y0 + k % (kTileX + 1), S, &I, &e, &fl))
            hard[atomicAdd(&n_hard, 1)] = (int16_t)k;
        cIh[k] = I.hi;
        cIl[k] = I.lo;
        cE[k] = e;
        cF[k] = (uint8_t)fl;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_hard; i += kRenderTpb) {
        const int k = hard[i];
        unsigned fl;
        const double I = corner_exact(g, K, z0 + k / (kTileX + 1), y0 + k % (kTileX + 1), S, &fl);
        const df d = df_from_double(I);
        cIh[k] = d.hi;
        // The sign decides a branch: a value too small for a float keeps it.
        cIl[k] = d.lo;
        if (d.hi == 0.0f && I < 0.0) cIh[k] = -1e-38f;
        cE[k] = 1e-14f;
        cF[k] = (uint8_t)fl;
    }
    __syncthreads();
    // Pass 3: the pixels; the undecided ones are listed (over the corners' lists).
    const int ty = threadIdx.x % kTileX, tz = threadIdx.x / kTileX;
    const int iy = y0 + ty, iz = z0 + tz;
    if (iy < S && iz < S) {
        float br[3] = {0.f, 0.f, 0.f};
        bool sure = true;
#pragma unroll
        for (int jz = 0; jz < 2; jz++)
#pragma unroll
            for (int jy = 0; jy < 2; jy++) {
                const int k = (tz + jz) * (kTileX + 1) + ty + jy;
                const uint8_t fl = cF[k];
                if (!(fl & 1)) continue;
                const df I{cIh[k], cIl[k]};
                const float e = cE[k];
                const bool red_spot = (fl & 2) != 0;
                if (I.hi >= 0.0f) {
                    br[0] = add_fast(br[0], kSmaxR, I, kImaxR - kSmaxR, e, &sure);
                    if (!red_spot) {
                        br[1] = add_fast(br[1], kSmaxG, I, kImaxG - kSmaxG, e, &sure);
                        br[2] = add_fast(br[2], kSmaxB, I, kImaxB - kSmaxB, e, &sure);
                    }
                } else {
                    br[0] = add_fast(br[0], kSmaxR, I, kSmaxR - kSminR, e, &sure);
                    if (!red_spot) {
                        br[1] = add_fast(br[1], kSmaxG, I, kSmaxG - kSminG, e, &sure);
                        // The reference adds to br[1] here, not br[2] (cuda.c:2523).
                        br[2] = add_fast(br[1], kSmaxB, I, kSmaxB - kSminB, e, &sure);
                    }
                }
            }
        // Uncertain roundings move a channel by an ulp or two (6e-5 each) of at most 1020.
        bool decided = sure;
        if (!sure) {
            decided = true;
#pragma unroll
            for (int ic = 0; ic < 3; ic++) {
                const float v = 0.25f * br[ic];
                if (fabsf(v - rintf(v)) < 5e-4f) decided = false;
            }
        }
        if (decided) {
            uint8_t* out = rgb + 3 * ((int64_t)iy + (int64_t)S * ((int64_t)iz + (int64_t)S * f));
#pragma unroll
            for (int ic = 0; ic < 3; ic++) out[ic] = channel(br[ic]);
        } else {
            todo[atomicAdd(&n_pixels, 1)] = (int16_t)threadIdx.x;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n_pixels; i += kRenderTpb) {
        const int px = todo[i] % kTileX, pz = todo[i] / kTileX;
        float br[3] = {0.f, 0.f, 0.f};
        for (int j = 0; j < 4; j++) {
            unsigned fl;
            const double I = corner_exact(g, K, z0 + pz + j / 2, y0 + px + j % 2, S, &fl);
            if (!(fl & 1)) continue;
            const bool red_spot = (fl & 2) != 0;
            if (I >= 0.0) {
                br[0] = add_exact(br[0], kSmaxR, I, kImaxR - kSmaxR);
                if (!red_spot) {
                    br[1] = add_exact(br[1], kSmaxG, I, kImaxG - kSmaxG);
                    br[2] = add_exact(br[2], kSmaxB, I, kImaxB - kSmaxB);
                }
            } else {
                br[0] = add_exact(br[0], kSmaxR, I, kSmaxR - kSminR);
                if (!red_spot) {
                    br[1] = add_exact(br[1], kSmaxG, I, kSmaxG - kSminG);
                    br[2] = add_exact(br[1], kSmaxB, I, kSmaxB - kSminB);
                }
            }
        }
        uint8_t* out = rgb + 3 * ((int64_t)(y0 + px) + (int64_t)S * ((int64_t)(z0 + pz) + (int64_t)S * f));
        for (int ic = 0; ic < 3; ic++) out[ic] = channel(br[ic]);
    }
}

#undef M_
#undef A_
#undef S_

struct RenderScratch {
    double* geo = nullptr;
    FrameConst* frames = nullptr;
    uint8_t* rgb = nullptr;
    cudaStream_t s = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ~RenderScratch()
    {
        cudaFree(geo);
        cudaFree(frames);
        cudaFree(rgb);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        if (s) cudaStreamDestroy(s);
    }
};

}  // namespace
}  // namespace ast

using namespace ast;

extern "C" int ast_render_frames(int32_t device, const double* geo, int32_t n_frames, int32_t size_pix, uint8_t* rgb,
                                 double* kernel_ms)
{
    if (!geo || !rgb || n_frames < 0 || size_pix < 2 || size_pix > 8192 || (size_pix & 1))
        return ast_set_error(AST_E_INVALID, "ast_render_frames: bad argument");
    if (kernel_ms) *kernel_ms = 0;
    if (n_frames == 0) return AST_OK;
    int rc = set_device(device);
    if (rc) return rc;
    const int64_t frame_bytes = 3ll * size_pix * size_pix;
    // Frames per launch: at most 2 GB of pixels on the device at once (the reference uses dNPLOT),
    // and at most 65 535 (the grid's y dimension).
    const int64_t chunk =
        std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(n_frames, 65535), (2ll << 30) / frame_bytes));
    RenderScratch d;
    if (cudaMalloc(&d.geo, sizeof(double) * kAstGeo * chunk) != cudaSuccess ||
        cudaMalloc(&d.frames, sizeof(FrameConst) * chunk) != cudaSuccess ||
        cudaMalloc(&d.rgb, (size_t)(frame_bytes * chunk)) != cudaSuccess) {
        cudaGetLastError();
        return ast_set_error(AST_E_NOMEM, "ast_render_frames: cudaMalloc failed");
    }
    AST_CUDA(cudaStreamCreateWithFlags(&d.s, cudaStreamNonBlocking));
    AST_CUDA(cudaEventCreate(&d.e0));
    AST_CUDA(cudaEventCreate(&d.e1));
    const unsigned blocks = (unsigned)(((size_pix + kTileX - 1) / kTileX) * ((size_pix + kTileY - 1) / kTileY));
    double total = 0;
    for (int64_t f0 = 0; f0 < n_frames; f0 += chunk) {
        const int64_t nf = std::min<int64_t>(chunk, n_frames - f0);
        AST_CUDA(cudaMemcpyAsync(d.geo, geo + kAstGeo * f0, sizeof(double) * kAstGeo * nf, cudaMemcpyHostToDevice, d.s));
        AST_CUDA(cudaEventRecord(d.e0, d.s));
        render_setup_kernel<<<(unsigned)((nf + 31) / 32), 32, 0, d.s>>>(d.geo, (int)nf, size_pix, d.frames);
        AST_CUDA(cudaGetLastError());
        render_kernel<<<dim3(blocks, (unsigned)nf), kRenderTpb, 0, d.s>>>(d.geo, d.frames, (int)nf, size_pix, d.rgb);
        AST_CUDA(cudaGetLastError());
        AST_CUDA(cudaEventRecord(d.e1, d.s));
        AST_CUDA(cudaMemcpyAsync(rgb + frame_bytes * f0, d.rgb, (size_t)(frame_bytes * nf), cudaMemcpyDeviceToHost, d.s));
        AST_CUDA(cudaStreamSynchronize(d.s));
        float ms = 0;
        AST_CUDA(cudaEventElapsedTime(&ms, d.e0, d.e1));
        total += ms;
    }
    if (kernel_ms) *kernel_ms = total;
    return AST_OK;
}
