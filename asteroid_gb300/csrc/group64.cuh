// group64.cuh -- the FP64 chi^2 of one parameter vector by a group of lanes.
//
// GB300's FP64 unit takes one instruction of a warp every 64 cycles, whatever its dependencies and
// however many of its lanes are active, and with four warps on an SM one every 19 cycles (measured,
// FMA chains of 1 to 8 independent operations, 1 to 32 active lanes).  So an evaluation that has
// its warp to itself takes the number of its FP64 instructions times 64 cycles, and spreading its
// components over idle lanes divides that number: eight lanes hold the six components of the state,
// one stage's two sines and two cosines are one call, its products two instructions, its update one; the
// magnitudes of G observations, one on each lane of the group, are one evaluation.  95 instructions
// an RK4 step and 267 / G + 2 an observation, against 252 and 267 on one lane (torque, evaluations; 159
// and 467 against 340 and 467 in the simplex search, trig64.cuh).
//
// Every operation is the thread path's (chi2_fp64) on the same operands, sums in observation order,
// so the results are its results bit for bit.  All 32 lanes of the warp call together, each group
// with its own parameters, on the same observations.
#pragma once
#include "model.cuh"

namespace ast {

__device__ __forceinline__ double shfl8(double v, int src) { return __shfl_sync(0xffffffffu, v, src, 8); }

// Derivative of the lane's component at the stage value f of every lane: roles 0..2 the angular
// velocity (mu_a = mu[role], mu_b = mu[3 + role]), 3 phi, 4 theta, 5 to 7 psi.
template <class TRIG>
__device__ __forceinline__ double group_rhs_torque(int role, double f, double mu_a, double mu_b)
{
    const double th = shfl8(f, 4), ps = shfl8(f, 5);
    const double v = TRIG::sin_or_cos(role & 1 ? ps : th, role & 2);
    const double s4 = shfl8(v, 0), s5 = shfl8(v, 1), c4 = shfl8(v, 2), c5 = shfl8(v, 3);
    const double y0 = shfl8(f, 0), y1 = shfl8(f, 1), y2 = shfl8(f, 2);
    // mu_a y' y'' + mu_b; (phi's numerator) y0 s5 + y1 c5; (theta) y0 c5 - y1 s5
    const double p = role < 3 ? mu_a : y1;
    const double q = role == 0 ? y1 : role == 1 ? y2 : role == 2 ? y0 : role == 3 ? c5 : s5;
    const double t = p * q;
    const double x = role < 3 ? t : y0;
    const double y = role == 0 ? y2 : role == 1 ? y0 : role == 2 ? y1 : role == 3 ? s5 : c5;
    const double z = role < 3 ? mu_b : role == 3 ? t : -t;
    const double r = x * y + z;
    const double f3 = TRIG::div(shfl8(r, 3), s4);
    const double f5 = y2 - f3 * c4;
    return role == 3 ? f3 : role >= 5 ? f5 : r;
}

// Free rotation: roles 3 phi, 4 theta, others psi; mu_a = mu[0] mu[2].  LAST: the step's fourth
// derivative.  Every derivative is the one product that it is in ode_free, and phi's enters psi's as
// it does there -- as a value of its own in the first three stages, in a fused multiply-add in the
// last, where nothing but the step's sum needs it beside (the compiler's choice there; the tests
// compare the two paths bit for bit).
template <bool LAST, class TRIG>
__device__ __forceinline__ double group_rhs_free(int role, double f, const double* mu, double mu_a)
{
    const double th = shfl8(f, 4), ps = shfl8(f, 5);
    const double v = TRIG::sin_or_cos(role & 1 ? 2.0 * ps : th, role & 2);
    const double s1 = shfl8(v, 0), s2 = shfl8(v, 1), c1 = shfl8(v, 2), c2 = shfl8(v, 3);
    // (phi) mu1 - mu2 c2; (theta) mu0 mu2 s1, whose sum with -0 is itself
    const double x = role == 4 ? mu_a : -mu[2];
    const double y = role == 4 ? s1 : c2;
    const double z = role == 4 ? -0.0 : mu[1];
    const double t = x * y + z;
    const double t3 = shfl8(t, 3);
    const double d = LAST ? mu[0] - mu[0] * t3 : mu[0] - __dmul_rn(mu[0], t3);
    const double a = role == 3 ? mu[0] : role == 4 ? t : c1;
    const double b = role == 3 ? t3 : role == 4 ? s2 : d;
    return a * b;
}

// One RK4 step of the lane's component (rk4_step).
template <bool TORQUE, class TRIG>
__device__ __forceinline__ double group_step(int role, double y, double h, const double* mu, double mu_a, double mu_b)
{
    auto rhs = [&](double f) {
        return TORQUE ? group_rhs_torque<TRIG>(role, f, mu_a, mu_b) : group_rhs_free<false, TRIG>(role, f, mu, mu_a);
    };
    const double K1 = rhs(y);
    const double K2 = rhs(y + 0.5 * h * K1);
    const double K3 = rhs(y + 0.5 * h * K2);
    const double K4 = TORQUE ? rhs(y + h * K3) : group_rhs_free<true, TRIG>(role, y + h * K3, mu, mu_a);
    return y + 1 / 6.0 * h * (K1 + 2 * K2 + 2 * K3 + K4);
}

// chi2_fp64 by the G lanes of a group (8 or 32; 32 lanes integrate in four equal eighths); the result
// and delta_V on every lane.  vmod_out, when non-null, receives the model magnitude of every
// observation (the reference's Nplot > 0 mode, cuda.c:699-704, without the delta_V shift); ang_out
// the Euler angles (phi, theta, psi); geo_out the renderer's geometry.
template <class CF, int G, class TRIG>
__device__ CF chi2_fp64_group(const DevModel& M, const ObsView& o, const double* params, CF* delta_V,
                              double* vmod_out = nullptr, double* ang_out = nullptr, double* geo_out = nullptr)
{
    static_assert(G == 8 || G == 32, "a state takes eight lanes");
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & (G - 1), role = threadIdx.x & 7;
    const int N_data = M.n_data, N_filters = M.n_filters;
    const bool nudge = (M.flags & AST_NUDGE) != 0;
    Fp64Setup S;
    fp64_setup(M, params, S);
    double y, mu_a, mu_b = 0.0;
    if (S.torque) {
        const int k = role < 6 ? role : 5;
        y = k == 0 ? S.y[0] : k == 1 ? S.y[1] : k == 2 ? S.y[2] : k == 3 ? S.y[3] : k == 4 ? S.y[4] : S.y[5];
        mu_a = role == 0 ? S.mu[0] : role == 1 ? S.mu[1] : S.mu[2];
        mu_b = role == 0 ? S.mu[3] : role == 1 ? S.mu[4] : S.mu[5];
    } else {
        y = role == 3 ? S.y[0] : role == 4 ? S.y[1] : S.y[2];
        mu_a = S.mu[0] * S.mu[2];
    }
    double phi = 0.0, theta = 0.0, psi = 0.0;  // of the lane's observation of the tile
    double sum_y2 = 0.0, sum_y = 0.0;          // of filter `lane`
    Fp64Minima Q;
    bool huge = false;
    for (int i = 0; i < N_data; i++) {
        if (i > 0) {
            const int N_steps = o.nst[i];
            const double h = o.h[i];
            if (S.torque) {
#pragma unroll 1
                for (int l = 0; l < N_steps; l++) y = group_step<true, TRIG>(role, y, h, S.mu, mu_a, mu_b);
            } else {
#pragma unroll 1
                for (int l = 0; l < N_steps; l++) y = group_step<false, TRIG>(role, y, h, S.mu, mu_a, mu_b);
            }
        }
        {
            const double a = shfl8(y, 3), b = shfl8(y, 4), c = shfl8(y, 5);
            if ((i & (G - 1)) == lane) {
                phi = a;
                theta = b;
                psi = c;
            }
        }
        if ((i & (G - 1)) != G - 1 && i != N_data - 1) continue;
        // The tile's magnitudes, one observation a lane.
        const int i0 = i & ~(G - 1), n = i - i0 + 1;
        const bool own = lane < n;
        const int k = own ? i0 + lane : i;
        const double Vmod = fp64_vmod<TRIG>(M, params, S, phi, theta, psi, o, k,
                                      geo_out && own ? geo_out + (int64_t)kAstGeo * k : nullptr);
        if (own && vmod_out) vmod_out[k] = Vmod;
        if (own && ang_out) {
            ang_out[3 * k] = phi;
            ang_out[3 * k + 1] = theta;
            ang_out[3 * k + 2] = psi;
        }
        // Per-filter sums in observation order (cuda.c:707-714), a filter a lane.
        const double yv = o.v[k] - Vmod, yv2 = yv * yv, w = o.w[k];
        const int f = o.f[k];
        for (int j = 0; j < n; j++) {
            const double aj = __shfl_sync(kAll, yv2, j, G), yj = __shfl_sync(kAll, yv, j, G),
                         wj = __shfl_sync(kAll, w, j, G);
            if (__shfl_sync(kAll, f, j, G) == lane) {
                sum_y2 = sum_y2 + aj * wj;
                sum_y = sum_y + yj * wj;
            }
        }
        if (nudge)
            for (int j = 0; j < n; j++) {
                const double Vj = __shfl_sync(kAll, Vmod, j, G);
                if (!huge && !fp64_minima(M, Q, i0 + j, o.t[i0 + j], Vj)) huge = true;
            }
    }
    double s2[AST_MAX_FILTERS], s1[AST_MAX_FILTERS];
    for (int m = 0; m < N_filters; m++) {
        s2[m] = __shfl_sync(kAll, sum_y2, m, G);
        s1[m] = __shfl_sync(kAll, sum_y, m, G);
    }
    if (huge) return (CF)kHuge;
    return fp64_finish<CF>(M, s2, s1, o.sum_w, Q, delta_V);
}

}  // namespace ast
