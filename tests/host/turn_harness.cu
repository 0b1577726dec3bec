// Host build of the compact-angle RK4 step (csrc/turn.cuh) for the CPU tests (compiled without
// floating-point contraction, as mixed_harness.cu).
#include <vector>
#include "mixed.cuh"
#include "prep.cuh"

using namespace ast;

namespace {
std::vector<float4> table()
{
    std::vector<float4> t(kTrigTable);
    for (int k = 0; k < kTrigTable; k++) t[k] = trig_table_entry(k);
    return t;
}
}  // namespace

extern "C" {

// sin and cos of the compact angles (k[2i + l] + e + t) 2pi/T: out[8i + 4l] = sin hi, lo, cos hi, lo.
void h_turn_sincos(int n, const int* k, const float* e, const float* t, float* out)
{
    const std::vector<float4> tab = table();
    for (int i = 0; i < n; i++) {
        df2 s, c;
        turn_sincos2(Turn2{4u * (uint32_t)k[2 * i], 4u * (uint32_t)k[2 * i + 1], make_float2(e[2 * i], e[2 * i + 1]),
                           make_float2(t[2 * i], t[2 * i + 1])},
                     reinterpret_cast<const float*>(tab.data() + kTrigPoints), &s, &c);
        const float v[8] = {s.hi.x, s.lo.x, c.hi.x, c.lo.x, s.hi.y, s.lo.y, c.hi.y, c.lo.y};
        for (int j = 0; j < 8; j++) out[8 * i + j] = v[j];
    }
}

// Angle in radians -> compact -> radians, reduced to [-pi, pi].
double h_turn_round_trip(double a, int turns)
{
    const Turn u = turn_from(df_from_double(a), turns);
    return df_to_double(turn_value(u.k, u.e, u.t, turns)) / turns;
}

// n steps of size h from y = (w0, w1, w2, phi, theta, psi), mu as the ODE's (torque 6, free 3), through
// mixed_advance.  The state comes back in place, angles in [-pi, pi].
void h_turn_steps(int torque, int n, double h, const double* mu, double* y)
{
    const std::vector<float4> tab = table();
    MixedState S;
    S.torque = torque != 0;
    S.bw = false;
    for (int k = 0; k < (torque ? 6 : 3); k++) {
        S.mu[k] = df_from_double(mu[k]);
        S.y[k] = df_from_double(torque ? y[k] : y[3 + k]);
    }
    mixed_begin(S);
    const df H = df_from_double(h), H6 = df_from_double(h / 6.0), Q = df_from_double(h / kTurnStep),
             C6 = df_from_double(kTurnStep / (6.0 * h));
    const int nst[2] = {0, n};
    const float4 hq[2] = {{}, {H.hi, H.lo, Q.hi, Q.lo}}, hw[2] = {{}, {H6.hi, H6.lo, C6.hi, C6.lo}};
    ObsView o = {};
    o.nst = nst;
    o.hq = hq;
    o.hw = hw;
    df a[3];
    mixed_advance<false>(S, o, 1, tab.data(), a);
    for (int k = 0; k < 3; k++) {
        if (torque) y[k] = df_to_double(S.s.w[k]) + (double)S.s.r[k];
        y[3 + k] = df_to_double(a[k]);
    }
}

// One step of the general step alone (spin_step_general).
void h_general_step(int torque, double h, const double* mu, double* y)
{
    const std::vector<float4> tab = table();
    MixedState S;
    S.torque = torque != 0;
    S.bw = false;
    for (int k = 0; k < (torque ? 6 : 3); k++) {
        S.mu[k] = df_from_double(mu[k]);
        S.y[k] = df_from_double(torque ? y[k] : y[3 + k]);
    }
    mixed_begin(S);
    const df H = df_from_double(h), H6 = df_from_double(h / 6.0), Q = df_from_double(h / kTurnStep),
             C6 = df_from_double(kTurnStep / (6.0 * h));
    spin_step_beyond(S, float4{H.hi, H.lo, Q.hi, Q.lo}, float4{H6.hi, H6.lo, C6.hi, C6.lo}, tab.data());
    df a[3];
    spin_angles(S.s, S.torque, a);
    for (int k = 0; k < 3; k++) {
        if (torque) y[k] = df_to_double(S.s.w[k]) + (double)S.s.r[k];
        y[3 + k] = df_to_double(a[k]);
    }
}

// From y at time 0 to time t, with the step constants of prep_obs_point.
void h_turn_interval(int torque, double t, double time_step, const double* mu, double* y)
{
    const std::vector<float4> tab = table();
    const ObsLayout L = ObsLayout::make(2);
    std::vector<char> block((size_t)L.bytes + 256);
    char* base = block.data() + (256 - (uintptr_t)block.data() % 256);
    DevModel M{};
    M.time_step = time_step;
    M.n_data = 2;
    ((double*)(base + L.off_t))[1] = t;
    for (int i = 0; i < 2; i++) prep_obs_point(M, base, L, 2, i);
    const ObsView o = L.view(base, 2);
    MixedState S;
    S.torque = torque != 0;
    S.bw = false;
    for (int k = 0; k < (torque ? 6 : 3); k++) {
        S.mu[k] = df_from_double(mu[k]);
        S.y[k] = df_from_double(torque ? y[k] : y[3 + k]);
    }
    mixed_begin(S);
    df a[3];
    mixed_advance<false>(S, o, 1, tab.data(), a);
    for (int k = 0; k < 3; k++) {
        if (torque) y[k] = df_to_double(S.s.w[k]) + (double)S.s.r[k];
        y[3 + k] = df_to_double(a[k]);
    }
}

}  // extern "C"
