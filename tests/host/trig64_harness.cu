// Host build of the FP64 table sine and cosine (csrc/trig64.cuh) and of the evaluation kernels'
// Lommel-Seeliger magnitude (csrc/model.cuh) for the CPU tests.
#include "model.cuh"

extern "C" void h_sincos_tab(int n, const double* x, double* out)
{
    for (int i = 0; i < n; i++) ast::sincos_tab(x[i], out + 2 * i, out + 2 * i + 1);
}

// v: b, c, the vectors to the Sun and the Earth in the body frame (b, c, a).
extern "C" void h_ls_algebraic(int n, const double* v, double* out)
{
    for (int i = 0; i < n; i++, v += 8)
        out[i] = ast::ls_algebraic(v[0], v[1], 1.0 / (v[0] * v[0]), 1.0 / (v[1] * v[1]), v[2], v[3], v[4], v[5], v[6], v[7]);
}

// out: u[i] / s[i], 1 / sqrt(|s[i]|).
extern "C" void h_quotients(int n, const double* u, const double* s, double* out)
{
    for (int i = 0; i < n; i++) {
        out[2 * i] = ast::quot(u[i], s[i]);
        out[2 * i + 1] = ast::inv_sqrt(fabs(s[i]));
    }
}

// out: 1 / s[i].
extern "C" void h_recip(int n, const double* s, double* out)
{
    for (int i = 0; i < n; i++) out[i] = ast::recip(s[i]);
}
