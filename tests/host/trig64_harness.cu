// Host build of the FP64 table sine and cosine (csrc/trig64.cuh) for the CPU tests.
#include "trig64.cuh"

extern "C" void h_sincos_tab(int n, const double* x, double* out)
{
    for (int i = 0; i < n; i++) ast::sincos_tab(x[i], out + 2 * i, out + 2 * i + 1);
}
