"""tests/test_trig64.py's bounds on the GPU, where an FP64 evaluation gets its sines, quotients and magnitudes: the
seeds come from the special function unit there, and products and sums are contracted."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from asteroid_gb300 import build
from tests.test_trig64 import (ROOT, mpmath, test_beyond, test_magnitude, test_magnitude_at_the_ends,  # noqa: F401
                               test_quotients, test_reciprocals, test_sincos)

pytestmark = pytest.mark.gpu


class _Device:
    """The device harness by the host harness's calls."""

    def __init__(self, lib):
        self.lib = lib

    def call(self, name, n, x, out):
        rc = getattr(self.lib, name)(n, x, out)
        assert rc == 0, f"{name}: CUDA error {rc}"

    def h_sincos_tab(self, n, x, out):
        self.call("h_sincos_tab", n, x, out)

    def h_ls_algebraic(self, n, v, out):
        self.call("h_ls_algebraic", n, v, out)

    def h_recip(self, n, s, out):
        self.call("h_recip", n, s, out)

    def h_quotients(self, n, u, s, out):
        us = np.concatenate([np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_double)), (n,)) for p in (u, s)])
        self.call("h_quotients_us", n, us.ctypes.data_as(C.c_void_p), out)


@pytest.fixture(scope="module")
def lib(gpu, tmp_path_factory):
    out = tmp_path_factory.mktemp("trig64") / "libtrig64_device.so"
    subprocess.run([build._nvcc(), *build.GENCODE, "-shared", "-O3", "-std=c++17", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    f"-I{build.PKG / 'csrc'}", f"-I{build.INCLUDE}", str(ROOT / "tests" / "host" / "trig64_device.cu"),
                    "-o", str(out), "-lcudart"], check=True, capture_output=True)
    return _Device(C.CDLL(str(out)))


@pytest.fixture(scope="module")
def sincos(lib):
    def run(x):
        x = np.ascontiguousarray(x, np.float64)
        r = np.empty((len(x), 2))
        lib.h_sincos_tab(len(x), x.ctypes.data_as(C.c_void_p), r.ctypes.data_as(C.c_void_p))
        return r

    return run


def test_seeds(lib):
    """Within 2^-20: the instructions read and write the upper 32 bits of a double, 20 of its significand.  An error
    of two units of that, one of the operand's and one of the result's, leaves quot's cubic step e^3 < 2^-57."""
    rng = np.random.default_rng(3)
    x = rng.choice([-1.0, 1.0], 40000) * rng.uniform(1, 2, 40000) * 2.0 ** rng.integers(-300, 300, 40000)
    x[:4] = 1.0, np.nextafter(2.0, 0), np.nextafter(1.0, 2), -2.0
    out = np.empty((len(x), 2))
    lib.call("h_seeds", len(x), x.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    e = np.abs(np.stack([out[:, 0] * x - 1, out[:, 1] * np.sqrt(np.abs(x)) - 1]))
    print(f"seeds: reciprocal {np.log2(e[0].max()):.2f}, root {np.log2(e[1].max()):.2f} (log2)")
    assert e.max() <= 2.0 ** -19
