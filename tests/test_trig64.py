"""The FP64 table sine and cosine (csrc/trig64.cuh), compiled for the host, against mpmath."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from asteroid_gb300 import build

mpmath = pytest.importorskip("mpmath")
ROOT = Path(__file__).resolve().parents[1]
STEP = 2 * np.pi / 1024


@pytest.fixture(scope="module")
def sincos(tmp_path_factory):
    out = tmp_path_factory.mktemp("trig64") / "libtrig64_harness.so"
    subprocess.run([build._nvcc(), "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-O2", "-std=c++17",
                    f"-I{build.PKG / 'csrc'}", f"-I{build.INCLUDE}", str(ROOT / "tests" / "host" / "trig64_harness.cu"),
                    "-o", str(out)], check=True, capture_output=True)
    lib = C.CDLL(str(out))

    def run(x):
        x = np.ascontiguousarray(x, np.float64)
        r = np.empty((len(x), 2))
        lib.h_sincos_tab(len(x), x.ctypes.data_as(C.c_void_p), r.ctypes.data_as(C.c_void_p))
        return r

    return run


# Every table point, the middles between them (either neighbour), one turn and many, and the zeros.
@pytest.mark.parametrize("x", [
    np.arange(-1100, 1100) * STEP, (np.arange(-1100, 1100) + 0.5) * STEP, (np.arange(1024) + 0.5) * STEP * (1 - 1e-16),
    np.arange(-50, 50) * np.pi / 2, np.geomspace(1e-300, 3.0, 400), -np.geomspace(3.0, 2.0 ** 40 - 1, 400), np.array([0.0, -0.0]),
], ids=["points", "middles", "below_middles", "zeros", "small", "large", "zero"])
def test_sincos(sincos, x):
    r = sincos(x)
    with mpmath.workprec(200):
        for xi, (s, c) in zip(x, r):
            for got, want in ((s, mpmath.sin(mpmath.mpf(float(xi)))), (c, mpmath.cos(mpmath.mpf(float(xi))))):
                # The last sum's rounding; the remainder's and the inner sum's, 2^-62 each, the remainder's sine's,
                # and cos r cut before r^6/720 -- none of the last four where the remainder is x itself.
                tol = 0.5 * np.spacing(abs(float(want)))
                tol += 3 * 2.0 ** -62 + 1.2e-18 if abs(xi) > STEP / 2 else 0.01 * np.spacing(abs(float(want)))
                assert abs(mpmath.mpf(float(got)) - want) <= tol, float(xi)


def test_beyond(sincos):
    x = np.array([2.0 ** 40, -1e15, 1e300, np.inf, -np.inf, np.nan])
    r = sincos(x)
    with np.errstate(invalid="ignore"):
        np.testing.assert_allclose(r, np.stack([np.sin(x), np.cos(x)], 1), rtol=0, atol=2.3e-16)
