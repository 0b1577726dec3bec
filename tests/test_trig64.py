"""The FP64 table sine and cosine (csrc/trig64.cuh) and the evaluation kernels' Lommel-Seeliger
magnitude (csrc/model.cuh), compiled for the host, against mpmath."""
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
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("trig64") / "libtrig64_harness.so"
    subprocess.run([build._nvcc(), "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-O2", "-std=c++17",
                    f"-I{build.PKG / 'csrc'}", f"-I{build.INCLUDE}", str(ROOT / "tests" / "host" / "trig64_harness.cu"),
                    "-o", str(out)], check=True, capture_output=True)
    return C.CDLL(str(out))


@pytest.fixture(scope="module")
def sincos(lib):
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


# The seeds' whole range of significands, both signs, over many binades (within a float's on the host).
def test_quotients(lib):
    rng = np.random.default_rng(7)
    n = 4000
    s = rng.choice([-1.0, 1.0], n) * rng.uniform(1, 2, n) * 2.0 ** rng.integers(-100, 100, n)
    s[:4] = 1.0, np.nextafter(2.0, 0), np.nextafter(1.0, 2), -2.0
    u = rng.normal(size=n) * 2.0 ** rng.integers(-100, 100, n)
    u[:2] = 0.0, -1.0
    out = np.empty((n, 2))
    lib.h_quotients(n, u.ctypes.data_as(C.c_void_p), s.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    with mpmath.workprec(200):
        for ui, si, (q, r) in zip(u, s, out):
            want = mpmath.mpf(float(ui)) / mpmath.mpf(float(si))
            assert abs(mpmath.mpf(float(q)) - want) <= 0.501 * np.spacing(abs(float(want)))
            want = 1 / mpmath.sqrt(abs(mpmath.mpf(float(si))))
            # e's own error, one rounding of x y (2^-53), enters by half; the last sum's rounding.
            assert abs(mpmath.mpf(float(r)) - want) <= 0.5 * np.spacing(float(want)) + 0.51 * 2.0 ** -53 * want


# Round and flat bodies, the angle between the scaled vectors on both sides of a right angle (each branch of the
# half-angle quotients).
@pytest.mark.parametrize("b,c", [(1.0, 1.0), (0.7, 0.4), (0.9, 0.02), (0.1, 0.05)])
def test_magnitude(lib, b, c):
    rng = np.random.default_rng(5)
    n = 300
    v = np.empty((n, 8))
    v[:, 0], v[:, 1] = b, c
    S = rng.normal(size=(n, 3))
    E = S + rng.normal(size=(n, 3)) * rng.choice([0.1, 1.0, 5.0], (n, 1))
    v[:, 2:5] = S / np.linalg.norm(S, axis=1, keepdims=True)
    v[:, 5:8] = E / np.linalg.norm(E, axis=1, keepdims=True)
    got = np.empty(n)
    lib.h_ls_algebraic(n, v.ctypes.data_as(C.c_void_p), got.ctypes.data_as(C.c_void_p))
    with mpmath.workprec(160):
        compared = 0
        for vi, g in zip(v, got):
            sb, sc, sa, eb, ec, ea = (mpmath.mpf(float(x)) for x in vi[2:])
            B, K = mpmath.mpf(b), mpmath.mpf(c)
            s = mpmath.sqrt(sb * sb / (B * B) + sc * sc / (K * K) + sa * sa)
            e = mpmath.sqrt(eb * eb / (B * B) + ec * ec / (K * K) + ea * ea)
            ca = (sb * eb / (B * B) + sc * ec / (K * K) + sa * ea) / (s * e)
            al = mpmath.acos(ca)
            if not 0.05 < al < 2.5:
                continue
            compared += 1
            sc_ = mpmath.sqrt(s * s + e * e + 2 * s * e * ca)
            la = mpmath.atan2(e * mpmath.sin(al) / sc_, (s + e * ca) / sc_)
            want = -2.5 * mpmath.log10(B * K * s * e / sc_ * (
                mpmath.cos(la - al) + mpmath.cos(la) + mpmath.sin(la) * mpmath.sin(la - al) *
                mpmath.log(1 / mpmath.tan(la / 2) / mpmath.tan((al - la) / 2))))
            # cos alpha' carries eight roundings, which sin alpha' turns into an angle; a magnitude moves by up to
            # 2.5 / ln 10 d ln B / d alpha', below 10 up to alpha' = 2.5.  The rest: twenty roundings of the factors.
            assert abs(g - want) <= (10 * 8 / mpmath.sin(al) + 1.09 * 20) * 2.0 ** -53 + 2.0 ** -52 * abs(want)
        assert compared > 50


def test_reciprocals(lib):
    rng = np.random.default_rng(8)
    n = 4000
    s = rng.choice([-1.0, 1.0], n) * rng.uniform(1, 2, n) * 2.0 ** rng.integers(-100, 100, n)
    s[:4] = 1.0, np.nextafter(2.0, 0), np.nextafter(1.0, 2), -2.0
    out = np.empty(n)
    lib.h_recip(n, s.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
    with mpmath.workprec(200):
        for si, r in zip(s, out):
            want = 1 / mpmath.mpf(float(si))
            # One rounding; the cubic step's e^3 < 2^-57 for a seed within 2^-19, a 16th of half an ulp.
            assert abs(mpmath.mpf(float(r)) - want) <= 0.54 * np.spacing(abs(float(want)))


def _magnitude(mp, b, c, ca, s, e):
    """The magnitude from the scaled vectors' angle and lengths (cuda.c:664-689)."""
    al = mp.acos(ca)
    h = mp.sqrt(s * s + e * e + 2 * s * e * ca)
    la = mp.atan2(e * mp.sin(al) / h, (s + e * ca) / h)
    return -2.5 * mp.log10(b * c * s * e / h * (mp.cos(la - al) + mp.cos(la) + mp.sin(la) * mp.sin(la - al) *
                                                mp.log(1 / mp.tan(la / 2) / mp.tan((al - la) / 2))))


# Opposition, where data are dense and half angles small, and close to pi, where the two vectors nearly cancel.
@pytest.mark.parametrize("b,c", [(1.0, 1.0), (0.7, 0.4), (0.9, 0.02)])
@pytest.mark.parametrize("near", [0.0, np.pi])
def test_magnitude_at_the_ends(lib, b, c, near):
    rng = np.random.default_rng(11)
    n = 200
    d = rng.normal(size=(n, 3))
    S = rng.normal(size=(n, 3))
    off = np.geomspace(1e-5, 0.05 if near == 0.0 else 0.5, n)[:, None]
    # Directions of the scaled vectors (x / b, y / c, z), off by the angle; then back to the body's.
    u = S / np.linalg.norm(S, axis=1, keepdims=True)
    w = np.cross(u, d)
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    r = (1.0 if near == 0.0 else -1.0) * np.cos(off) * u + np.sin(off) * w
    v = np.empty((n, 8))
    v[:, 0], v[:, 1] = b, c
    for k, x in ((2, u), (5, r)):
        x = x * np.array([b, c, 1.0])
        v[:, k:k + 3] = x / np.linalg.norm(x, axis=1, keepdims=True)
    got = np.empty(n)
    lib.h_ls_algebraic(n, v.ctypes.data_as(C.c_void_p), got.ctypes.data_as(C.c_void_p))
    u53 = mpmath.mpf(2) ** -53
    with mpmath.workprec(200):
        B, K = mpmath.mpf(b), mpmath.mpf(c)
        for vi, g in zip(v, got):
            sb, sc, sa, eb, ec, ea = (mpmath.mpf(float(x)) for x in vi[2:])
            s = mpmath.sqrt(sb * sb / (B * B) + sc * sc / (K * K) + sa * sa)
            e = mpmath.sqrt(eb * eb / (B * B) + ec * ec / (K * K) + ea * ea)
            ca = (sb * eb / (B * B) + sc * ec / (K * K) + sa * ea) / (s * e)
            want = _magnitude(mpmath, B, K, ca, s, e)
            # What eight roundings of cos alpha' (kept a cosine) and four of each length move it by, and twenty of the
            # factors; sin alpha', 1 - cos and the sum of the vectors lose what the angle's cosine loses.
            tol = 1.09 * 20 * u53 + 2 * u53 * abs(want)
            one = mpmath.mpf(1) - u53 ** 2
            for k in (-1, 1):
                moved = max(-one, min(one, ca + 8 * k * u53))
                tol += abs(_magnitude(mpmath, B, K, moved, s, e) - want)
                tol += abs(_magnitude(mpmath, B, K, ca, s * (1 + 4 * k * u53), e) - want)
                tol += abs(_magnitude(mpmath, B, K, ca, s, e * (1 + 4 * k * u53)) - want)
            assert abs(g - want) <= tol, (float(mpmath.acos(ca)), float(g - want), float(tol))
