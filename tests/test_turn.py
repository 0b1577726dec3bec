"""The mixed path's RK4 step on compact angles (csrc/turn.cuh), compiled for the host, against
plain FP64: the table's sin and cos, the angle's round trip, the step itself in both rotations."""
import ctypes as C
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

from asteroid_gb300 import build

ROOT = Path(__file__).resolve().parents[1]
T = 4096
STEP = 2 * math.pi / T


@pytest.fixture(scope="module")
def lib(built, tmp_path_factory):
    out = tmp_path_factory.mktemp("turn") / "libturn_harness.so"
    subprocess.run([build._nvcc(), "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-O2", "-std=c++17",
                    f"-I{build.PKG / 'csrc'}", f"-I{build.INCLUDE}", str(ROOT / "tests" / "host" / "turn_harness.cu"),
                    "-o", str(out)], check=True, capture_output=True)
    lib = C.CDLL(str(out))
    lib.h_turn_round_trip.restype = C.c_double
    lib.h_turn_round_trip.argtypes = [C.c_double, C.c_int]
    lib.h_turn_steps.argtypes = [C.c_int, C.c_int, C.c_double, C.c_void_p, C.c_void_p]
    return lib


def P(a):
    return a.ctypes.data_as(C.c_void_p)


# |e| at both ends and the middle of its range, every octant's table points and beyond one turn.
@pytest.mark.parametrize("e", [0.0, 1e-6, 0.25, 0.499, 0.5, -0.5])
def test_sin_and_cos_of_compact_angles(lib, e):
    k = np.array([0, 1, 2, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 3071, 3072, 3073, 4095, 4096, 8191, -1, -1024],
                 np.int32)
    n = len(k) // 2
    t = np.linspace(-1.5e-5, 1.5e-5, len(k)).astype(np.float32)
    ee = np.full(len(k), e, np.float32)
    out = np.zeros(4 * len(k), np.float32)
    lib.h_turn_sincos(n, P(k), P(ee), P(t), P(out))
    out = out.reshape(-1, 4).astype(np.float64)
    a = ((k % T) + ee.astype(np.float64) + t) * STEP
    # Three roundings of v <= 3e-7, two of a sum below 7e-7, at 2^-24 each, and the FP64 argument.
    tol = 3 * 3e-7 * 2.0 ** -24 + 2 * 7e-7 * 2.0 ** -24 + 2e-15
    assert np.max(np.abs(out[:, 0] + out[:, 1] - np.sin(a))) <= tol
    assert np.max(np.abs(out[:, 2] + out[:, 3] - np.cos(a))) <= tol


@pytest.mark.parametrize("turns", [1, 2])
def test_round_trip(lib, turns):
    for a in [0.0, 1e-9, 0.1, -0.1, 3.0, -3.0, 3.1415, -3.1415, 0.5 * STEP, 1.5 * STEP, 7.0, -40.0, 1234.5]:
        r = lib.h_turn_round_trip(a, turns)
        # A product and a reduction of double-floats below 2 pi: a few u^2 of it; 1234.5 enters with u^2 of itself.
        assert abs((r - a + math.pi) % (2 * math.pi) - math.pi) <= 1e-13 + 2.0 ** -47 * abs(a)
        assert abs(r) <= math.pi + 1e-6


def _rk4(torque, h, mu, y):
    def f(y):
        if torque:
            s5, c5, s4, c4 = math.sin(y[5]), math.cos(y[5]), math.sin(y[4]), math.cos(y[4])
            k3 = (y[0] * s5 + y[1] * c5) / s4
            return np.array([mu[0] * y[1] * y[2] + mu[3], mu[1] * y[2] * y[0] + mu[4], mu[2] * y[0] * y[1] + mu[5], k3,
                             y[0] * c5 - y[1] * s5, y[2] - k3 * c4])
        k0 = mu[0] * (mu[1] - mu[2] * math.cos(2 * y[5]))
        return np.array([0, 0, 0, k0, mu[0] * mu[2] * math.sin(y[4]) * math.sin(2 * y[5]), math.cos(y[4]) * (mu[0] - k0)])

    k1 = f(y)
    k2 = f(y + 0.5 * h * k1)
    k3 = f(y + 0.5 * h * k2)
    k4 = f(y + h * k3)
    return y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


# rate: rad/day; 3e6 rad/day advances an angle by 4800 turns a step, which the general step takes.
@pytest.mark.parametrize("torque", [1, 0])
@pytest.mark.parametrize("rate,h", [(0.5, 1e-2), (30.0, 1e-2), (60.0, 5e-3), (60.0, 1e-5), (3e6, 1e-2)])
def test_one_step_matches_fp64(lib, torque, rate, h):
    rng = np.random.default_rng(int(rate) + torque)
    for _ in range(50):
        y = np.concatenate([rng.uniform(-rate, rate, 3), rng.uniform(-3, 3, 1), rng.uniform(0.3, 2.8, 1), rng.uniform(-3, 3, 1)])
        y = np.array([float(np.float32(v)) for v in y])
        mu = np.concatenate([rng.uniform(-0.5, 0.5, 3), rng.uniform(-1, 1, 3)]) if torque else np.array([rate, 0.7, 0.2])
        if rate > 1e5:
            mu[:3] = [0.0, 0.0, 0.0] if torque else [rate, 0.7, 0.0]
        got = y.copy()
        lib.h_turn_steps(torque, 1, h, P(mu), P(got))
        ref = _rk4(torque, h, mu, y)
        # A few u^2 of the increment (the rate times h, amplified by 1/sin(theta)^2 <= 11.5) and of pi.
        tol = 2.0 ** -48 * (40 * 11.5 * (1 + rate * h) ** 2 + 16 * math.pi)
        if rate > 1e5:
            assert np.all(np.isfinite(got))  # thousands of turns a step: the outcome is noise, but finite
            continue
        d = (got[3:] - ref[3:] + math.pi) % (2 * math.pi) - math.pi
        assert np.max(np.abs(d)) <= tol
        if torque:
            assert np.max(np.abs(got[:3] - ref[:3])) <= tol * (1 + rate)


@pytest.mark.parametrize("torque", [1, 0])
def test_a_thousand_steps_keep_the_phase(lib, torque):
    y = np.array([9.0, -14.0, 25.0, 0.3, 1.2, -0.7])
    mu = np.array([0.31, -0.22, -0.09, 0.01, -0.02, 0.015]) if torque else np.array([28.0, 0.75, 0.11])
    got, ref = y.copy(), y.copy()
    lib.h_turn_steps(torque, 1000, 0.01, P(mu), P(got))
    for _ in range(1000):
        ref = _rk4(torque, 0.01, mu, ref)
    d = (got[3:] - ref[3:] + math.pi) % (2 * math.pi) - math.pi
    # 300 rad at u^2 systematically (the constants' own rounding), ten times that for the random part.
    assert np.max(np.abs(d)) <= 10 * 300 * 2.0 ** -48


# From the same time twice to the shortest and an ordinary interval: where the step's size in table points, or its
# inverse, leaves a float's range the state stays as it is.
@pytest.mark.parametrize("torque", [1, 0])
@pytest.mark.parametrize("t", [0.0, 5e-324, 1e-45, 1e-40, 1e-30, 1e-18, 1e-12, 1e-3])
def test_intervals_down_to_nothing(lib, torque, t):
    lib.h_turn_interval.argtypes = [C.c_int, C.c_double, C.c_double, C.c_void_p, C.c_void_p]
    y = np.array([9.0, -14.0, 25.0, 0.25, 1.25, -0.75])
    mu = np.array([0.31, -0.22, -0.09, 0.01, -0.02, 0.015]) if torque else np.array([28.0, 0.75, 0.11])
    got = y.copy()
    lib.h_turn_interval(torque, t, 1e-2, P(mu), P(got))
    ref = _rk4(torque, t, mu, y)
    tol = 2.0 ** -48 * (40 * 11.5 * (1 + 30 * t) ** 2 + 16 * math.pi)  # as a step's above
    assert np.max(np.abs((got[3:] - ref[3:] + math.pi) % (2 * math.pi) - math.pi)) <= tol
    if torque:
        assert np.max(np.abs(got[:3] - ref[:3])) <= (tol * 31 if t > 1e-17 else 0.0)


# The general step (an angle that advances by more than 1000 turns in a step) where its outcome is determined: free
# rotation about the body axis, mu = (L, Ip, 0), theta constant, phi and psi linear.
@pytest.mark.parametrize("rate", [1e6, -1e6, 3e6, 2e7])
@pytest.mark.parametrize("theta", [0.4, 1.2, 2.7])
def test_the_general_step_of_free_rotation(lib, rate, theta):
    y = np.array([0.0, 0.0, 0.0, 0.25, float(np.float32(theta)), -0.7])
    mu = np.array([rate, 0.7, 0.0])
    got = y.copy()
    lib.h_turn_steps(0, 1, 1e-2, P(mu), P(got))
    ref = _rk4(0, 1e-2, mu, y)
    # Ten roundings of u^2 = 2^-48 of the angle's advance (twice it, of 2 psi) and of FP64's, and of pi.
    tol = (10 * 2.0 ** -48 + 10 * 2.0 ** -53) * 2 * abs(rate) * 1e-2 + 16 * math.pi * 2.0 ** -48
    d = (got[3:] - ref[3:] + math.pi) % (2 * math.pi) - math.pi
    assert np.max(np.abs(d)) <= tol
    assert abs(abs(got[4]) - theta) < 1e-6  # (theta itself does not advance)


# With torque: rotation about the long axis alone, so that only psi advances, and w2 by the torque.
@pytest.mark.parametrize("rate", [1e6, -3e6, 2e7])
def test_the_general_step_with_torque(lib, rate):
    y = np.array([0.0, 0.0, float(np.float32(rate)), 0.25, 1.2, -0.7])
    mu = np.array([0.0, 0.0, 0.31, 0.0, 0.0, 8192.0])
    got = y.copy()
    lib.h_turn_steps(1, 1, 1e-2, P(mu), P(got))
    ref = _rk4(1, 1e-2, mu, y)
    tol = (10 * 2.0 ** -48 + 10 * 2.0 ** -53) * abs(rate) * 1e-2 + 16 * math.pi * 2.0 ** -48
    d = (got[3:] - ref[3:] + math.pi) % (2 * math.pi) - math.pi
    assert np.max(np.abs(d)) <= tol
    assert np.max(np.abs(got[:3] - ref[:3])) <= 4 * 2.0 ** -48 * abs(rate)


# The general step alone, at rates that the compact step takes: its own h, h/2, h/6 and h/3, all of mu, both layouts.
@pytest.mark.parametrize("torque", [1, 0])
@pytest.mark.parametrize("rate,h", [(0.5, 1e-2), (30.0, 1e-2), (60.0, 5e-3)])
def test_the_general_step_at_ordinary_rates(lib, torque, rate, h):
    lib.h_general_step.argtypes = [C.c_int, C.c_double, C.c_void_p, C.c_void_p]
    rng = np.random.default_rng(int(rate) + torque)
    for _ in range(50):
        y = np.concatenate([rng.uniform(-rate, rate, 3), rng.uniform(-3, 3, 1), rng.uniform(0.3, 2.8, 1), rng.uniform(-3, 3, 1)])
        y = np.array([float(np.float32(v)) for v in y])
        mu = np.concatenate([rng.uniform(-0.5, 0.5, 3), rng.uniform(-1, 1, 3)]) if torque else np.array([rate, 0.7, 0.2])
        got = y.copy()
        lib.h_general_step(torque, h, P(mu), P(got))
        ref = _rk4(torque, h, mu, y)
        # As test_one_step_matches_fp64's, with the general step's own sin and cos (1e-13, dfloat.cuh) an advance.
        tol = 2.0 ** -48 * (40 * 11.5 * (1 + rate * h) ** 2 + 16 * math.pi) + 4e-13 * (1 + rate * h) * 11.5
        d = (got[3:] - ref[3:] + math.pi) % (2 * math.pi) - math.pi
        assert np.max(np.abs(d)) <= tol
        if torque:
            assert np.max(np.abs(got[:3] - ref[:3])) <= tol * (1 + rate)
