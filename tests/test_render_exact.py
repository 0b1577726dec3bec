"""Frames shaded in double-float with error bounds (csrc/animate.cu) against the oracle's FP64, byte for byte:
flattened and round bodies, grazing and back light, the spot on the limb, frame sizes off the tile."""
import numpy as np
import pytest

from asteroid_gb300 import api

pytestmark = pytest.mark.gpu


def _geometry(rng, b, c, e_body=None, s_body=None):
    """One snapshot: random body axes, Earth and Sun (or those given, in the body frame b, c, a)."""
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    unit = lambda v: np.asarray(v, float) / np.linalg.norm(v)
    e = unit(rng.normal(size=3)) if e_body is None else unit(e_body)
    s = unit(rng.normal(size=3)) if s_body is None else unit(s_body)
    return np.concatenate([[b, c], q.T @ e, e, s, q.ravel()])


CASES = {
    "ordinary": lambda r: [_geometry(r, *r.uniform(0.15, 1.0, 2)) for _ in range(6)],
    "flat": lambda r: [_geometry(r, b, c) for b, c in ((0.9, 0.01), (0.02, 0.01), (0.5, 0.1), (1.0, 0.03))],
    "sphere": lambda r: [_geometry(r, 1.0, 1.0), _geometry(r, 1.0, 1.0, (0, 0, 1), (0, 0, 1)),
                         _geometry(r, 1.0, 1.0, (0, 0, 1), (0, 0, -1)), _geometry(r, 1.0, 1.0, (0, 0, 1), (1, 0, 0))],
    "along_axes": lambda r: [_geometry(r, 0.6, 0.3, e, s) for e in ((1, 0, 0), (0, 1, 0), (0, 0, 1)) for s in ((1, 0, 0), (0, 1, 1e-9))],
    "spot": lambda r: [_geometry(r, 0.7, 0.5, (1, y, 0.02), (0.8, 0.1, 0.1)) for y in (0.0, 0.5, 5.0, 50.0)],
    "no_projection": lambda r: [np.concatenate([[0.5, 0.4, 0, 1, 0], np.eye(3)[1], np.eye(3)[0], np.eye(3).ravel()])],
}


@pytest.mark.parametrize("size", [2, 34, 250, 600])
@pytest.mark.parametrize("case", sorted(CASES))
def test_frames_equal_fp64(gpu, oracle_mod, case, size):
    geo = np.ascontiguousarray(CASES[case](np.random.default_rng(size)))
    got, _ = api.render_frames(geo, size)
    assert np.array_equal(got, oracle_mod.render(geo, size))
