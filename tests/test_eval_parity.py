"""The FP64 evaluation that ships against the search's expressions, compiled alike.

build.build_parity_engine(contract=True) evaluates in the reference's own expressions, CUDA's sincos, division and
inverse functions, which its uncontracted twin ties to the reference kernel (tests/test_ref_kernel_nofma.py).  What
ast_eval_batch runs -- the table's sines, quot and inv_sqrt, the rearranged magnitude -- differs from it by rounding
only, and must stay as close to it as tests/test_ref_kernel.py asks of the reference kernel, another program with the
same contractions: 1e-12 relative chi^2 for most, and what the vector's own sensitivity to one ulp of its parameters
explains for the rest.

That library is loaded in a child process (AST_ENGINE_LIB)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
GOLDEN = ROOT / "tests" / "golden"
if __name__ == "__main__":
    sys.path[:0] = [str(ROOT), str(ROOT / "oracle")]

from asteroid_gb300 import api  # noqa: E402


def _vectors(fx, m):
    rng = np.random.default_rng(37)
    i_L = api.param_names(m).index("L")
    P = [np.array(p) for p in fx["params"]]
    while len(P) < 256:
        p = api.x2params(m, rng.uniform(0, 1, m.n_params), reopt=0)
        if p is not None and p[i_L] * m.time_step <= 0.5:
            P.append(p)
    return np.array(P)


def _evaluate(n):
    """chi^2 of every fixture's vectors, n of them a call (lane groups or, tiled past their range, threads)."""
    from tests.test_oracle_pin import load_fixture

    out = {}
    for path in sorted(GOLDEN.glob("ref_*.json")):
        fx, m, obs = load_fixture(path)
        P = _vectors(fx, m)
        with api.Engine(m, obs) as eng:
            out[path.stem] = eng.eval(np.tile(P, (-(-n // len(P)), 1)), api.PREC_FP64)[0][:len(P)]
    return out


@pytest.mark.gpu
def test_shipped_evaluations_agree_with_the_librarys_functions(gpu, oracle_mod, tmp_path):
    from asteroid_gb300 import build
    from tests.test_gpu_eval import well_conditioned
    from tests.test_oracle_pin import load_fixture
    from tests.test_ref_kernel import ROUNDING_SLACK, RTOL

    lib = build.build_parity_engine(contract=True)
    f = tmp_path / "library.npz"
    r = subprocess.run([sys.executable, str(Path(__file__).resolve()), str(f)], cwd=str(ROOT),
                       env=dict(os.environ, AST_ENGINE_LIB=str(lib)), stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-4000:]
    ref = np.load(f)
    for n in (256, 152 * 33):
        for name, got in _evaluate(n).items():
            fx, m, obs = load_fixture(GOLDEN / f"{name}.json")
            want = ref[name]
            good, cond = well_conditioned(oracle_mod, m, obs, _vectors(fx, m), return_cond=True)
            assert not np.any(good & (np.isfinite(want) != np.isfinite(got))), name
            fin = good & np.isfinite(want) & np.isfinite(got)
            rel = np.abs(got[fin] - want[fin]) / np.abs(want[fin])
            print(f"{name}, {n} a call: {fin.sum()} of {len(want)}, max rel {rel.max():.2e}, <= 1e-12: {np.mean(rel <= RTOL):.3f}, "
                  f"within: {np.mean(rel <= np.maximum(RTOL, ROUNDING_SLACK * cond[fin])):.3f}")
            assert fin.sum() >= 100, name
            assert rel.max() <= 1e-10, name
            assert np.mean(rel <= np.maximum(RTOL, ROUNDING_SLACK * cond[fin])) >= 0.95, name
            assert np.mean(rel <= RTOL) >= 0.82, name


if __name__ == "__main__":
    np.savez(sys.argv[1], **_evaluate(256))
