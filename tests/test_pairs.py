"""The mixed evaluation by integrator and photometer warps (csrc/mixed.cuh) against the thread path, bit
for bit: ast_eval_batch picks two photometers an integrator up to 32 vectors per SM, one up to 128
per SM, and one thread a vector beyond."""
import numpy as np
import pytest

from asteroid_gb300 import api
from tests.test_group64 import _object, _sms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [api.PREC_MIXED, api.PREC_MIXED_RHS32])
@pytest.mark.parametrize("flags,n,filters,span", [
    ("TORQUE,ACC", 65, 1, 2.0), ("TORQUE,INTERP", 24, 3, 1.0), ("BC,INTERP,ACC", 23, 2, 1.0), ("BW_BALL,ACC", 31, 8, 2.0),
    ("ACC", 13, 1, 3.0), ("TORQUE,INTERP,ACC,NUDGE", 161, 2, 2.0), ("NUDGE", 39, 1, 2.0), ("TORQUE,RMSD,ACC", 40, 2, 1.5)])
def test_pairs_equal_threads(gpu, flags, n, filters, span, precision):
    model, obs, P = _object(flags, n, filters, n + filters, span)
    sms = _sms()
    big = np.tile(P, (-(-129 * sms // len(P)), 1))
    with api.Engine(model, obs) as eng:
        chi2, dv = eng.eval(big, precision)  # a thread a vector
        for count in (1, 33, 32 * sms, 32 * sms + 1, 64 * sms + 17, 128 * sms):
            c, d = eng.eval(big[:count], precision)
            assert np.array_equal(c, chi2[:count], equal_nan=True), count
            assert np.array_equal(d, dv[:count], equal_nan=True), count
    assert np.isfinite(chi2).mean() > 0.3
