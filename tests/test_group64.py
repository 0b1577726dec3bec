"""The FP64 evaluation by groups of lanes (csrc/group64.cuh) against the thread path, bit for bit.

ast_eval_batch picks 32 lanes a vector up to four vectors per SM, 8 up to 32 per SM (28 with torque and many steps
an observation), and one thread a vector beyond; the same vectors evaluated in one large call and in small ones must give the same
bits, whatever the variant, the number of observations (tiles of 8 and 32, remainders) and filters."""
import ctypes as C

import numpy as np
import pytest

from asteroid_gb300 import api

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _object(flags, n, filters, seed, span):
    rng = np.random.default_rng(seed)
    model = api.make_model(flags, 1e-2, (20.0, 4800.0))
    t = np.sort(rng.uniform(0, span, n))
    unit = rng.normal(size=(2, n, 3)) * 0.05 + np.array([[0.8, 0.5, 0.3], [0.9, 0.4, -0.1]])[:, None]
    unit /= np.linalg.norm(unit, axis=2, keepdims=True)
    f = rng.integers(0, filters, n).astype(np.int32)
    f[:filters] = np.arange(filters)
    eph = np.array([-1.0, 0.5 * span, span + 1.0])
    e = np.array([[0.8, 0.79, 0.78], [0.5, 0.51, 0.52], [0.3, 0.3, 0.3]])
    s = np.array([[0.9, 0.9, 0.89], [0.4, 0.41, 0.42], [-0.1, -0.1, -0.1]])
    k = 3 if flags.find("NUDGE") >= 0 else 0
    obs = api.Obs(t - t[0], rng.normal(22, 0.4, n).astype(np.float32), rng.uniform(20, 200, n).astype(np.float32), f, unit[0],
                  unit[1], e, s, eph, np.linspace(0, span, k).astype(np.float32), np.full(k, 22.5, np.float32))
    P = []
    i_L = api.param_names(model).index("L")
    while len(P) < 700:
        p = api.x2params(model, rng.uniform(0, 1, model.n_params), reopt=1)
        if p is not None:
            p[i_L] = rng.uniform(5, 60)
            P.append(p)
    P[3][0] = np.nan  # a vector without a model
    return model, obs, np.array(P)


@pytest.mark.parametrize("flags,n,filters,span", [
    ("TORQUE,ACC", 300, 1, 4.0), ("TORQUE,INTERP", 97, 3, 1.0), ("BC,INTERP,ACC", 64, 2, 1.0), ("BC", 33, 1, 6.0),
    ("BW_BALL,ACC", 32, 4, 2.0), ("BW_BALL,TORQUE", 31, 8, 0.2), ("TORQUE,P_PSI,ACC", 40, 8, 3.0), ("ACC", 13, 1, 3.0),
    ("TORQUE,INTERP,ACC,NUDGE", 161, 2, 2.0), ("NUDGE", 39, 1, 2.0), ("TORQUE,RMSD,ACC", 65, 2, 1.5)])
def test_lane_groups_equal_threads(gpu, flags, n, filters, span):
    model, obs, P = _object(flags, n, filters, n + filters, span)
    sms = _sms()
    with api.Engine(model, obs) as eng:
        big = np.tile(P, (-(-33 * sms // len(P)), 1))
        chi2, dv = eng.eval(big)  # a thread a vector
        for count in (1, 3, 4 * sms, min(700, 4 * sms + 1), 4 * sms + 5):
            count = min(count, len(P))
            c, d = eng.eval(P[:count])
            assert np.array_equal(c, chi2[:count], equal_nan=True)
            assert np.array_equal(d, dv[:count], equal_nan=True)
        some = np.tile(P, (7, 1))[: 32 * sms]  # the most that lane groups take
        c, d = eng.eval(some)
        assert np.array_equal(c, chi2[: len(some)], equal_nan=True)
        assert np.array_equal(d, dv[: len(some)], equal_nan=True)
    assert np.isfinite(chi2[np.isfinite(chi2)]).sum() > 0.3 * len(chi2)


@pytest.mark.parametrize("flags,chains,group,kw", [
    ("TORQUE,P_PSI,ACC", 1, 1, {}), ("TORQUE,P_PSI", 33, 33, dict(n_stages=2)), ("BC,INTERP,ACC", 700, 7, {}),
    ("TORQUE,INTERP,ACC,NUDGE", 640, 64, dict(reopt=True)), ("BW_BALL,ACC", 4000, 250, dict(evals_cap=16))])
def test_fits_by_lane_groups_equal_threads(gpu, flags, chains, group, kw):
    """A fit of few chains runs by lane groups unless a geometry is asked for; both give the same chains."""
    model, obs, P = _object(flags, 48, 2, 5, 1.0)
    kw = dict(dict(evals_cap=40, n_stages=1), **kw)
    if kw.get("reopt"):
        kw["params0"] = P[0]
    with api.Engine(model, obs) as eng:
        a = eng.fit(n_chains=chains, group_size=group, seed=9, **kw)
        lanes_ctas = eng.fit_launch()["ctas"]
        b = eng.fit(n_chains=chains, group_size=group, seed=9, tpb=32, **kw)
        assert lanes_ctas > eng.fit_launch()["ctas"] or chains == 1
        eng.fit_begin(n_chains=chains, group_size=group, seed=9, **kw)  # in bounded steps
        for _ in range(1000):
            if eng.fit_step(3):
                break
        c = eng.fit_end()
    for r in (a, c):
        for k in ("best_f", "best_params", "best_dv", "chain_f"):
            assert np.array_equal(getattr(r, k), getattr(b, k), equal_nan=True), k
        assert r.n_evals == b.n_evals and r.n_fits == b.n_fits


# The most chains by lane groups, and one more, with few steps an observation (3) and many: with torque, whose steps
# have more FP64 instructions to spread, and without; the ball's magnitudes have fewer.
@pytest.mark.parametrize("flags,span,per_sm", [
    ("TORQUE,ACC", 1.0, 32), ("TORQUE,ACC", 3.0, 28), ("TORQUE", 6.0, 24), ("TORQUE,P_PSI", 3.0, 32), ("TORQUE,BW_BALL,ACC", 1.0, 28), ("ACC", 3.0, 32),
    ("BW_BALL", 6.0, 28)])
def test_where_fits_by_lane_groups_end(gpu, flags, span, per_sm):
    model, obs, P = _object(flags, 33, 2, 5, span)
    n = per_sm * _sms()
    with api.Engine(model, obs) as eng:
        for chains, lanes in ((n, 8), (n + 1, 1)):
            a = eng.fit(n_chains=chains, group_size=1, seed=9, evals_cap=13)
            assert eng.fit_launch()["ctas"] == -(-chains * lanes // 32)
            b = eng.fit(n_chains=chains, group_size=1, seed=9, evals_cap=13, tpb=32)
            for k in ("best_f", "best_params", "best_dv", "chain_f"):
                assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=True), k
