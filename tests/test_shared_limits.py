"""A kernel's limit on dynamic shared memory holds for every context and thread of the process: a call that
needs little of it must not take it from one that needs much.  Large and small fits and batches stepped in
turn, and evaluations from two threads, against the same calls alone, bit for bit."""
import threading

import numpy as np
import pytest

from asteroid_gb300 import api
from tests.test_group64 import _object

pytestmark = pytest.mark.gpu

KEYS = ("best_f", "best_params", "best_dv")


def _same(a, b):
    for k in KEYS:
        assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=True), k


# The paired mixed kernel with three integrators a CTA and with one; observation blocks staged in shared
# memory, of 400 points and of 40.
@pytest.mark.parametrize("precision,large,small,kw", [
    (api.PREC_MIXED, (48, 14336), (48, 64), {}), (api.PREC_MIXED_RHS32, (48, 14336), (48, 64), {}),
    (api.PREC_MIXED, (400, 256), (40, 256), dict(tpb=128, stage_obs=1)),
    (api.PREC_FP64, (400, 256), (40, 256), dict(tpb=128, stage_obs=1))])
def test_fits_in_turn_equal_fits_alone(gpu, precision, large, small, kw):
    def begin(eng, chains):
        eng.fit_begin(n_chains=chains, group_size=32, seed=3, evals_cap=14, precision=precision, **kw)

    objects = [_object("ACC", n, 2, 5, 1.0)[:2] for n, _ in (large, small)]
    chains = (large[1], small[1])
    ref = []
    for (model, obs), c in zip(objects, chains):
        with api.Engine(model, obs) as eng:
            ref.append(eng.fit(n_chains=c, group_size=32, seed=3, evals_cap=14, precision=precision, **kw))
    with api.Engine(*objects[0]) as a, api.Engine(*objects[1]) as b:
        begin(a, chains[0])
        begin(b, chains[1])
        assert a.fit_launch()["smem"] > b.fit_launch()["smem"] > 0
        done = [False, False]
        for _ in range(1000):
            done = [d or e.fit_step(3) for d, e in zip(done, (a, b))]
            if all(done):
                break
        got = [a.fit_end(), b.fit_end()]
    for g, r in zip(got, ref):
        _same(g, r)


@pytest.mark.parametrize("geometry", [None, dict(tile=32)])
def test_batches_in_turn_equal_batches_alone(gpu, geometry):
    """Pairs, three integrators a CTA and one; warp tiles, CTAs of four warps and of two."""
    model, obs, _ = _object("TORQUE,ACC", 60, 2, 7, 1.0)

    def batch(chains, tpb):
        b = api.Batch(precision=api.PREC_MIXED, acc=True)
        b.add(model, obs, n_chains=chains, group_size=32, seed=4, evals_cap=14)
        if geometry:
            b.set_geometry(tpb=tpb, refill=32, **geometry)
        return b

    def run(*batches):
        done = [False] * len(batches)
        for _ in range(1000):
            done = [d or b.step(3)[0] for d, b in zip(done, batches)]
            if all(done):
                break
        return [b.result(0) for b in batches]

    sizes = ((14336, 128), (64, 64))
    ref = []
    for size in sizes:
        with batch(*size) as b:
            ref += run(b)
    with batch(*sizes[0]) as a, batch(*sizes[1]) as b:
        for g, r in zip(run(a, b), ref):
            _same(g, r)


def test_evaluations_from_two_threads(gpu):
    model, obs, P = _object("TORQUE,ACC", 20, 2, 9, 0.5)
    counts = (14000, 1000)
    sets = [np.tile(P, (-(-n // len(P)), 1))[:n] for n in counts]
    engines = [api.Engine(model, obs) for _ in counts]
    ref = [e.eval(p, api.PREC_MIXED) for e, p in zip(engines, sets)]
    failed = []

    def loop(k):
        try:
            for _ in range(200):
                c, d = engines[k].eval(sets[k], api.PREC_MIXED)
                assert np.array_equal(c, ref[k][0], equal_nan=True) and np.array_equal(d, ref[k][1], equal_nan=True)
        except Exception as e:  # shown by the assertion below
            failed.append((k, e))

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for e in engines:
        e.close()
    assert not failed, failed
