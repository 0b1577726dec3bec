"""The mixed evaluation by integrator and photometer warps (csrc/mixed.cuh) against the thread path, bit
for bit: ast_eval_batch picks pairs, two photometers an integrator, up to 128 vectors per SM, and one thread a vector
beyond."""
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


@pytest.mark.parametrize("precision", [api.PREC_MIXED, api.PREC_MIXED_RHS32])
def test_both_register_budgets_of_the_thread_kernel(gpu, precision):
    """The full register file up to two CTAs of 128 an SM, three CTAs beyond: the same bits."""
    model, obs, P = _object("TORQUE,ACC", 33, 2, 8, 1.0)
    n = 256 * _sms()
    big = np.tile(P, (-(-3 * n // 2 // len(P)), 1))[:3 * n // 2]
    with api.Engine(model, obs) as eng:
        chi2, dv = eng.eval(big, precision)
        for count in (n, n + 1):
            c, d = eng.eval(big[:count], precision)
            assert np.array_equal(c, chi2[:count], equal_nan=True) and np.array_equal(d, dv[:count], equal_nan=True)


@pytest.mark.parametrize("flags,chains,group,kw", [
    ("TORQUE,P_PSI,ACC", 1, 1, {}), ("TORQUE,P_PSI", 33, 33, dict(n_stages=2)), ("BC,INTERP,ACC", 700, 7, {}),
    ("TORQUE,INTERP,ACC,NUDGE", 640, 64, dict(reopt=True)), ("BW_BALL,ACC", 6000, 250, dict(evals_cap=16)),
    ("TORQUE,ACC", 14336, 256, dict(evals_cap=14, precision=api.PREC_MIXED_RHS32))])
def test_fits_by_pairs_equal_threads(gpu, flags, chains, group, kw):
    """A mixed fit of few chains runs by pairs unless a geometry is asked for; both give the same chains."""
    model, obs, P = _object(flags, 48, 2, 5, 1.0)
    kw = dict(dict(evals_cap=40, n_stages=1, precision=api.PREC_MIXED), **kw)
    if kw.get("reopt"):
        kw["params0"] = P[0]
    with api.Engine(model, obs) as eng:
        a = eng.fit(n_chains=chains, group_size=group, seed=9, **kw)
        assert eng.fit_launch()["tpb"] <= 128 and eng.fit_launch()["smem"] > 18000  # a PairChain
        b = eng.fit(n_chains=chains, group_size=group, seed=9, tpb=32, **kw)
        eng.fit_begin(n_chains=chains, group_size=group, seed=9, **kw)  # in bounded steps
        for _ in range(1000):
            if eng.fit_step(3):
                break
        c = eng.fit_end()
    for r in (a, c):
        for k in ("best_f", "best_params", "best_dv", "chain_f"):
            assert np.array_equal(getattr(r, k), getattr(b, k), equal_nan=True), k
        assert r.n_evals == b.n_evals and r.n_fits == b.n_fits


@pytest.mark.parametrize("acc", [True, False])
def test_batches_by_pairs_equal_threads(gpu, acc):
    """A batch of few chains runs by pairs unless a geometry is asked for: objects of uneven size, a warp that
    straddles two of them, one with NUDGE, run whole and in bounded steps."""
    end = ",ACC" if acc else ""
    objects = [_object(f + end, n, nf, n, span) for f, n, nf, span in
               (("TORQUE", 60, 2, 1.0), ("BC,INTERP", 33, 1, 2.0), ("BW_BALL", 29, 4, 0.5), ("INTERP,NUDGE", 41, 1, 1.0))]
    chains = (64, 48, 16, 33)  # the second and third share a warp

    def batch(steps=0, **geometry):
        with api.Batch(precision=api.PREC_MIXED, acc=acc) as b:
            for (model, obs, P), c in zip(objects, chains):
                b.add(model, obs, n_chains=c, group_size=c, seed=4, evals_cap=30)
            if steps:
                while not b.step(steps)[0]:
                    pass
            else:
                b.run(**geometry)
            c = b.counters()
            return [b.result(i) for i in range(len(objects))], c

    ref, c0 = batch(tpb=128, refill=1)
    for got, c in (batch(), batch(steps=5)):
        assert c["refill"] == 32 and c["tpb"] == 32 and c["n_evals"] == c0["n_evals"]
        for r, g in zip(ref, got):
            for k in ("best_f", "best_params", "best_dv"):
                assert np.array_equal(getattr(r, k), getattr(g, k), equal_nan=True)


def test_a_requested_geometry_is_not_run_by_the_paired_graph(gpu):
    """Three warps a CTA, refill 32, two CTAs: a paired launch of one integrator a CTA and a launch of one thread
    a chain alike.  The batch's graph is recorded again for the second, whose time tells which kernel ran."""
    model, obs, P = _object("TORQUE,ACC", 300, 2, 3, 0.05)

    def batch():
        b = api.Batch(precision=api.PREC_MIXED, acc=True, n_slots=192)
        b.add(model, obs, n_chains=64, group_size=32, seed=4, evals_cap=60, reopt=True, params0=P[0])
        return b

    def ms(b, **geometry):
        t = min(b.run(**geometry) for _ in range(3))
        return t, b.result(0)

    with batch() as b:
        threads, ref = ms(b, tpb=96, refill=32)
    with batch() as b:
        pairs, r = ms(b)
        after, g = ms(b, tpb=96, refill=32)
        assert b.counters()["tpb"] == 96 and b.counters()["ctas"] == 2
    assert pairs < 0.85 * threads  # the two kernels' times are told apart
    assert after > 0.92 * threads, (pairs, threads, after)
    for k in ("best_f", "best_params", "best_dv"):
        assert np.array_equal(getattr(r, k), getattr(ref, k), equal_nan=True)
        assert np.array_equal(getattr(g, k), getattr(ref, k), equal_nan=True)


# One integrator to four, and where threads take over: with torque at the third or fourth (a start from the prior,
# without a period's range, or from a model; few steps an observation or many), with NUDGE at the third, with the FP32
# right-hand side and few steps at the fourth.
@pytest.mark.parametrize("flags,chains,span,precision,reopt,integrators", [
    ("ACC", 4864, 1.0, api.PREC_MIXED, False, 1), ("ACC", 19456, 1.0, api.PREC_MIXED, False, 4), ("ACC", 19488, 1.0, api.PREC_MIXED, False, 0),
    ("TORQUE,ACC", 9728, 1.0, api.PREC_MIXED, False, 2), ("TORQUE,ACC", 9760, 1.0, api.PREC_MIXED, False, 0),
    ("TORQUE,ACC", 9760, 5.0, api.PREC_MIXED, False, 3), ("TORQUE,ACC", 14624, 5.0, api.PREC_MIXED, False, 0),
    ("TORQUE,ACC", 14624, 12.0, api.PREC_MIXED, False, 4), ("TORQUE,ACC", 14592, 1.0, api.PREC_MIXED, True, 3),
    ("TORQUE", 14624, 1.0, api.PREC_MIXED, True, 0), ("TORQUE", 14624, 5.0, api.PREC_MIXED, True, 4),
    ("TORQUE,P_PSI,ACC", 9760, 1.0, api.PREC_MIXED, False, 3), ("TORQUE,P_PSI,ACC", 14624, 1.0, api.PREC_MIXED, False, 0), ("NUDGE", 9728, 1.0, api.PREC_MIXED, True, 2), ("NUDGE", 9760, 5.0, api.PREC_MIXED, True, 0),
    ("TORQUE,ACC", 14592, 1.0, api.PREC_MIXED_RHS32, False, 3), ("TORQUE,ACC", 14624, 1.0, api.PREC_MIXED_RHS32, True, 0),
    ("TORQUE", 14624, 0.4, api.PREC_MIXED, True, 4), ("TORQUE,NUDGE", 9760, 12.0, api.PREC_MIXED, True, 3),
    ("TORQUE,NUDGE", 9760, 1.0, api.PREC_MIXED_RHS32, True, 3),
    ("TORQUE,ACC", 14624, 5.0, api.PREC_MIXED_RHS32, True, 4)])
def test_where_fits_by_pairs_end(gpu, flags, chains, span, precision, reopt, integrators):
    if _sms() != 152:
        pytest.skip("the chain counts are those of 152 SMs")
    model, obs, P = _object(flags, 48, 2, 5, span)
    kw = dict(reopt=True, params0=P[0]) if reopt else {}
    with api.Engine(model, obs) as eng:
        a = eng.fit(n_chains=chains, group_size=32, seed=2, evals_cap=13, precision=precision, **kw)
        g = eng.fit_launch()
        # A PairChain is some 27 KB; the block of 48 points is 8.
        assert (g["tpb"] // 32 if g["smem"] > 18000 else 0) == integrators, g
        b = eng.fit(n_chains=chains, group_size=32, seed=2, evals_cap=13, precision=precision, tpb=128, **kw)
    for k in ("best_f", "best_params", "best_dv", "chain_f"):
        assert np.array_equal(getattr(a, k), getattr(b, k), equal_nan=True), k


def test_a_paired_geometry_read_back_selects_the_pairs(gpu):
    """What ast_batch_geometry returns, given to ast_batch_run or ast_batch_set_geometry of another batch, runs the
    same kernel (told by its time) with the same results; beside fields that do not go with it, pair counts as 0."""
    model, obs, P = _object("TORQUE,ACC", 300, 2, 3, 0.05)

    def batch():
        b = api.Batch(precision=api.PREC_MIXED, acc=True)
        b.add(model, obs, n_chains=4864, group_size=32, seed=4, evals_cap=30, reopt=True, params0=P[0])
        return b

    with batch() as b:
        pairs, ref = min(b.run() for _ in range(3)), b.result(0)
        c = b.counters()
        g = {k: c[k] for k in ("tpb", "refill", "tile", "pair") if k in c}
    with batch() as b:
        threads = min(b.run(tpb=128) for _ in range(3))
    assert pairs < 0.85 * threads
    with batch() as b:
        again = min(b.run(**g) for _ in range(3))
        assert b.counters()["pair"] == g["pair"] > 0 and b.counters()["ctas"] == c["ctas"]
        run = b.result(0)
    with batch() as b:
        b.set_geometry(**g)
        step = 0.0
        while True:
            done, ms = b.step(8)
            step += ms
            if done:
                break
        stepped = b.result(0)
    assert again < 1.1 * pairs and step < 1.3 * pairs, (pairs, threads, again, step)
    with batch() as b:
        for other in (dict(g, tpb=64), dict(g, refill=1), dict(g, tile=8), dict(g, pair=5, tpb=160)):
            b.set_geometry(**other)
            assert b.counters()["pair"] == 0
    for r in (run, stepped):
        for k in ("best_f", "best_params", "best_dv"):
            assert np.array_equal(getattr(r, k), getattr(ref, k), equal_nan=True)


def test_the_tuner_times_pairs(gpu):
    """A tuned batch of few chains is no slower than one that is not, and gives the same results."""
    model, obs, P = _object("TORQUE,ACC", 300, 2, 3, 0.05)
    got = []
    for tune in (False, True):
        with api.Batch(precision=api.PREC_MIXED, acc=True) as b:
            b.add(model, obs, n_chains=4864, group_size=32, seed=4, evals_cap=30, reopt=True, params0=P[0])
            if tune:
                t = b.tune(evals_per_slot=4)
            got.append((min(b.run() for _ in range(3)), b.result(0)))
            if tune:
                assert t["pair"] > 0 and t["tpb"] == 32 * t["pair"] and b.counters()["pair"] == t["pair"]
    assert got[1][0] < 1.1 * got[0][0], (got[0][0], got[1][0])
    for k in ("best_f", "best_params", "best_dv"):
        assert np.array_equal(getattr(got[0][1], k), getattr(got[1][1], k), equal_nan=True)
