"""ast_fit_noalloc with the observation block staged in shared memory, which takes a geometry: with none asked for, few
chains run by lane groups or pairs, which read the block through L1 (tests/test_zz_no_alloc.py).  480 points are
a block of 65 KB, above the 48 KB that need a launch attribute; 2000 points do not fit and are read through L1.  A fresh
process, whose first fit is ast_fit_noalloc, so that no earlier ast_fit sets the attribute."""
import subprocess
import sys
import tempfile
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if __name__ == "__main__":
    for p in (str(ROOT), str(ROOT / "oracle")):
        if p not in sys.path:
            sys.path.insert(0, p)

from asteroid_gb300 import api  # noqa: E402
from tests.test_zz_no_alloc import _fit, _noalloc, _same  # noqa: E402


@pytest.mark.gpu
def test_noalloc_stages_the_block_in_a_fresh_process(gpu):
    r = subprocess.run([sys.executable, str(Path(__file__).resolve()), "fresh"], cwd=str(ROOT), stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=600)
    print(r.stdout[-4000:])
    assert r.returncode == 0, r.stdout[-4000:]


def _fresh_process_main() -> int:
    import oracle
    from asteroid_gb300 import synth

    oracle.load()
    fit_cfg = api.fit_cfg  # _noalloc takes its configuration from it

    def staged(**kw):
        cfg, keep = fit_cfg(**kw)
        cfg.tpb, cfg.stage_obs = 128, 1
        return cfg, keep

    with tempfile.TemporaryDirectory() as d:
        for name, block in (("c1", True), ("c2", False)):
            s = synth.generate(name, Path(d) / name, vmod_fn=lambda m, o, p: oracle.model_curve(m, o, p))
            for prec in (api.PREC_FP64, api.PREC_MIXED):
                args = (s, 256, 128, 2, 31, 10, prec)
                api.fit_cfg = staged
                got = [_noalloc(*args) for _ in range(2)]
                api.fit_cfg = fit_cfg
                with api.Engine(s.model, s.obs) as eng:
                    ref = eng.fit(n_chains=256, group_size=128, n_stages=2, seed=31, evals_cap=10, precision=prec, tpb=128,
                                  stage_obs=1)
                    smem = eng.fit_launch()["smem"]
                assert (smem > 48 << 10) if block else smem == 0, (name, smem)
                for g in got:
                    _same(g, ref, (name, prec, "staged"))
                    _same(g, _fit(*args), (name, prec, "default geometry"))
                print(f"{name} ({s.obs.n_data} points, precision {prec}): {smem} bytes staged, equal to ast_fit")
    return 0


if __name__ == "__main__" and len(sys.argv) > 1 and sys.argv[1] == "fresh":
    sys.exit(_fresh_process_main())
