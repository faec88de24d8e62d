"""A hybrid batch whose persistent CTAs walk several tiles each, of problems
with TMA tensor maps (even my) and without (odd my) in turn: the same steps
and states as separate solvers.  Tolerance 1e-5 relative L-infinity, the
FP32 arithmetic's bar for the batch (the two kernels' contractions differ)."""
import numpy as np
import pytest

from conftest import interior, rel_linf
from finess_b200 import problems as P
from finess_b200._abi import FIN_PREC_HYBRID, FIN_WENO_JS, FIN_WENO_Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weno", [FIN_WENO_Z, FIN_WENO_JS])
def test_hybrid_batch_of_many_tiles(weno):
    from finess_b200.batch import Batch, first_dt, load_indicator
    from finess_b200.solver import Solver
    W, z = load_indicator()
    sizes = [(301, 300), (256, 333), (280, 322), (333, 257), (96, 402), (401, 64)]   # about 2300 tiles
    probs = []
    for k, (mx, my) in enumerate(sizes):
        rng = np.random.default_rng(k)
        p = P.riemann_params(n=mx, weno=weno)
        p.my, p.yhigh, p.precision = my, my / mx, FIN_PREC_HYBRID
        q = P.random_riemann_state(p, rng) * (1.0 + 0.02 * rng.standard_normal((mx + 2 * p.mbc, my + 2 * p.mbc, 1)))
        probs.append((p, q, first_dt(p, q)))
    tend = 3.5 * min(dt for _, _, dt in probs)
    with Batch([p for p, _, _ in probs]) as b:
        b.set_indicator(W, z, 2, 1e-3, 2)
        for k, (_, q, _) in enumerate(probs):
            b.set_state(k, q)
        _, steps = b.solve(tend, [dt for _, _, dt in probs])
        got = [b.get_state(k)[0] for k in range(len(probs))]
    for k, (p, q, dt) in enumerate(probs):
        with Solver(p) as s:
            s.set_indicator(W, z, 2, 1e-3, 2)
            s.set_state(q)
            _, n = s.FinSolveRK(tend, [0.0, dt, p.max_dt])
            ref, _ = s.get_state()
        assert n == steps[k]
        assert rel_linf(interior(p, got[k]), interior(p, ref)) <= 1e-5
