"""solve! keeps its workspace with the plan: solves of every mode one after the other on one plan, with
and without weights, equal the first solve of a fresh plan (to the solver tests' 1e-9: the adjoint's
atomic additions differ at round-off), and a zero field or no iterations leave zeros."""
import numpy as np
import pytest

from helpers import cap_points, cn, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,B", [(128, 1), (96, 3)])
def test_solves_in_a_row(pf, O, cuda, L, B):
    rng = np.random.default_rng(L)
    th, ph = cap_points(4001, rng=rng)
    kw = dict(lmax=L, tol=1e-8, ntrans=B, fft_lengths="minimal")
    f = np.asfortranarray(cn(rng, len(th), B)) if B > 1 else cn(rng, len(th))
    w = rng.random(len(th)) + 0.5
    prior = [1.0 / (1 + l) ** 2 for l in range(L + 1)]
    kept = pf.Plan(th, ph, **kw)
    for mode, kws in [("cg", {}), ("wiener", dict(prior=prior, w=w)), ("cg", dict(w=w)), ("minnorm", {}), ("cg", {})]:
        run = lambda p: pf.solve(pf.zeros_alm(L, B), p, to_dev(f), mode=mode, rtol=1e-14, maxiter=5, **kws)  # noqa: E731
        (a, ia), (b, ib) = run(kept), run(pf.Plan(th, ph, **kw))
        assert ia["iters"] == ib["iters"] == 5
        assert rel(to_host(a), to_host(b)) < 1e-9 and abs(ia["relres"] - ib["relres"]) < 1e-9 * ib["relres"]
    a, info = pf.solve(pf.zeros_alm(L, B), kept, to_dev(0 * f), maxiter=5)
    assert info["iters"] == 0 and info["relres"] == 0.0 and not to_host(a).any()
    a, info = pf.solve(pf.zeros_alm(L, B), kept, to_dev(f), maxiter=0)
    assert info["iters"] == 0 and not to_host(a).any()
