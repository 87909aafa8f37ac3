"""The order of a batch's ring items (by classes of cost, plan by plan within a class): a few plans and
many, of every kind that a batch merges (one and several transforms, FP64 and mixed, Direct, a given
segment length, none, deterministic), against the same plans applied one by one."""
import numpy as np
import pytest

from helpers import cap_points, rel

pytestmark = pytest.mark.gpu

SPECS = [  # (lmax, cap, ntrans, keywords)
    (300, 0.35, 4, {}), (257, 0.3, 1, {}), (512, 0.3, 2, dict(precision="mixed", tol=1e-6)),
    (130, 0.5, 3, dict(segment_degrees=64)), (200, 0.4, 2, dict(segment_degrees=-1)),
    (256, 0.35, 1, dict(deterministic=True)), (90, 0.5, 2, dict(method="direct")), (400, 0.35, 7, {})]


@pytest.mark.parametrize("copies", [0, 1, 5])
def test_order(pf, O, cuda, copies):
    import torch
    torch.manual_seed(copies)
    rng = np.random.default_rng(copies)
    plans = []
    for L, cap, B, kw in (SPECS * copies if copies else SPECS[1:2] + SPECS[3:5]):
        th, ph = cap_points(700, theta_star=cap, rng=rng)
        plans.append(pf.Plan(th, ph, lmax=L, ntrans=B, fft_lengths="minimal", **{"tol": 1e-8, **kw}))
    batch = pf.Batch(plans, nstreams=4)
    alms = [pf.zeros_alm(p.lmax, p.ntrans, device=cuda) for p in plans]
    fins = [pf.zeros_field(p.npts, p.ntrans, device=cuda) for p in plans]
    for t in alms + fins:
        t.real.normal_()
        t.imag.normal_()
    fb = [pf.zeros_field(p.npts, p.ntrans, device=cuda) for p in plans]
    ab = [pf.zeros_alm(p.lmax, p.ntrans, device=cuda) for p in plans]
    batch.forward(fb, alms)
    batch.adjoint(ab, fins)
    torch.cuda.synchronize()
    for p, a, f, fbi, abi in zip(plans, alms, fins, fb, ab):
        # sums of up to 512 terms in another order (512 x 1.1e-16 of the largest), or the mixed form's
        # FP32 spreading with its atomic additions in another order
        tol = 2e-6 if p.info["precision"] == 1 else 1e-12
        assert rel(fbi.cpu().numpy(), (p * a).cpu().numpy()) < 1e-12, p
        assert O.alm_reldiff(abi.cpu().numpy(), (p.H * f).cpu().numpy(), p.lmax) < tol, p
