"""The NUFFT's column stages as one kernel each way (csrc/nufft_cols.cu): every radix and their
products as the Theta and the fine length, odd lengths, one column, ragged column blocks, several
transforms, grids on the library chain's side of the rule. Against the oracle's stretched leaf with the
same fine grid at the device parity bounds (forward 1e-11, adjoint 1e-10 of the largest value)."""
import numpy as np
import pytest

from helpers import cap_points, cn, plan_grid, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,cap,grid,B", [
    (128, 0.35, None, 1),
    (200, 0.35, (343, 640), 1), (200, 0.35, (450, 648), 2), (200, 0.35, (486, 1024), 3), (200, 0.35, (625, 700), 1),
    (300, 0.3, (512, 1280), 1), (300, 0.3, (729, 1280), 1), (300, 0.3, (1024, 1296), 2), (300, 0.3, (1260, 1280), 1),
    (300, 0.3, (2401, 1280), 1), (300, 0.3, (3200, 1280), 1), (300, 0.3, (3300, 1280), 1), (300, 0.3, (1001, 1280), 1),
    (700, 0.3, None, 5)])
def test_lengths(pf, O, cuda, L, cap, grid, B):
    rng = np.random.default_rng(L + B)
    th, ph = cap_points(1500, theta_star=cap, rng=rng)
    p = pf.Plan(th, ph, lmax=L, tol=1e-8, ntrans=B, method="stretch", fft_lengths=grid or "minimal")
    S = O.Stretch(th, ph, L, 1e-8, nufft="es", nufft_grid=plan_grid(p), ntrans=B)
    alm = O.rand_alm(L, ntrans=B, rng=rng)
    g = np.asfortranarray(cn(rng, len(th), B))
    f = to_host(p * to_dev(alm if B > 1 else alm[:, :, 0])).reshape(len(th), B, order="F")
    a = to_host(p.H * to_dev(g if B > 1 else g[:, 0])).reshape(alm.shape, order="F")
    assert rel(f, S.forward(alm)) < 1e-11
    assert O.alm_reldiff(a, S.adjoint(g), L) < 1e-10


@pytest.mark.parametrize("t0,t1", [(0.7, 1.1), (1.3, 1.9), (2.6, 3.14)])
def test_interior_and_southern(pf, O, cuda, t0, t1):
    rng = np.random.default_rng(5)
    L = 250
    th, ph = t0 + (t1 - t0) * rng.random(2001), 0.3 + 0.8 * rng.random(2001)
    p = pf.Plan(th, ph, lmax=L, tol=1e-8, method="stretch", fft_lengths="minimal")
    S = O.Stretch(th, ph, L, 1e-8, nufft="es", nufft_grid=plan_grid(p))
    alm = O.rand_alm(L, rng=rng)
    g = cn(rng, len(th))
    assert rel(to_host(p * to_dev(alm[:, :, 0])), S.forward(alm)[:, 0]) < 1e-11
    assert O.alm_reldiff(to_host(p.H * to_dev(g)), S.adjoint(g[:, None])[:, :, 0], L) < 1e-10
