"""The forward ring pass with an order's degrees split over a block's warps (csrc/ring.cu), every ring
column against the oracle's ring pass at the ring parity bound (1e-11 of the largest value): band limits
on both sides of one to four pieces of 64 degrees, several transforms, both precisions (the mixed
form's forward ring pass is FP64 too), tiles with one to four rings a lane."""
import numpy as np
import pytest

from helpers import cap_points, plan_grid, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [40, 66, 67, 130, 131, 194, 195, 258, 259, 400])
@pytest.mark.parametrize("B,precision", [(1, "fp64"), (2, "fp64"), (4, "fp64"), (7, "fp64"), (1, "mixed"), (5, "mixed")])
def test_ring_columns(pf, O, cuda, L, B, precision):
    rng = np.random.default_rng(L + B)
    tol = 1e-6 if precision == "mixed" else 1e-8
    th, ph = cap_points(300, theta_star=1.2, rng=rng)
    p = pf.Plan(th, ph, lmax=L, tol=tol, ntrans=B, precision=precision, method="stretch", fft_lengths="minimal")
    assert p.info["kind"] == "pole" and p.info["precision"] == (1 if precision == "mixed" else 0)
    S = O.Stretch(th, ph, L, tol, nufft="es", nufft_grid=plan_grid(p), ntrans=B)
    alm = O.rand_alm(L, ntrans=B, rng=rng)
    n = p.info["nrings"]
    G = to_dev(np.zeros((n, 2 * L + 1, B), np.complex128, order="F"))
    pf.ring_forward(p, to_dev(alm), G)
    assert rel(to_host(G), S.rings.rings_from_alm(alm)) < 1e-11
