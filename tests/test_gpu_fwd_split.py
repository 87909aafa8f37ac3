"""The forward ring pass with an order's degrees split over the warps of a block (csrc/ring.cu): one to
four pieces, orders at the band limit, tiles of one ring and of every lane count, several transforms.
Against the oracle's ring pass at the ring parity bound (1e-11 of the largest value)."""
import numpy as np
import pytest

from helpers import cap_points, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [5, 66, 67, 130, 131, 194, 258, 400])
@pytest.mark.parametrize("B", [1, 2, 4, 7])
def test_split_degrees(pf, O, cuda, L, B):
    # 64-degree pieces begin at l = m + 2 + 64 q: band limits on both sides of 1, 2, 3 and 4 of them
    rng = np.random.default_rng(L + B)
    th, ph = cap_points(600, theta_star=1.2 if L < 60 else 0.6, rng=rng)
    kw = dict(lmax=L, tol=1e-4 if L < 60 else 1e-8, ntrans=B)
    try:
        p = pf.Plan(th, ph, method="stretch", **kw)
    except pf.RefusedGeometry:
        p = pf.Plan(th, ph, method="direct", **kw)
    alm = O.rand_alm(L, ntrans=B, rng=rng)
    f = to_host(p * to_dev(alm if B > 1 else alm[:, :, 0])).reshape(len(th), B, order="F")
    ref = O.Direct(th, ph, L, B).forward(alm)
    assert rel(f, ref) < 10 * kw["tol"]
    # each column is the single plan's, whose rings are tiled otherwise
    one = pf.Plan(th, ph, method=p.info["kind"] if p.info["kind"] == "direct" else "stretch", lmax=L, tol=kw["tol"],
                  fft_lengths=(p.info["nf1"], p.info["nf2"]) if p.info["nf1"] else "minimal")
    for b in range(B):
        f1 = to_host(one * to_dev(np.asfortranarray(alm[:, :, b])))
        assert np.max(np.abs(f1 - f[:, b])) < 1e-11 * np.max(np.abs(f1))
