"""The Direct leaf's applies with the points' phases inside the ring passes (csrc/ring.cu): one point to
several tiles, one order to several groups, one to seven transforms, poles and repeated longitudes.
Against the oracle's Direct sum at the Direct leaf's bounds (1e-12 of the largest value; dot test)."""
import numpy as np
import pytest

from helpers import cn, dot_rel, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,M,B", [(0, 1, 1), (1, 33, 1), (40, 1, 2), (17, 31, 3), (64, 129, 1), (65, 300, 7),
                                   (200, 1025, 1), (90, 5000, 4), (33, 20000, 2)])
def test_direct_apply(pf, O, cuda, L, M, B):
    rng = np.random.default_rng(L + M)
    th, ph = np.arccos(1 - 2 * rng.random(M)), 7 * rng.random(M) - 1
    if M > 3:
        th[:2], th[2], ph[3] = 1e-9, np.pi - 1e-9, ph[0]  # (the oracle has no value at a pole itself)
    p = pf.Plan(th, ph, lmax=L, ntrans=B, method="direct")
    alm = O.rand_alm(L, ntrans=B, rng=rng)
    g = np.asfortranarray(cn(rng, M, B))
    a_in, g_in = (alm, g) if B > 1 else (np.asfortranarray(alm[:, :, 0]), g[:, 0])
    f, a = to_host(p * to_dev(a_in)), to_host(p.H * to_dev(g_in))
    D = O.Direct(th, ph, L, B)
    assert rel(f.reshape(M, B, order="F"), D.forward(alm)) < 1e-12
    assert O.alm_reldiff(a.reshape(alm.shape, order="F"), D.adjoint(g), L) < 1e-12
    assert dot_rel(f, g_in, a_in, a) < 1e-12
    assert np.array_equal(f, to_host(p * to_dev(a_in)))  # a fixed order of sums
