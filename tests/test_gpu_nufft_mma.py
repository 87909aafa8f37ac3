"""The NUFFT passes on the FP64 matrix instruction (csrc/nufft_mma.cu) at the edges of their tiles:
every kernel width, groups and items that are full, partial or single points, dense and sparse
strips, longitudes at the grid's seam, grids whose rows wrap. They are compared with the bins'
kernels (the deterministic option) on the same grid, whose sums have the same terms in another
order: at most a few hundred terms of one magnitude each, so 1e-13 of the largest value."""
import numpy as np
import pytest

from helpers import cap_points, cn, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


def _tol(w):
    return 1.0001 * 10.0 ** (1 - w)


def _compare(pf, O, th, ph, L, w, B=1, seed=0, **kw):
    rng = np.random.default_rng(seed)
    kw = dict(lmax=L, tol=_tol(w), ntrans=B, fft_lengths="minimal", method="stretch", **kw)
    new, old = pf.Plan(th, ph, **kw), pf.Plan(th, ph, deterministic=True, **kw)
    assert new.info["nufft_w"] == w and plan_sizes(new) == plan_sizes(old)
    alm = O.rand_alm(L, ntrans=B, rng=rng)
    alm = alm if B > 1 else alm[:, :, 0]
    g = np.asfortranarray(cn(rng, len(th), B)) if B > 1 else cn(rng, len(th))
    f1, f2 = to_host(new * to_dev(alm)), to_host(old * to_dev(alm))
    assert np.max(np.abs(f1 - f2)) <= 1e-13 * np.max(np.abs(f2))
    a1, a2 = to_host(new.H * to_dev(g)), to_host(old.H * to_dev(g))
    assert O.alm_reldiff(a1, a2, L) < 1e-13


def plan_sizes(p):
    return [p.info[k] for k in ("nf1", "nf2", "row0", "nrows", "ncols")]


@pytest.mark.parametrize("w", range(4, 17))
def test_every_width(pf, O, cuda, w):
    rng = np.random.default_rng(w)
    _compare(pf, O, *cap_points(5003, rng=rng), 200, w)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 31, 33, 257])
@pytest.mark.parametrize("w", [9, 11])
def test_few_points(pf, O, cuda, w, M):
    # one point, one group, a group and a point, one batch and more; the cap's rim fixes the geometry
    rng = np.random.default_rng(M)
    th, ph = cap_points(M, rng=rng)
    th[0] = 0.349
    _compare(pf, O, th, ph, 300, w)


@pytest.mark.parametrize("w,B", [(9, 1), (11, 3), (16, 1)])
def test_crowded_cells_and_the_seam(pf, O, cuda, w, B):
    # 3,000 points in one cell (one strip is many items), a ring of points, longitudes around 0
    rng = np.random.default_rng(8)
    th = np.concatenate([np.full(3000, 0.3) + 1e-6 * rng.random(3000), np.full(2000, 0.2),
                         0.349 * np.sqrt(rng.random(500))])
    ph = np.concatenate([np.full(3000, 1.0) + 1e-6 * rng.random(3000), 2 * np.pi * rng.random(2000),
                         np.where(rng.random(500) < 0.5, 1e-9 * rng.random(500), 2 * np.pi - 1e-3 * rng.random(500))])
    _compare(pf, O, th, ph, 256, w, B=B)


@pytest.mark.parametrize("w,bin_rows,bin_cols", [(9, 1, 0), (11, 5, 2), (13, 0, 1)])
def test_item_shapes(pf, O, cuda, w, bin_rows, bin_cols):
    rng = np.random.default_rng(3)
    _compare(pf, O, *cap_points(4001, rng=rng), 200, w, bin_rows=bin_rows, bin_cols=bin_cols)


@pytest.mark.parametrize("w", [2, 9, 12, 16])
@pytest.mark.parametrize("n1,n2", [(1, 1), (3, 40), (41, 2), (64, 64)])
def test_wrapping_rows(pf, O, cuda, n1, n2, w):
    # the NUFFT seam keeps every fine row, so windows wrap in both dimensions; small grids are
    # narrower than a window. Against the direct sum, to the kernel's own error (200 tol, the
    # reference's bound)
    rng = np.random.default_rng(n1 + n2)
    M, tol = 300, _tol(w)
    x, y = 2 * np.pi * rng.random(M), 2 * np.pi * rng.random(M)
    c = np.asfortranarray(cn(rng, n1, n2))
    out = to_dev(np.zeros(M, np.complex128))
    pf.NUFFT(2, n1, n2, 1, x, y, tol).exec(to_dev(c), out)
    assert rel(to_host(out), O.nufft_direct(2, n1, n2, 1, x, y, c)[:, 0]) < 200 * tol
    v = cn(rng, M)
    modes = to_dev(np.zeros((n1, n2), np.complex128, order="F"))
    pf.NUFFT(1, n1, n2, -1, x, y, tol).exec(to_dev(v), modes)
    assert rel(to_host(modes), O.nufft_direct(1, n1, n2, -1, x, y, v)[:, :, 0]) < 200 * tol
