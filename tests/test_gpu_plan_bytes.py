"""The device memory that a plan reports counts what it took on after its build: a Direct plan's column
array in a batch, a solve's kept workspace, the host staging; and a server's budget goes by that."""
import numpy as np
import pytest

from helpers import cap_points, cn, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 3])
def test_bytes_grow(pf, cuda, B):
    rng = np.random.default_rng(B)
    L, th, ph = 96, *cap_points(2001, rng=rng)
    M, nc = len(th), (L + 1) * (2 * L + 1)
    p = pf.Plan(th, ph, lmax=L, tol=1e-8, ntrans=B, method="direct")
    built = p.workspace_bytes()
    batch = pf.Batch([p])
    columns = 16 * M * (2 * L + 1) * B
    in_batch = p.workspace_bytes()
    assert in_batch == built + columns + 16 * M * B  # and the field that a batch works on
    del batch
    f = to_dev(np.asfortranarray(cn(rng, M, B)) if B > 1 else cn(rng, M))
    pf.solve(pf.zeros_alm(L, B), p, f, maxiter=2)
    solved = p.workspace_bytes()
    assert 0 <= solved - in_batch - 16 * B * (3 * nc + M) < 65536
    # the server takes the plan with what its host copies still need, and not with a byte less
    missing = 16 * B * (2 * nc + M)
    for short in (1, 0):
        server = pf.Server(hbm_budget_gb=(solved + missing - short) / 1e9 * (1 + 1e-15))
        if short:
            with pytest.raises(Exception, match="budget"):
                server.add(p)
        else:
            server.add(p)
        server.close()
    assert p.workspace_bytes() == solved + missing


def test_bytes_of_boxes(pf, cuda):
    rng = np.random.default_rng(7)
    a, b = cap_points(1500, theta_star=0.3, rng=rng), cap_points(1500, theta_star=0.3, rng=rng)
    th, ph = np.concatenate([a[0], np.pi - b[0]]), np.concatenate([a[1], b[1]])
    p = pf.Plan(th, ph, lmax=128, tol=1e-8, method="multibox")
    assert p.info["kind"] == "multibox" and len(p.boxes()) == 2
    built = p.workspace_bytes()
    assert built == p.info["device_bytes"]
    pf.solve(pf.zeros_alm(128, 1), p, to_dev(cn(rng, len(th))), maxiter=2)
    assert 0 <= p.workspace_bytes() - built - 16 * (3 * 129 * 257 + len(th)) < 65536
