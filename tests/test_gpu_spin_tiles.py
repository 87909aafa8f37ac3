"""Spin plans small enough for ring tiles of 32 or 64 rings against the same plan with tiles of 128
(what a deterministic plan keeps): both directions, degree counts that are and are not whole blocks
of 16, and the exact-transpose identity."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("L,n,spin,B", [(33, 200, 1, 1), (160, 2500, 2, 1), (239, 3000, -2, 3), (500, 9000, 2, 1),
                                        (700, 9000, 2, 2)])
def test_tiles_agree(pf, O, cuda, L, n, spin, B):
    rng = np.random.default_rng(17 + L)
    th, ph = 0.5 * np.sqrt(rng.random(n)), 2 * np.pi * rng.random(n)
    tol = 1e-8
    small = pf.Plan(th, ph, lmax=L, tol=tol, ntrans=B, spin=spin)
    large = pf.Plan(th, ph, lmax=L, tol=tol, ntrans=B, spin=spin, deterministic=True)
    gen = torch.Generator(device="cuda").manual_seed(3)

    def rand(x):
        return x.copy_(torch.randn(x.shape, dtype=torch.complex128, device="cuda", generator=gen))

    alm, g = rand(pf.zeros_alm(L, B)), rand(pf.zeros_field(n, B))
    out = []
    for p in (small, large):
        f, a = pf.zeros_field(n, B), pf.zeros_alm(L, B)
        p.mul(f, alm)
        p.mul_adjoint(a, g)
        torch.cuda.synchronize()
        out.append((f, a))
    # sums of at most 2 L terms in another order
    assert _rel(out[0][0], out[1][0]) < 1e-12
    assert _rel(out[0][1], out[1][1]) < 1e-12
    # rows l < max(|m|, |s|) of the adjoint are zero, so the full products are the identity's sides
    f, a = out[0]
    lhs = torch.sum(f.conj() * g).item()
    rhs = torch.sum(alm.conj() * a).item()
    assert abs(lhs - rhs) < 1e-11 * float(f.norm() * g.norm())
