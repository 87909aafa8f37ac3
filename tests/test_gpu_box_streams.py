"""A MultiBox plan's boxes run on streams of their own, forked from the caller's and joined to it:
several boxes, the adjoint's scratch arrays enough for all of them and fewer than the boxes (16
transforms at lmax 512: one array of 135 MB for two boxes), repeated without a wait in between, on
a stream that is not the default one, and as a captured graph."""
import numpy as np
import pytest
import torch

from helpers import cn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,B", [(512, 1), (512, 16)])
def test_boxes_on_their_streams(pf, O, cuda, L, B):
    rng = np.random.default_rng(91)
    n, r = 400, 0.15
    # caps at the poles and two patches at the equator, which share a box
    cap = r * np.sqrt(rng.random(n))
    th = np.concatenate([cap, np.pi - cap, np.pi / 2 + r * (rng.random(2 * n) - 0.5)])
    ph = np.concatenate([2 * np.pi * rng.random(2 * n), 1.0 + r * rng.random(n), 4.0 + r * rng.random(n)])
    M = len(th)
    p = pf.Plan(th, ph, lmax=L, tol=1e-8, ntrans=B, method="multibox")
    boxes = p.boxes()
    assert len(boxes) == 3
    gen = torch.Generator(device="cuda").manual_seed(5)

    def rand(like):
        x = torch.randn(like.shape, dtype=torch.complex128, device="cuda", generator=gen)
        return like.copy_(x)

    alm, g = rand(pf.zeros_alm(L, B)), rand(pf.zeros_field(M, B))
    fref, aref = pf.zeros_field(M, B), pf.zeros_alm(L, B)
    for b in boxes:
        idx = b["indices"]
        pb = pf.Plan(th[idx], ph[idx], lmax=L, tol=1e-8, ntrans=B, method="stretch",
                     fft_lengths=(b["nf1"], b["nf2"]))
        fb, ab, gb = pf.zeros_field(len(idx), B), pf.zeros_alm(L, B), pf.zeros_field(len(idx), B)
        ti = torch.as_tensor(np.asarray(idx, dtype=np.int64), device="cuda")
        gb.copy_(g[ti])
        pb.mul(fb, alm)
        pb.mul_adjoint(ab, gb)
        fref[ti] = fb
        aref += ab
    f, a = pf.zeros_field(M, B), pf.zeros_alm(L, B)

    def check():
        # the forward is the same arithmetic; the adjoint's sums agree to their order
        torch.cuda.synchronize()
        assert torch.equal(f, fref)
        assert float((a - aref).abs().max() / aref.abs().max()) < 1e-13

    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for _ in range(3):
            f.zero_()
            p.mul(f, alm)
            a.zero_()
            p.mul_adjoint(a, g)
    check()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        p.mul(f, alm)
        p.mul_adjoint(a, g)
    for _ in range(2):
        f.zero_()
        a.zero_()
        graph.replay()
        check()
