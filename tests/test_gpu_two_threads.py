"""Plans applied from two host threads at once, each thread with a plan and a stream of its own: the
limit on a kernel's dynamic shared memory belongs to the kernel, so no plan's launch may lower it under
another's. Every apply has to succeed, and the last ones give the plan's own serial result (forward bit
for bit, adjoint to the round-off of its atomic additions)."""
import ctypes
import threading

import numpy as np
import pytest

from helpers import cap_points, cn, rel, to_dev, to_host

pytestmark = pytest.mark.gpu

APPLIES = 4000


def apply_from_two_threads(pf, O, plans, seed):
    import importlib

    import torch
    lib = importlib.import_module("pfsht_b200._lib").load()
    rng = np.random.default_rng(seed)
    work = []
    for p in plans:
        alm, g = to_dev(O.rand_alm(p.lmax, rng=rng)[:, :, 0]), to_dev(cn(rng, p.npts))
        f, a = pf.zeros_field(p.npts, device="cuda"), pf.zeros_alm(p.lmax, device="cuda")
        work.append((p, alm, g, f, a, torch.cuda.Stream(), to_host(p * alm), to_host(p.H * g)))
    torch.cuda.synchronize()
    failed, start = [0] * len(work), threading.Barrier(len(work))

    def loop(k):
        # the library's own calls, which hold no interpreter lock
        p, alm, g, f, a, stream, _, _ = work[k]
        s, h = ctypes.c_void_p(stream.cuda_stream), p._h
        fwd = [ctypes.c_void_p(t.data_ptr()) for t in (alm, f)]
        adj = [ctypes.c_void_p(t.data_ptr()) for t in (g, a)]
        start.wait(timeout=60)
        for i in range(APPLIES):
            failed[k] += lib.pfsht_forward(h, *fwd, s) != 0
            if i % 8 == 0:
                failed[k] += lib.pfsht_adjoint(h, *adj, s) != 0
            if i % 64 == 0:
                stream.synchronize()
        stream.synchronize()

    threads = [threading.Thread(target=loop, args=(k,)) for k in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == [0] * len(work)
    for p, alm, g, f, a, stream, f0, a0 in work:
        assert np.array_equal(to_host(f), f0)
        assert rel(to_host(a), a0) < 1e-11


@pytest.mark.parametrize("sizes", [[(64, 0.6, "minimal"), (700, 0.3, "minimal")],      # 7 and 18 KB a block
                                   [(64, 0.6, "minimal"), (300, 0.3, (3200, 1280))]])  # 7 and 100 KB
def test_column_kernels(pf, O, cuda, sizes):
    rng = np.random.default_rng(1)
    plans = [pf.Plan(*cap_points(1500, theta_star=t, rng=rng), lmax=L, tol=1e-8, method="stretch", fft_lengths=n)
             for L, t, n in sizes]
    apply_from_two_threads(pf, O, plans, 2)


# interpolation tiles of 57 and 110 KB
@pytest.mark.parametrize("rows", [(100, 200)])
def test_interpolation_tiles(pf, O, cuda, rows):
    rng = np.random.default_rng(3)
    plans = [pf.Plan(*cap_points(1500, theta_star=0.35, rng=rng), lmax=256, tol=1e-8, method="stretch",
                     fft_lengths="minimal", bin_rows=r) for r in rows]
    apply_from_two_threads(pf, O, plans, 4)
