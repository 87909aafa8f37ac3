"""Timed cases: what a user's program does with this package, through its public entry points.

A pass of an "apply" case is one synthesis mul!(f, plan, alm) and one exact adjoint
mul!(alm, plan', f) on arrays resident on the GPU; "host" does the same on page-locked host
arrays, "batch" on many uneven plans in one Batch, and "solve" runs a few conjugate-gradient
iterations on the normal equations. `prepare` makes the points, the plan, the coefficients and
the field that a program holds before the call.

Sizes are the ones this repository's benchmark and tests use: a 20-degree polar cap with
4 (lmax theta)^2 points at lmax 256, 1024 and 2048, uneven caps of 5 to 30 degrees with up to 8
transforms, off-pole patches, two separate caps, whole-sphere point sets and spin weight 2.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from __graft_entry__ import load_package  # noqa: E402

pf = load_package()

DEV = "cuda"
CAP20 = math.radians(20.0)


def listed():
    """The cases and what each stands for in use."""
    return [
        # a few hundred scattered targets at low band limit: the smallest calls (AUTO answers Direct)
        dict(name="scatter_64", kind="apply", geom="sphere", lmax=64, npts=400),
        # a whole-sky catalogue of about 49,000 points (AUTO answers Direct)
        dict(name="sky_191", kind="apply", geom="sphere", lmax=191, npts=49152),
        # the small benchmark workload
        dict(name="cap_256", kind="apply", geom="cap", lmax=256, npts=31941, tol=1e-8),
        # a survey patch away from the poles at the default tolerance, odd sizes
        dict(name="patch_511", kind="apply", geom="patch", lmax=511, npts=100003),
        # four maps on the same points (the benchmark's middle workload with ntrans = 4)
        dict(name="cap_1024_n4", kind="apply", geom="cap", lmax=1024, npts=511063, tol=1e-8, ntrans=4),
        # the headline workload; the fine-grid lengths that a plan's own timing settles on
        dict(name="cap_2048", kind="apply", geom="cap", lmax=2048, npts=2044253, tol=1e-8,
             nf1=1458, nf2=4096),
        # the same in mixed precision
        dict(name="cap_2048_mixed", kind="apply", geom="cap", lmax=2048, npts=2044253, tol=1e-6,
             precision="mixed", nf1=1458, nf2=4096),
        # a polarisation map: spin 2 on a southern cap
        dict(name="spin_1024", kind="apply", geom="south", lmax=1024, npts=262147, tol=1e-8, spin=2),
        # two fields far apart on the sky (AUTO answers MultiBox)
        dict(name="twocaps_512", kind="apply", geom="twocaps", lmax=512, npts=40000, tol=1e-8),
        # a farm of uneven plans applied together
        dict(name="batch_16", kind="batch", nplans=16, lmax_lo=128, lmax_hi=1024, mix=4),
        # map making: conjugate gradients on the normal equations
        dict(name="solve_384", kind="solve", geom="cap", lmax=384, npts=71868, tol=1e-8, iters=8),
        # maps that live in host memory
        dict(name="host_768", kind="host", geom="cap", lmax=768, npts=131071, tol=1e-8),
    ]


#: most work of a drawn case: multiply-adds of the retained (l, m, ring or point) triples times
#: transforms, and points times transforms
MOST_TRIPLES, MOST_POINTS = 3.2e8, 2.05e6
#: exact() is left out above this many (point, degree, order) steps
EXACT_STEPS = 4.5e10


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above."""
    while True:
        kind = rng.choice(["apply"] * 7 + ["batch", "solve", "host"])
        if kind == "batch":
            return dict(kind="batch", nplans=rng.randint(3, 12), lmax_lo=rng.randint(96, 160),
                        lmax_hi=rng.randint(320, 800), mix=rng.randint(0, 10 ** 6))
        geom = rng.choice(["cap", "cap", "south", "patch", "twocaps", "sphere"])
        if geom == "sphere":
            lmax, npts = _log_int(rng, 32, 512), _log_int(rng, 100, 60000)
        else:
            lmax = _log_int(rng, 128, 2048)
            npts = _log_int(rng, max(200, 0.02 * lmax * lmax), max(2000, 0.5 * lmax * lmax))
        if kind in ("solve", "host"):
            lmax, npts = min(lmax, 1024), min(npts, 300000)
        c = dict(kind=kind, geom=geom, lmax=lmax, npts=npts,
                 tol=rng.choice([1e-4, 1e-6, 1e-8, 1e-8, 1e-10, 1e-12]),
                 extent=round(rng.uniform(5.0, 30.0), 2))
        if kind == "solve":
            c.update(geom=rng.choice(["cap", "patch"]), iters=rng.randint(2, 8), tol=1e-8)
        else:
            c["ntrans"] = rng.choice([1, 1, 1, 2, 3, 4, 7])
            if kind == "apply" and rng.random() < 0.2:
                c["spin"] = rng.choice([1, 2, -2])
            elif c["tol"] >= 1e-6 and rng.random() < 0.5:
                c["precision"] = "mixed"
        b = c.get("ntrans", 1) * (c.get("iters", 0) + 1) * (2 if c.get("spin") else 1)
        if _triples(c) * b <= MOST_TRIPLES and npts * b <= MOST_POINTS:
            return c


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _extent(case):
    return math.radians(case.get("extent", 20.0))


def _band(gen, n, t0, t1):
    """n colatitudes, area-uniform between t0 and t1."""
    u = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    return torch.acos(math.cos(t0) + (math.cos(t1) - math.cos(t0)) * u)


def _points(case, gen):
    n, geom, e = case["npts"], case["geom"], _extent(case)
    turn = 2 * math.pi * torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    if geom == "cap":
        return _band(gen, n, 0.0, e), turn
    if geom == "south":
        return _band(gen, n, math.pi - e, math.pi), turn
    if geom == "patch":
        return _band(gen, n, 0.7, 0.7 + e), 0.4 + turn * (1.2 * e / (2 * math.pi))
    if geom == "twocaps":
        h = n // 2
        r = min(e, 0.25)
        th = torch.cat([_band(gen, h, 0.0, r), _band(gen, n - h, math.pi - 0.8 * r, math.pi)])
        return th, turn
    return _band(gen, n, 0.0, math.pi), turn


def _alm(lmax, ntrans, spin, gen):
    """complex N(0,1)/(l+1) in the valid slots, zeros in the padding; column-major."""
    nr, nc = lmax + 1, 2 * lmax + 1
    row = torch.arange(nr, device=DEV)[None, :]
    col = torch.arange(nc, device=DEV)[:, None]
    if spin:
        m = (col - lmax).abs()
        l, ok = row.expand(nc, nr), row >= m.clamp(min=abs(spin))
    else:
        m = (col + 1) // 2
        l, ok = row + m, row + m <= lmax
    z = torch.randn(ntrans, nc, nr, 2, generator=gen, device=DEV, dtype=torch.float64)
    a = torch.view_as_complex(z) * (ok / (l + 1.0))
    a = a.permute(2, 1, 0)
    return a[:, :, 0] if ntrans == 1 else a


def _field(npts, ntrans, gen):
    z = torch.randn(ntrans, npts, 2, generator=gen, device=DEV, dtype=torch.float64)
    f = torch.view_as_complex(z).permute(1, 0)
    return f[:, 0] if ntrans == 1 else f


def _plan(case, th, ph):
    tol = case.get("tol", 1e-10)
    if "nf1" in case:
        lengths = (case["nf1"], case["nf2"])
    else:
        # fine-grid lengths fixed by the sizes wherever another length would show in the result
        lengths = "timed" if tol <= 1e-10 else "minimal"
    return pf.Plan(th, ph, lmax=case["lmax"], tol=tol, ntrans=case.get("ntrans", 1),
                   precision=case.get("precision", "fp64"), spin=case.get("spin", 0), fft_lengths=lengths)


def _batch_specs(case):
    """Uneven plans: lmax log-uniform, caps of 5 to 30 degrees, 1 to 8 transforms, half of them
    mixed at tol 1e-6 and half FP64 at 1e-8."""
    r = random.Random(case["mix"])
    out = []
    for k in range(case["nplans"]):
        lmax = _log_int(r, case["lmax_lo"], case["lmax_hi"])
        ext = r.uniform(5.0, 30.0)
        npts = max(64, int(round(4 * (lmax * math.radians(ext)) ** 2)))
        mixed = r.random() < 0.5
        out.append(dict(kind="apply", geom="cap", lmax=lmax, npts=npts, extent=ext, ntrans=r.randint(1, 8),
                        tol=1e-6 if mixed else 1e-8, precision="mixed" if mixed else "fp64"))
    return out


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _inputs(case, gen):
    th, ph = _points(case, gen)
    b = case.get("ntrans", 1)
    return th, ph, _alm(case["lmax"], b, case.get("spin", 0), gen), _field(case["npts"], b, gen)


def _to_pinned(x, out):
    out[...] = x.cpu().numpy()
    return out


def prepare(case, seed):
    gen = _gen(seed)
    if case["kind"] == "batch":
        s = dict(kind="batch", plans=[], alms=[], gs=[], fs=[], outs=[])
        for spec in _batch_specs(case):
            th, ph, alm, g = _inputs(spec, gen)
            s["plans"].append(_plan(spec, th, ph))
            s["alms"].append(alm)
            s["gs"].append(g)
            s["fs"].append(pf.zeros_field(spec["npts"], spec["ntrans"], device=DEV))
            s["outs"].append(pf.zeros_alm(spec["lmax"], spec["ntrans"], device=DEV))
        s["batch"] = pf.Batch(s["plans"])
        return s
    th, ph, alm, g = _inputs(case, gen)
    s = dict(kind=case["kind"], plan=_plan(case, th, ph), alm=alm, g=g)
    b = case.get("ntrans", 1)
    dev = "pinned" if case["kind"] == "host" else DEV
    s["f"], s["out"] = pf.zeros_field(case["npts"], b, device=dev), pf.zeros_alm(case["lmax"], b, device=dev)
    if case["kind"] == "host":
        s["alm"] = _to_pinned(alm, pf.zeros_alm(case["lmax"], b, device="pinned"))
        s["g"] = _to_pinned(g, pf.zeros_field(case["npts"], b, device="pinned"))
    s["iters"] = case.get("iters", 0)
    return s


def run(s):
    """One pass."""
    if s["kind"] == "batch":
        s["batch"].forward(s["fs"], s["alms"])
        s["batch"].adjoint(s["outs"], s["gs"])
        return {"f": s["fs"], "alm": s["outs"]}
    if s["kind"] == "solve":
        alm, info = pf.solve(s["out"], s["plan"], s["g"], mode="cg", rtol=1e-14, maxiter=s["iters"])
        return {"alm": alm, "iters": info["iters"]}
    pf.mul(s["f"], s["plan"], s["alm"])
    pf.mul(s["out"], s["plan"].H, s["g"])
    return {"f": s["f"], "alm": s["out"]}


# ---------------------------------------------------------------------------------------
# work: what one pass cannot do without
# ---------------------------------------------------------------------------------------
def _spans(case):
    e = _extent(case)
    if case["geom"] == "twocaps":
        r = min(e, 0.25)
        return [(0.0, r), (math.pi - 0.8 * r, math.pi)]
    return {"cap": [(0.0, e)], "south": [(math.pi - e, math.pi)], "patch": [(0.7, 0.7 + e)]}[case["geom"]]


def _triples(case):
    """(l, m, ring) triples with l sin(theta) >= m on rings pi / lmax apart; for whole-sphere point
    sets, (l, m, point)."""
    L = case["lmax"]
    if case["geom"] == "sphere":
        return 0.5 * case["npts"] * (L + 1) ** 2
    tot = 0.0
    for a, b in _spans(case):
        for k in range(32):
            s = math.sin(a + (b - a) * (k + 0.5) / 32)
            # orders m <= L s, degrees from m / s to L
            tot += (L * L * s / 2) * (L * (b - a) / math.pi) / 32
    return tot


def work(case):
    if case["kind"] == "batch":
        each = [work(c) for c in _batch_specs(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    L, n, b = case["lmax"], case["npts"], case.get("ntrans", 1)
    coef = 16.0 * (L + 1) ** 2 * b
    field = 16.0 * n * b
    # synthesis reads the coefficients and writes the field, the adjoint the reverse; the
    # points' coordinates are read once in each
    bytes_ = 2 * (coef + field + 16.0 * n)
    # five multiply-adds per triple (two of them per spin order)
    ring = 10.0 * _triples(case) * b * (2 if case.get("spin") else 1)
    flops = ring
    if case["geom"] != "sphere":
        w = math.ceil(1 - math.log10(case.get("tol", 1e-10)))
        flops += 4.0 * (w * w + w) * n * b
    sweeps = case["iters"] + 0.5 if case["kind"] == "solve" else 1
    return {"bytes": bytes_ * sweeps, "flops": 2 * flops * sweeps}


# ---------------------------------------------------------------------------------------
# exact values: the transform's definition in 64 bits, order by order and point by point
# ---------------------------------------------------------------------------------------
def _exact_apply(case, th, ph, alm, g):
    """f = sum a_lm sY_lm at the points and alm = sum conj(sY_lm) g, by the three-term recurrences
    over l of the normalised associated Legendre functions or Wigner d functions."""
    L, spin, B = case["lmax"], case.get("spin", 0), case.get("ntrans", 1)
    alm, g = alm.reshape(L + 1, 2 * L + 1, B), g.reshape(-1, B)
    M = g.shape[0]
    f64 = dict(dtype=torch.float64, device=DEV)
    f = torch.zeros(M, B, dtype=torch.complex128, device=DEV)
    out = torch.zeros_like(alm)
    ms = torch.arange(-L, L + 1, **f64) if spin else torch.arange(0, L + 1, **f64)
    n = -spin
    l0 = torch.maximum(ms.abs(), torch.tensor(float(abs(spin)), **f64)).long()
    # normalisation of the first degree of each order
    lg = torch.lgamma
    if spin:
        j = l0.double()
        # d^j_{m n} with j = max(|m|, |n|): one term of the general sum
        small = torch.where(ms.abs() >= abs(n), torch.full_like(ms, n), ms)
        logc = 0.5 * (lg(2 * j + 1) - lg(j + small + 1) - lg(j - small + 1))
        # power of cos(t/2) is |m + n|, of sin(t/2) is |m - n|
        pc, ps = (ms + n).abs(), (ms - n).abs()
        # d^j_{j n}: (-1)^(j-n); d^j_{-j n}: +; d^j_{m j}: +; d^j_{m -j}: (-1)^(j+m)
        par = torch.where(ms.abs() >= abs(n), torch.where(ms >= 0, ms - n, torch.zeros_like(ms)),
                          torch.where(torch.full_like(ms, n) >= 0, torch.zeros_like(ms), ms - n))
        sgn = 1.0 - 2.0 * (par.long().abs() % 2)
    else:
        # P_mm = (-1)^m sqrt((2m+1)/(4 pi) prod (2k-1)/(2k)) sin^m
        logc = 0.5 * (torch.log((2 * ms + 1) / (4 * math.pi)) + lg(2 * ms + 1.0) - 2 * ms * math.log(2.0)
                      - 2 * lg(ms + 1.0))
        sgn = 1.0 - 2.0 * (ms.long() % 2)
    nm = len(ms)
    LB, CH = 32, max(256, int(2 ** 23 // nm))
    for c0 in range(0, M, CH):
        t = th[c0:c0 + CH]
        P = len(t)
        x = torch.cos(t)[None, :]
        if spin:
            e = torch.special.xlogy(pc[:, None], torch.cos(t / 2).clamp(min=0)[None, :]) + \
                torch.special.xlogy(ps[:, None], torch.sin(t / 2)[None, :])
        else:
            e = torch.special.xlogy(ms[:, None], torch.sin(t)[None, :])
        seed = sgn[:, None] * torch.exp(e + logc[:, None])
        ph_c = torch.exp(1j * ms[:, None] * ph[c0:c0 + CH][None, :])
        gc = g[c0:c0 + CH]
        if spin:
            G = torch.view_as_real(ph_c.conj()[:, :, None] * gc[None]).reshape(nm, P, 2 * B)
        else:
            gp = torch.view_as_real(ph_c.conj()[:, :, None] * gc[None]).reshape(nm, P, 2 * B)
            gm = torch.view_as_real(sgn[:, None, None] * ph_c[:, :, None] * gc[None]).reshape(nm, P, 2 * B)
            G = torch.cat([gp, gm], 2)
        F = torch.zeros(nm, P, G.shape[2], **f64)
        p1, p2 = torch.zeros(nm, P, **f64), torch.zeros(nm, P, **f64)
        blk = torch.zeros(nm, LB, P, **f64)
        tmp = torch.empty(nm, P, **f64)
        for lb in range(0, L + 1, LB):
            nl = min(LB, L + 1 - lb)
            for i in range(nl):
                l = lb + i
                if spin:
                    k = float(l - 1)  # degree l from l - 1 and l - 2
                    if l >= 2:
                        den = torch.sqrt(((l * l) - ms * ms).clamp(min=0) * max(l * l - n * n, 0)) * k
                        ok = (l > l0) & (den > 0)
                        den = torch.where(ok, den, torch.ones_like(den))
                        a1 = torch.where(ok, (2 * k + 1) * k * (k + 1) / den, torch.zeros_like(den))
                        a2 = torch.where(ok, (2 * k + 1) * ms * n / den, torch.zeros_like(den))
                        b = torch.where(ok, (k + 1) * torch.sqrt(((k * k) - ms * ms).clamp(min=0) *
                                                                 max(k * k - n * n, 0)) / den, torch.zeros_like(den))
                        torch.mul(x, a1[:, None], out=tmp)
                        tmp -= a2[:, None]
                        tmp *= p1
                        tmp.addcmul_(p2, -b[:, None])
                    else:
                        tmp.zero_()
                else:
                    d = torch.where(ms < l, (l - ms) * (l + ms), torch.ones_like(ms))
                    a = torch.where(ms < l, torch.sqrt((2 * l - 1.0) * (2 * l + 1.0) / d), torch.zeros_like(ms))
                    b = torch.where(ms < l - 1, torch.sqrt(((2 * l + 1.0) / max(2 * l - 3.0, 1.0) * (l - ms - 1)
                                                            * (l + ms - 1) / d).clamp(min=0)), torch.zeros_like(ms))
                    torch.mul(x, p1, out=tmp)
                    tmp *= a[:, None]
                    tmp.addcmul_(p2, -b[:, None])
                first = (l0 == l).nonzero()[:, 0]
                if len(first):
                    tmp[first] = seed[first]
                p2, p1, tmp = p1, tmp, p2
                blk[:, i].copy_(p1)
                if spin:
                    blk[:, i] *= math.sqrt((2 * l + 1) / (4 * math.pi))
            # coefficients of these degrees, order by order
            A = torch.zeros(nm, nl, G.shape[2], **f64)
            li = torch.arange(lb, lb + nl, device=DEV)[None, :]
            if spin:
                cols = [(torch.arange(nm, device=DEV)[:, None].expand(nm, nl), li.expand(nm, nl), li >= l0[:, None])]
            else:
                mm = torch.arange(nm, device=DEV)[:, None]
                row = (li - mm).clamp(min=0)
                cols = [((2 * mm).expand(nm, nl), row, li >= mm),
                        ((2 * mm - 1).clamp(min=0).expand(nm, nl), row, (li >= mm) & (mm > 0))]
            R = torch.bmm(blk[:, :nl], G)
            for q, (col, row, ok) in enumerate(cols):
                s = sgn[:, None, None] if q == 1 else 1.0
                v = torch.where(ok[:, :, None], alm[row, col], torch.zeros((), dtype=alm.dtype, device=DEV)) * s
                A[:, :, 2 * B * q:2 * B * (q + 1)] = torch.view_as_real(v.contiguous()).reshape(nm, nl, 2 * B)
                w = torch.view_as_complex(R[:, :, 2 * B * q:2 * B * (q + 1)].reshape(nm, nl, B, 2).contiguous())
                out.index_put_((row[ok], col[ok]), w[ok], accumulate=True)
            F += torch.bmm(blk[:, :nl].transpose(1, 2), A)
        for q in range(G.shape[2] // (2 * B)):
            w = torch.view_as_complex(F[:, :, 2 * B * q:2 * B * (q + 1)].reshape(nm, P, B, 2).contiguous())
            e = ph_c if q == 0 else ph_c.conj()
            f[c0:c0 + P] += (w * e[:, :, None]).sum(0)
    return (f[:, 0], out[:, :, 0]) if B == 1 else (f, out)


def _steps(case):
    return float(case["npts"]) * case["lmax"] ** 2 * (2 if case.get("spin") else 1) * \
        (1 + case.get("ntrans", 1)) / 2


def exact(case, seed):
    gen = _gen(seed)
    if case["kind"] == "batch":
        fs, outs, left = [], [], EXACT_STEPS
        for spec in _batch_specs(case):
            x = _inputs(spec, gen)
            f = a = None
            if _steps(spec) <= left:
                f, a = _exact_apply(spec, *x)
                left -= _steps(spec)
            fs.append(f)
            outs.append(a)
        return None if left == EXACT_STEPS else {"f": fs, "alm": outs}
    if case["kind"] == "solve" or _steps(case) > EXACT_STEPS:
        return None
    f, a = _exact_apply(case, *_inputs(case, gen))
    if case["kind"] == "host":
        f, a = f.cpu().numpy(), a.cpu().numpy()
    return {"f": f, "alm": a}
