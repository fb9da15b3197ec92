"""The measured cases: calls that a user's program makes, over the sizes and options in use.

A case names a call of the public API, the point cloud, the size, the wavenumber, the
order and the leaf size. ``prepare`` builds what the program keeps (plans, charges,
moved positions), ``run`` is one call, ``exact`` the O(N^2) sum of the same problem in
64 bits by plain torch, ``work`` the operations and bytes the call cannot do without.
"""
import math

import numpy as np
import torch

import hfmm_b200
from hfmm_b200.batch import Batch
from hfmm_b200.kernels import LAPLACE, yukawa
from hfmm_b200.learned import AutoPlan

# the O(N^2) sum of a larger cloud takes more than about 20 seconds
EXACT_PAIRS = 3.0e11


def _case(name, call, **kw):
    c = dict(call=call, cloud="uniform", n=1000, k=1.0, p=4, leaf=64, mixed=False, compress=0.0,
             cplx=True, targets=0, problems=1, tol=0.0)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: the default order and leaf size on a few hundred points with
        # real charges (the reference's own check grid); latency and launches count
        _case("tiny_default", "evaluate", n=256, k=1.0, p=4, leaf=16, cplx=False),
        # the plain FP64 path at the CPU-runnable configuration: 20,000 points, one
        # wavelength across the cube, order 8, potential and field
        _case("fp64_20k_p8", "evaluate_field", n=20000, k=2 * math.pi, p=8, leaf=64),
        # the plain path at the conservative order of a 1e-6 tolerance
        _case("fp64_20k_p12", "evaluate_field", n=20000, k=10.0, p=12, leaf=64),
        # potential alone of real charges, the reference's evaluate, at an odd size
        _case("fp64_real_100k_p6", "evaluate", n=100003, k=5.0, p=6, leaf=64, cplx=False),
        # plain FP64 at the headline's size and the lowest order that meets its tolerance
        _case("fp64_1m_p8", "evaluate_field", n=1000000, k=10.0, p=8, leaf=64),
        # an adaptive tree in FP64: half the points on a sphere, half in eight clusters
        _case("fp64_adaptive_60k_p6", "evaluate_field", cloud="adaptive", n=60000, k=12.0, p=6, leaf=64),
        # the mixed-precision evaluate with the low-rank M2L, the headline's order and leaf
        # size: a full depth-5 tree
        _case("mixed_500k_p8", "evaluate_field", n=500000, k=10.0, p=8, leaf=64, mixed=True, compress=1e-7),
        # the same on a sphere and clusters: all four interaction lists are long
        _case("mixed_adaptive_200k_p8", "evaluate_field", cloud="adaptive", n=200000, k=20.0, p=8, leaf=128,
              mixed=True, compress=1e-7),
        # moving points: the plan's tree and lists rebuilt in place, then an evaluate
        _case("moving_100k_p6", "moving", n=100000, k=5.0, p=6, leaf=64, mixed=True, compress=1e-6),
        # the certified front door from host arrays to host arrays, order picked by the network
        _case("auto_250k_tol1e-5", "auto", n=250000, k=10.0, tol=1e-5),
        # uneven problems in one graph launch
        _case("batch_4x50k_p6", "batch", n=50000, k=8.0, p=6, leaf=64, mixed=True, compress=1e-6, problems=4),
        # the FP64 direct sum that certifies an evaluate of a million points
        _case("referee_1m_x1024", "direct_at", n=1000000, k=10.0, targets=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _wave(rng, p):
    """A wavenumber that order p resolves on a unit cube."""
    return round(rng.uniform(0.5, 3.0 if p <= 4 else 8.0 if p <= 6 else 25.0), 3)


def draw(rng):
    call = rng.choice(["evaluate", "evaluate_field", "evaluate_field", "mixed", "mixed", "mixed",
                       "moving", "auto", "batch", "direct_at", "kernel"])
    if call in ("evaluate", "evaluate_field"):
        p = rng.choice([3, 4, 5, 6, 7, 8, 8, 9, 10])
        n = _log(rng, 200, 250000 if p <= 8 else 60000)
        return _case(None, call, cloud=rng.choice(["uniform", "uniform", "adaptive"]) if n > 2000 and p <= 8 else "uniform",
                     n=n, k=_wave(rng, p), p=p, leaf=rng.choice([32, 64, 64, 128]), cplx=call == "evaluate_field")
    if call == "mixed":
        p = rng.choice([6, 7, 8, 8, 9])
        return _case(None, "evaluate_field", cloud=rng.choice(["uniform", "uniform", "adaptive"]),
                     n=_log(rng, 10000, 400000), k=_wave(rng, p), p=p, leaf=rng.choice([64, 64, 128]),
                     mixed=True, compress=1e-7, cplx=rng.random() < 0.8)
    if call == "moving":
        p = rng.choice([4, 5, 6, 7])
        mixed = p >= 6 and rng.random() < 0.6
        return _case(None, "moving", n=_log(rng, 5000, 200000), k=_wave(rng, p), p=p, leaf=64,
                     mixed=mixed, compress=1e-6 if mixed else 0.0)
    if call == "auto":
        return _case(None, "auto", n=_log(rng, 50000, 300000), k=round(rng.uniform(1.0, 20.0), 3),
                     tol=rng.choice([1e-3, 1e-4, 1e-5]))
    if call == "batch":
        p = rng.choice([5, 6, 7])
        return _case(None, "batch", n=_log(rng, 5000, 60000), k=_wave(rng, p), p=p, leaf=64, mixed=p >= 6,
                     compress=1e-6 if p >= 6 else 0.0, problems=rng.choice([2, 3, 4, 5]))
    if call == "direct_at":
        return _case(None, "direct_at", n=_log(rng, 5000, 1000000), k=round(rng.uniform(0.5, 40.0), 3),
                     targets=_log(rng, 64, 4096), cplx=rng.random() < 0.7)
    # the screened-Coulomb kernel, or Laplace where the screening is zero
    return _case(None, "kernel", n=_log(rng, 500, 150000), k=rng.choice([0.0, round(rng.uniform(0.5, 8.0), 3)]),
                 p=rng.choice([4, 5, 6, 7]), leaf=64, cplx=False)


def _points(rng, cloud, n):
    if cloud == "uniform":
        return rng.uniform(0.0, 1.0, (n, 3))
    h = n // 2
    d = rng.normal(size=(h, 3))
    sphere = 0.5 + 0.5 * d / np.linalg.norm(d, axis=1, keepdims=True)
    centres = rng.uniform(0.1, 0.9, (8, 3))
    clusters = centres[rng.integers(0, 8, n - h)] + 0.03 * rng.normal(size=(n - h, 3))
    return np.concatenate([sphere, clusters])


def _charges(rng, n, cplx):
    q = rng.normal(size=n)
    return q + 1j * rng.normal(size=n) if cplx else q


def _sizes(case):
    """The sizes and wavenumbers of a batch's problems: uneven, the first the largest."""
    return [(max(64, int(case["n"] * (1.0 - 0.23 * i)) - 7 * i), case["k"] * (1.0 - 0.15 * i))
            for i in range(case["problems"])]


def _inputs(case, seed):
    """Points and charges of each problem of the case, and the check targets."""
    rng = np.random.default_rng([seed, case["n"]])
    sizes = _sizes(case) if case["call"] == "batch" else [(case["n"], case["k"])]
    out = []
    for n, k in sizes:
        x = _points(rng, case["cloud"], n)
        q = _charges(rng, n, case["cplx"])
        if case["call"] == "moving":   # where the points move to, inside the unit cube
            start, x = x, np.clip(x + rng.normal(scale=0.01, size=(n, 3)), 0.0, 1.0)
        else:
            start = x
        out.append((start, x, q, k))
    targets = np.sort(rng.choice(case["n"], size=min(case["targets"], case["n"]), replace=False)).astype(np.int32)
    return out, targets


def prepare(case, seed):
    probs, targets = _inputs(case, seed)
    start, x, q, k = probs[0]
    call, p, leaf = case["call"], case["p"], case["leaf"]
    comp = case["compress"] or None
    prec = hfmm_b200.PREC_MIXED if case["mixed"] else hfmm_b200.PREC_FP64
    s = dict(call=call, prec=prec)
    if call == "auto":
        s["plan"] = AutoPlan(x, k, tol=case["tol"])
        s["q"] = q                       # host charges: the copies are part of the call
        return s
    dev = lambda a: torch.as_tensor(a).cuda()
    if call == "batch":
        states = [hfmm_b200.setup(xi, ki, p=p, N_max=leaf, m2l_compress=comp) for _, xi, _, ki in probs]
        s["batch"] = Batch(states, n_streams=4)
        s["batch"].bind([dev(qi) for _, _, qi, _ in probs], field=True, precision=prec)
        return s
    s["q"] = dev(q)
    if call == "kernel":
        spec = yukawa(k) if k > 0 else LAPLACE
        s["state"] = hfmm_b200.kernel_setup(x, spec, p=p, N_max=leaf)
        return s
    if call == "moving":
        depth = max(2, math.ceil(math.log(max(case["n"] / leaf, 1.0), 8)))
        s["state"] = hfmm_b200.setup(start, k, p=p, N_max=leaf, max_depth=depth, m2l_compress=comp,
                                     domain=((0.0, 0.0, 0.0), 1.0))
        s["x"] = dev(x)
        return s
    s["state"] = hfmm_b200.setup(x, k, p=p, N_max=leaf, m2l_compress=comp)
    if call == "direct_at":
        s["q_re"] = s["q"].real.contiguous() if case["cplx"] else s["q"]
        s["q_im"] = s["q"].imag.contiguous() if case["cplx"] else None
        s["targets"] = dev(targets)
    return s


def run(s):
    call = s["call"]
    if call == "evaluate":
        return hfmm_b200.evaluate(s["state"], s["q"], s["prec"])
    if call == "evaluate_field":
        return hfmm_b200.evaluate_field(s["state"], s["q"], s["prec"])
    if call == "moving":
        hfmm_b200.rebuild(s["state"], s["x"])
        return hfmm_b200.evaluate_field(s["state"], s["q"], s["prec"])
    if call == "auto":
        return s["plan"].evaluate_field(s["q"])
    if call == "batch":
        s["batch"].launch()
        return s["batch"].outputs
    if call == "direct_at":
        return hfmm_b200.direct_at(s["state"], s["q_re"], s["q_im"], s["targets"], field=True)
    return hfmm_b200.kernel_evaluate(s["state"], s["q"])


def _weights(d2, k, real, field):
    """Kernel and field weights of a block of squared distances; a point has none on itself."""
    ir = torch.where(d2 > 0, torch.rsqrt(d2), torch.zeros((), dtype=d2.dtype, device=d2.device))
    kr = (d2 * ir).mul_(k)
    if real:
        w = torch.exp(-kr).mul_(ir).div_(4 * math.pi)
        return w, (w * (1.0 + kr) * ir * ir if field else None)
    w = torch.polar(ir, kr)
    return w, (w * torch.complex(ir * ir, ir * -k) if field else None)


def _sum(x, q, k, real, field, targets=None):
    """sum_j q_j G(|x_i - x_j|) and the field -grad of it, in 64 bits; the kernel is
    symmetric, so a block of pairs serves its rows and its columns."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.as_tensor(x, device=dev) - 0.5
    q = torch.as_tensor(q, device=dev)
    q = q.double() if real else q.to(torch.complex128)
    qx = torch.cat([q[:, None], q[:, None] * x], 1) if field else None
    t = None if targets is None else torch.as_tensor(targets, device=dev).long()
    y = x if t is None else x[t]
    phi = torch.zeros(len(y), dtype=q.dtype, device=dev)
    acc = torch.zeros((len(y), 4), dtype=q.dtype, device=dev) if field else None
    rows, cols = 4096, 4096
    for i in range(0, len(y), rows):
        a = slice(i, min(i + rows, len(y)))
        for j in range(0 if t is not None else i, len(x), cols):
            b = slice(j, min(j + cols, len(x)))
            d2 = None
            for c in range(3):
                d = y[a, c, None] - x[None, b, c]
                d2 = d * d if d2 is None else d2.addcmul_(d, d)
            w, f = _weights(d2, k, real, field)
            phi[a] += w @ q[b]
            if field:
                acc[a] += f @ qx[b]
            if t is None and j > i:
                phi[b] += w.T @ q[a]
                if field:
                    acc[b] += f.T @ qx[a]
    return phi, (y * acc[:, :1] - acc[:, 1:] if field else None)


def exact(case, seed):
    probs, targets = _inputs(case, seed)
    call = case["call"]
    if sum(float(len(x)) ** 2 for _, x, _, _ in probs) > EXACT_PAIRS and call != "direct_at":
        return None
    if call == "batch":
        return [_sum(x, q, k, False, True) for _, x, q, k in probs]
    _, x, q, k = probs[0]
    if call == "direct_at":
        return _sum(x, q, k, False, True, targets)
    if call in ("evaluate", "kernel"):
        return _sum(x, q, k, call == "kernel", False)[0]
    return _sum(x, q, k, False, True)


def work(case):
    """Charges and positions in, results out; near pairs at the leaf size the points have
    (27 boxes around a point), the surface sums of every point, and one multiply-add per
    surface value, column and one of 189 translations a box."""
    n = float(case["n"])
    if case["call"] == "direct_at":
        return {"bytes": 40.0 * n + 64.0 * case["targets"], "flops": 40.0 * n * case["targets"]}
    ns = [float(m) for m, _ in _sizes(case)] if case["call"] == "batch" else [n]
    p = case["p"] if case["call"] != "auto" else 4 + max(0, round(-math.log10(case["tol"])) - 3)
    surf = 6 * p * p - 12 * p + 8
    cols = 2 if case["cplx"] else 1
    nbytes = flops = 0.0
    for m in ns:
        depth = max(2, math.ceil(math.log(max(m / case["leaf"], 1.0), 8)))
        boxes = 8.0 ** depth
        nbytes += m * (24 + 8 * cols + (16 if case["call"] in ("evaluate", "kernel") else 64))
        flops += 30.0 * 27 * m * max(1.0, m / boxes) + 2 * 30.0 * m * surf + boxes * surf * 189 * 4 * cols
    return {"bytes": nbytes, "flops": flops}
