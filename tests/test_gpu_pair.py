"""The FP64 pair arithmetic of the particle kernels and the referee (own reciprocal square
root, phase reduction and sine / cosine series) against extended precision: one unit source,
targets at separations over twelve decades, wavenumbers that take the phase from 0 across the
switch to the general form at 1e5. Tolerance: 1 / r and the weights carry a few roundings
(8 eps), and rounding k r moves the phase by eps k r (2 eps k r)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("k", [0.0, 1e-3, 2.5, -7.0, 311.0, 9.0e4, 3.0e6])
def test_single_source(k):
    import torch
    import hfmm_b200
    rng = np.random.default_rng(5)
    n = 4096
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    pos = d * (10.0 ** rng.uniform(-11.0, 1.0, n))[:, None]
    pos[0] = 0.0
    q = np.zeros(n, complex)
    q[0] = 1.0
    st = hfmm_b200.setup(pos, 1.0, p=3, N_max=64, max_depth=2)
    st.k = k   # the referee takes its wavenumber from the state: only it runs here
    phi, E = hfmm_b200.direct(st, q, np.arange(1, n), field=True)
    x = pos[1:].astype(np.longdouble)
    r = np.sqrt((x ** 2).sum(1))
    kr = np.longdouble(k) * r
    w = (np.cos(kr) + 1j * np.sin(kr)) / r
    f = w * (1 - 1j * kr) / r ** 2
    tol = 8 * EPS + 2 * EPS * np.abs(kr)
    assert (np.abs(phi - w) * r < tol).all()
    err = np.abs(E - f[:, None] * x).max(1) * r ** 2 / (1 + np.abs(kr))
    assert (err < 2 * tol).all()
    st.close()


@pytest.mark.parametrize("kappa", [None, 2.0])
@pytest.mark.parametrize("cplx", [False, True])
def test_referee_leaves_out_nan_points(cplx, kappa):
    """A source whose position is no number has no distance to the target and adds nothing:
    the sums are those without it, to the rounding of another summation order (2 eps a source)."""
    import torch
    import hfmm_b200
    from hfmm_b200.kernels import yukawa
    rng = np.random.default_rng(9)
    n = 700
    pos, q = rng.uniform(size=(n, 3)), rng.normal(size=n) + (1j * rng.normal(size=n) if cplx else 0.0)
    st = hfmm_b200.setup(pos, 2.0, p=3, N_max=64) if kappa is None else hfmm_b200.kernel_setup(pos, yukawa(kappa), p=3)
    out = []
    for bad in (0.0, np.nan):
        x, c = pos.copy(), q.copy()
        x[[100, 650], 1] += bad
        c[[100, 650]] = 0.0
        st.positions = torch.as_tensor(x).cuda()   # the referee reads them from the state
        out.append(hfmm_b200.direct(st, c, np.arange(20), field=True))
    for a, b in zip(*out):
        assert np.isfinite(b).all() and np.abs(a - b).max() <= 2 * n * EPS * np.abs(a).max()
    st.close()


@pytest.mark.parametrize("k", [0.5, 24.0, 26.0, 400.0, 6000.0])
def test_near_field_accuracy(k):
    """The FP64 near field of one box against extended precision, on points of a lattice of
    spacing 2^-10, whose squared distances are exact. The phase then carries one rounding of r
    and one of k r: the bar is the error that these two alone make (10 % for the spread of four
    clouds' mean) and four eps for the weights and sums. A third rounding in r is over it where
    k is large."""
    import hfmm_b200
    errs, bars = [], []
    for seed in range(4):
        rng = np.random.default_rng([seed, 3])
        n = 1000
        pos, q = rng.integers(0, 1024, (n, 3)) / 1024.0, rng.normal(size=n) + 1j * rng.normal(size=n)
        pos[0], pos[-1] = 0.0, 1.0   # extent 1: the kernel's form changes at k = 25
        st = hfmm_b200.setup(pos, k, p=3, N_max=n, max_depth=1)
        phi = hfmm_b200.evaluate_field(st, q)[0]
        st.close()

        def total(r, kr):
            w = np.exp(1j * kr.astype(np.longdouble)) / r.astype(np.longdouble)
            np.fill_diagonal(w, 0)
            return w @ q.astype(np.clongdouble)
        d = pos[:, None] - pos[None]
        d2 = (d.astype(np.longdouble) ** 2).sum(-1)
        np.fill_diagonal(d2, 1)
        exact = total(np.sqrt(d2), np.longdouble(k) * np.sqrt(d2))
        r = np.sqrt(d2).astype(np.float64)
        rounded = total(np.sqrt(d2), k * r)
        errs.append(float(np.linalg.norm(phi - exact) / np.linalg.norm(exact)))
        bars.append(float(np.linalg.norm(rounded - exact) / np.linalg.norm(exact)))
    assert np.mean(errs) < 1.1 * np.mean(bars) + 4 * EPS


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("scale", [1e-90, 1e-60, 1e-12, 1.0, 1e12, 1e90])
def test_any_unit_of_length(scale, cplx):
    """The same problem in another unit of length, k times extent unchanged: phi and E scale by
    1 / scale and 1 / scale^2. To 1e-9: the damped decodes' rounding, which the scaled tables
    draw anew, amplified as in the parity tests at their loosest."""
    import hfmm_b200
    rng = np.random.default_rng(21)
    n = 2000
    pos, q = rng.uniform(size=(n, 3)), rng.normal(size=n) + (1j * rng.normal(size=n) if cplx else 0.0)
    out = []
    for s in (1.0, scale):
        st = hfmm_b200.setup(pos * s, 3.0 / s, p=5, N_max=32)
        phi, E = hfmm_b200.evaluate_field(st, q)
        st.close()
        out.append((phi * s, (E * s) * s))
    for a, b in zip(*out):
        assert np.isfinite(b).all() and np.linalg.norm(a - b) <= 1e-9 * np.linalg.norm(a)
