"""The mixed path where the charges span many orders of magnitude: two clusters in opposite
corners, one with charges 2^e of the other's. With a screened kernel the weak cluster's
results are its own, so its error against FP64 is measured by itself, at the mixed path's 2e-6;
kappa on both sides of the line (kappa x extent = 2) where the M2L's operand planes hold.
With Helmholtz the strong cluster's field reaches everywhere and sets the scale."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [None, 1e-7])
@pytest.mark.parametrize("kappa", [0.0, 1.9, 2.2, 8.0, 40.0, "helmholtz"])
def test_weak_cluster(kappa, eps):
    import hfmm_b200
    from hfmm_b200.kernels import LAPLACE, helmholtz, yukawa
    rng = np.random.default_rng(11)
    n = 8000
    pos = np.concatenate([np.clip(c + 0.04 * rng.normal(size=(n // 2, 3)), 0, 1) for c in (0.1, 0.9)])
    pos[0], pos[-1] = 0.0, 1.0   # the domain is the unit cube
    q = rng.normal(size=n)
    spec = helmholtz(9.0) if kappa == "helmholtz" else yukawa(kappa) if kappa else LAPLACE
    st = hfmm_b200.kernel_setup(pos, spec, p=8, N_max=48, m2l_compress=eps)
    for e in (0, 18, 26, 40):
        v = q.copy()
        v[: n // 2] *= 2.0 ** e
        for x, y in zip(hfmm_b200.evaluate_field(st, v, hfmm_b200.PREC_MIXED), hfmm_b200.evaluate_field(st, v)):
            assert O.relative_error(x[n // 2:], y[n // 2:]) < 2e-6
    st.close()


@pytest.mark.parametrize("eps", [None, 1e-7])
@pytest.mark.parametrize("kind,k", [("laplace", 0.0), ("yukawa", 1.9), ("helmholtz", 0.01), ("helmholtz", 1.0)])
def test_field_on_a_weak_deep_cluster(kind, k, eps):
    """Two clusters a thousandth of the domain wide (depth 10): the strong one's field at the weak
    one is 1 / r^2 of its charges, what its densities' rounding leaves there 1 / (box side)^2."""
    import hfmm_b200
    from hfmm_b200.kernels import LAPLACE, helmholtz, yukawa
    rng = np.random.default_rng(12)
    n = 20000
    pos = np.concatenate([np.clip(c + 0.0005 * rng.normal(size=(n // 2, 3)), 0, 1) for c in (0.05, 0.95)])
    pos[0], pos[-1] = 0.0, 1.0
    q = rng.normal(size=n)
    spec = LAPLACE if kind == "laplace" else yukawa(k) if kind == "yukawa" else helmholtz(k)
    st = hfmm_b200.kernel_setup(pos, spec, p=8, N_max=24, m2l_compress=eps)
    assert st.max_depth >= 8
    for e in (0, 26, 34):
        v = q.copy()
        v[: n // 2] *= 2.0 ** e
        for x, y in zip(hfmm_b200.evaluate_field(st, v, hfmm_b200.PREC_MIXED), hfmm_b200.evaluate_field(st, v)):
            assert O.relative_error(x[n // 2:], y[n // 2:]) < 2e-6
    st.close()


@pytest.mark.parametrize("p", [5, 6])
@pytest.mark.parametrize("shift", [-40, 0, 3, 20])
def test_scaled_host_tables(monkeypatch, p, shift):
    """M2L tables given by the host are used as given, whatever their size: with every entry
    times 2^shift (and the other tables as they are) mixed still follows FP64 on the same plan."""
    import hfmm_b200
    from cases import complex_uniform
    tables = hfmm_b200.level_tables
    monkeypatch.setattr(hfmm_b200, "level_tables",
                        lambda *a, **k: dict(tables(*a, **k), M2L_K=tables(*a, **k)["M2L_K"] * 2.0 ** shift))
    pos, q = complex_uniform(6000)
    st = hfmm_b200.setup(pos, 5.0, p=p, N_max=24, tables="host")
    for x, y in zip(hfmm_b200.evaluate_field(st, q, hfmm_b200.PREC_MIXED), hfmm_b200.evaluate_field(st, q)):
        assert np.isfinite(x).all() and O.relative_error(x, y) < 2e-6
    st.close()
