"""The charge columns of one evaluate do not disturb each other: an imaginary column far smaller
than the real one keeps its own accuracy, and a column of zeros adds nothing. The expected
result is that of the columns evaluated one by one as real charges, by linearity. With one
family (Laplace, screened Coulomb) the imaginary part is the imaginary column's alone; with
two and a small wavenumber it is the sum of the small sin family and the small column.
Bars: the 3e-12 of the convolution's tests in FP64, the mixed path's 2e-6, on the imaginary
parts by themselves."""
import numpy as np
import pytest

import oracle as O
from cases import complex_uniform

pytestmark = pytest.mark.gpu
SCALES = [1.0, 1e-4, 1e-8, 0.0]


def _columns(n):
    pos, q = complex_uniform(n)
    return pos, q.real.copy(), q.imag.copy()


@pytest.mark.parametrize("kappa", [0.0, 5.0])
@pytest.mark.parametrize("precision,tol", [(0, 3e-12), (1, 2e-6)])
def test_one_family(kappa, precision, tol):
    import hfmm_b200
    from hfmm_b200.kernels import LAPLACE, yukawa
    pos, a, b = _columns(9000)
    st = hfmm_b200.kernel_setup(pos, yukawa(kappa) if kappa else LAPLACE, p=6, N_max=32)
    alone = hfmm_b200.evaluate_field(st, b, precision=precision)
    for s in SCALES:
        for x, y in zip(hfmm_b200.evaluate_field(st, a + 1j * s * b, precision=precision), alone):
            assert O.relative_error(x.imag, s * y.real) < tol if s else (x.imag == 0).all()
        for x, y in zip(hfmm_b200.evaluate_field(st, s * b + 1j * a, precision=precision), alone):
            assert O.relative_error(x.real, s * y.real) < tol if s else (x.real == 0).all()
    st.close()


@pytest.mark.parametrize("precision,tol", [(0, 3e-12), (1, 2e-6)])
def test_two_families_small_wavenumber(precision, tol):
    import hfmm_b200
    pos, a, b = _columns(9000)
    st = hfmm_b200.setup(pos, 1e-6, p=6, N_max=32)
    one, two = (hfmm_b200.evaluate(st, v) for v in (a, b))
    for s in SCALES:
        x = hfmm_b200.evaluate_field(st, a + 1j * s * b, precision=precision)[0]
        y = one + 1j * s * two
        assert O.relative_error(x.imag, y.imag) < tol and O.relative_error(x.real, y.real) < tol
    st.close()


@pytest.mark.parametrize("small,large", [(1e-290, 1.0), (1.0, 1e280), (1e-290, 1e-5)])
def test_columns_far_apart(small, large):
    """Columns hundreds of orders of magnitude apart, at a wavenumber that keeps the results
    apart: each by itself as accurate as alone, whichever is the larger."""
    import hfmm_b200
    pos, a, b = _columns(6000)
    st = hfmm_b200.setup(pos, 0.0, p=5, N_max=32)   # two families, the sin family's sums all zero
    one, two = (hfmm_b200.evaluate_field(st, v) for v in (a, b))
    for x, u, v in zip(hfmm_b200.evaluate_field(st, a * large + 1j * b * small), one, two):
        assert O.relative_error(x.real / large, u.real) < 3e-12 and O.relative_error(x.imag / small, v.real) < 3e-12
    for x, u, v in zip(hfmm_b200.evaluate_field(st, a * small + 1j * b * large), one, two):
        assert O.relative_error(x.real / small, u.real) < 3e-12 and O.relative_error(x.imag / large, v.real) < 3e-12
    st.close()


@pytest.mark.parametrize("s", [1.0, 1e-8])
def test_streamed_rows_of_a_plane(s):
    """A streamed plan whose workspace holds no plane of complex frequencies (p = 2, five levels)
    transforms the columns apart."""
    import hfmm_b200
    pos, a, b = _columns(20000)
    st = hfmm_b200.setup(pos, 1e-6, p=2, N_max=32, max_depth=5, stream_tables=True)
    one, two = (hfmm_b200.evaluate(st, v) for v in (a, b))
    x, y = hfmm_b200.evaluate_field(st, a + 1j * s * b)[0], one + 1j * s * two
    assert O.relative_error(x.imag, y.imag) < 3e-12 and O.relative_error(x.real, y.real) < 3e-12
    st.close()
