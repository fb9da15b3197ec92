"""The FP64 GEMM's two tile sizes on the same boxes: one charge column of the finest level
is under the line of the small tiles, two columns are over it. Evaluation is linear, so a
complex charge vector has to give what its real and imaginary parts give one by one, to
3e-12, the bar of the order-12 parity tests. Orders whose surface points leave part of a
tile's rows empty (8, 56 and 218 points)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
TOL = 3e-12


@pytest.mark.parametrize("p,depth,height", [(2, 5, 0.5), (4, 5, 0.5), (7, 4, 1.0)])
def test_two_tile_sizes(p, depth, height):
    import hfmm_b200
    rng = np.random.default_rng(p)
    n = 8 ** depth * 6
    pos = rng.uniform(size=(n, 3)) * [1.0, 1.0, height]
    pos[:2] = [[0, 0, 0], [1, 1, height]]
    q = rng.normal(size=n) + 1j * rng.normal(size=n)
    st = hfmm_b200.setup(pos, 4.0, p=p, N_max=1, max_depth=depth)
    both = hfmm_b200.evaluate_field(st, q)
    re = hfmm_b200.evaluate_field(st, q.real.copy())
    im = hfmm_b200.evaluate_field(st, q.imag.copy())
    for x, a, b in zip(both, re, im):
        assert np.isfinite(x).all() and O.relative_error(x, a + 1j * b) < TOL
    st.close()
