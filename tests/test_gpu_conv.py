"""The FP64 M2L by convolution (the default with device tables) against the dense M2L tables
(tables="host") on the same points: potentials and fields agree to 3e-12, the bar of the
order-12 parity tests (two summation orders of the oracle differ by up to 4.1e-13 there).
Orders at the lattice's edges (p = 2, 3: lines of two and three points), partial groups of
slots, absent children, one and two families and charge columns. Streamed plans run the same
kernels in a smaller workspace: whole planes of frequencies give the same bits, rows of one
plane the same numbers."""
import numpy as np
import pytest

import oracle as O
from cases import complex_uniform, sphere_clusters, uniform

pytestmark = pytest.mark.gpu
TOL = 3e-12

CASES = [(2, 400, 1.0, 8, complex_uniform), (3, 700, 2.0, 8, uniform), (4, 6000, 3.0, 16, complex_uniform),
         (5, 3000, 6.0, 24, sphere_clusters), (7, 9000, 0.0, 32, complex_uniform), (9, 4000, 8.0, 40, uniform)]


@pytest.mark.parametrize("p,n,k,leaf,cloud", CASES)
def test_matches_dense_tables(p, n, k, leaf, cloud):
    import hfmm_b200
    pos, q = cloud(n)
    a = hfmm_b200.setup(pos, k, p=p, N_max=leaf)
    b = hfmm_b200.setup(pos, k, p=p, N_max=leaf, tables="host")
    for charges in ([q, q.real.copy()] if np.iscomplexobj(q) else [q]):
        for x, y in zip(hfmm_b200.evaluate_field(a, charges), hfmm_b200.evaluate_field(b, charges)):
            assert np.isfinite(x).all() and O.relative_error(x, y) < TOL
    a.close()
    b.close()


@pytest.mark.parametrize("p,depth,same_bits", [(3, 4, True), (2, 5, False)])
def test_chunks_of_frequencies(p, depth, same_bits):
    """A streamed plan's workspace (316 matrices per family) holds one plane of one family
    at (3, 4) and one row of a plane at (2, 5)."""
    import hfmm_b200
    pos, q = complex_uniform(20000)
    a = hfmm_b200.setup(pos, 2.0, p=p, N_max=32, max_depth=depth)
    b = hfmm_b200.setup(pos, 2.0, p=p, N_max=32, max_depth=depth, stream_tables=True)
    for x, y in zip(hfmm_b200.evaluate_field(a, q), hfmm_b200.evaluate_field(b, q)):
        assert np.array_equal(x, y) if same_bits else O.relative_error(x, y) < TOL
    a.close()
    b.close()
