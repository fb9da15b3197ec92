"""The mixed M2L's FP16 operand planes at the ends of their range. Every plane is scaled by
a power of two from the largest magnitude of its operand, so charges multiplied by a power of
two give the same bits multiplied by it (no overflow, nothing flushed; the FP32 near field
stays inside its range at 2^+-60), and zero charges give zeros. Ranks from the loosest
compression to none (k-chunks of one to four steps, row blocks of 64 and 128), real and
complex charges, sources gathered (clusters) and from the grid (uniform).
One charge 2^30 times the others sets every plane's scale: the error against FP64 on the same
plan stays at the mixed path's bar, 2e-6 in the norm, which that charge carries (what is left
of the weaker charges' own results: test_gpu_mixed_range.py)."""
import numpy as np
import pytest

import oracle as O
from cases import complex_uniform, sphere_clusters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,eps,cloud,n,leaf", [
    (5, None, complex_uniform, 9000, 24), (6, 1e-3, complex_uniform, 9000, 24),
    (7, 1e-5, sphere_clusters, 6000, 16), (8, 1e-7, complex_uniform, 9000, 24),
    (9, None, sphere_clusters, 6000, 32)])
def test_power_of_two_charges(p, eps, cloud, n, leaf):
    import hfmm_b200
    pos, q = cloud(n)
    q = q + 1j * np.roll(q.real, 7)
    st = hfmm_b200.setup(pos, 5.0, p=p, N_max=leaf, m2l_compress=eps)
    run = lambda v, prec=hfmm_b200.PREC_MIXED: hfmm_b200.evaluate_field(st, v, precision=prec)  # noqa: E731
    for v in (q, q.real.copy()):
        base = run(v)
        for e in (-60, 60):
            for x, y in zip(run(v * 2.0 ** e), base):
                assert np.isfinite(x).all() and np.array_equal(x, y * 2.0 ** e)
        assert all((x == 0).all() for x in run(v * 0.0))
        one = v.copy()
        one[n // 2] *= 2.0 ** 30
        for x, y in zip(run(one), run(one, hfmm_b200.PREC_FP64)):
            assert O.relative_error(x, y) < (2e-6 if eps in (None, 1e-7) else 2e-6 + eps)
    st.close()
