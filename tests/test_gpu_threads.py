"""Evaluates of plans of different orders on several threads at once: the kernels that every
order shares (the convolution's transforms, the surface sums) need another amount of shared
memory for each, and every call gets its own. Results as of the same calls one by one, bit for
bit."""
import threading

import numpy as np
import pytest

from cases import complex_uniform

pytestmark = pytest.mark.gpu


def test_orders_side_by_side():
    import torch
    import hfmm_b200
    orders = [5, 6, 7, 8, 5, 6, 7, 8]
    plans, want, got, errors = [], [], [None] * len(orders), []
    for i, p in enumerate(orders):
        pos, q = complex_uniform(2000, seed=i)
        st = hfmm_b200.setup(pos, 3.0, p=p, N_max=48)
        want.append(hfmm_b200.evaluate(st, q.real.copy()))
        plans.append((st, torch.as_tensor(q.real.copy()).cuda(), torch.empty(len(q), dtype=torch.complex128, device="cuda")))
    torch.cuda.synchronize()
    start = threading.Barrier(len(orders))

    def work(i):
        st, q, phi = plans[i]
        try:
            s = torch.cuda.Stream()
            start.wait()
            for _ in range(400):
                hfmm_b200.evaluate_into(st, q, None, phi, stream=s)
            hfmm_b200.check_errors(st, s)
            got[i] = phi.cpu().numpy()
        except Exception as e:   # noqa: BLE001 -- reported by the assert below
            errors.append(f"order {orders[i]}: {e}")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(orders))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    for st, _, _ in plans:
        st.close()
