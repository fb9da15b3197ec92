"""Plans built, rebuilt, used and dropped on several threads at once share the library's kept
memory blocks (csrc/devmem.cu): each result equals the one of the same plan alone, bit for
bit, and once no plan is left the memory is free again."""
import threading

import numpy as np
import pytest

from cases import complex_uniform

pytestmark = pytest.mark.gpu


def _work(seed, out):
    import torch
    import hfmm_b200
    got = []
    with torch.cuda.stream(torch.cuda.Stream()):
        for i in range(3):
            pos, q = complex_uniform(1500 + 700 * i, seed=seed)
            st = hfmm_b200.setup(pos, 2.0, p=4, N_max=24, max_depth=3, domain=((0.0, 0.0, 0.0), 1.0))
            got.append(hfmm_b200.evaluate_field(st, q))
            hfmm_b200.rebuild(st, pos[::-1].copy())
            got.append(hfmm_b200.evaluate_field(st, q))
            st.close()
    out[seed] = got


def test_threads_share_blocks():
    import torch
    alone, together = {}, {}
    for s in range(4):
        _work(s, alone)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    threads = [threading.Thread(target=_work, args=(s, together)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for s in range(4):
        for a, b in zip(alone[s], together[s]):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > before - (64 << 20)
