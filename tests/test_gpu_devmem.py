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


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
@pytest.mark.parametrize("what", ["close", "direct"])
def test_other_threads_capture(mode, what):
    """A plan closed, or a direct sum run, on one thread leaves a stream capture of another
    thread whole (in the modes that let other threads allocate and free): the captured evaluate
    gives the same bits."""
    import torch
    import hfmm_b200
    pos, q = complex_uniform(3000)
    a = hfmm_b200.setup(pos, 3.0, p=4, N_max=48)
    b = hfmm_b200.setup(pos, 2.0, p=4, N_max=48)
    tg = np.arange(50)
    hfmm_b200.direct(b, q, tg)
    qd = torch.as_tensor(q.real.copy()).cuda()
    phi = torch.empty(len(q), dtype=torch.complex128, device="cuda")
    hfmm_b200.evaluate_into(a, qd, None, phi)
    want = phi.cpu().numpy()
    # the direct sum's own stream and inputs, so that torch allocates nothing in the capture
    side = torch.cuda.Stream()
    tgd = torch.as_tensor(tg.astype(np.int32)).cuda()
    with torch.cuda.stream(side):
        hfmm_b200.direct_at(b, qd, None, tgd, stream=side)
    torch.cuda.synchronize()

    def other():
        with torch.cuda.stream(side):
            b.close() if what == "close" else hfmm_b200.direct_at(b, qd, None, tgd, stream=side)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        hfmm_b200.evaluate_into(a, qd, None, phi)
        t = threading.Thread(target=other)
        t.start()
        t.join()
    phi.zero_()
    graph.replay()
    assert np.array_equal(phi.cpu().numpy(), want)
    a.close()
    b.close()


def test_plan_closed_while_it_runs():
    """A plan closed with evaluates still in flight: they finish on its own memory, which only
    then serves the plans built after it."""
    import torch
    import hfmm_b200
    pos, q = complex_uniform(60000)
    small = hfmm_b200.setup(pos[:4000], 2.0, p=4, N_max=24)   # keeps the store of blocks open
    want_small = hfmm_b200.evaluate_field(small, q[:4000])
    qd = torch.as_tensor(q.real.copy()).cuda()
    want = None
    for _ in range(3):
        st = hfmm_b200.setup(pos, 3.0, p=6, N_max=32)
        phi = [torch.zeros(len(q), dtype=torch.complex128, device="cuda") for _ in range(8)]
        side = torch.cuda.Stream()
        torch.cuda.synchronize()
        for x in phi:
            hfmm_b200.evaluate_into(st, qd, None, x, stream=side)
        st.close()
        other = hfmm_b200.setup(pos[:4000], 2.0, p=4, N_max=24)
        got = hfmm_b200.evaluate_field(other, q[:4000])
        other.close()
        assert all(np.array_equal(x, y) for x, y in zip(got, want_small))
        torch.cuda.synchronize()
        want = phi[0].cpu().numpy() if want is None else want
        assert all(np.array_equal(x.cpu().numpy(), want) for x in phi)
    small.close()
