"""Counted queries of one mesh or torus from several threads, each on its own stream: every
call's count is that of the same call alone, during the overlap and after it."""
import threading

import numpy as np
import pytest

from helpers import torus_points, uniform_points

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import torch

    import mcleap_gb300 as M
    from mcleap_gb300 import build as B

    assert torch.cuda.is_available()
    B.build()
    M.lib()
    return M


def together(jobs, rounds):
    """Run the jobs at the same time, `rounds` times each; what they returned."""
    got = [[] for _ in jobs]
    start = threading.Barrier(len(jobs))

    def work(i):
        start.wait()
        for _ in range(rounds):
            got[i].append(jobs[i]())

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return got


@pytest.mark.parametrize("threads", [2, 4, 12])
def test_mesh_queries_overlap(M, threads):
    import torch

    n, ring, near = 60000, 6, 8
    b = M.MeshBatch.from_points([uniform_points(n, 5)])
    V = b.V
    r = torch.full((1,), 8192.0 / np.sqrt(n) * 1.5, dtype=torch.float32, device="cuda")
    lists = [torch.arange(k, V, k + 1, dtype=torch.int32, device="cuda") for k in range(threads)]

    def job(i):
        s = torch.cuda.Stream()
        out = torch.empty(V * near, dtype=torch.int32, device="cuda")
        if i % 4 == 0:
            return lambda: b.one_ring(ring, out, layout=1, stream=s)
        if i % 4 == 1:
            return lambda: b.one_ring_list(lists[i], ring, out, stream=s)
        if i % 4 == 2:
            return lambda: b.frnn(r, near, out, stream=s)
        return lambda: b.frnn_list(r, lists[i], near, out, stream=s)

    jobs = [job(i) for i in range(threads)]
    torch.cuda.synchronize()
    alone = [j() for j in jobs]
    assert all(a > 0 for a in alone)
    for i, got in enumerate(together(jobs, 200)):
        assert got == [alone[i]] * 200, i
    assert [j() for j in jobs] == alone
    b.close()


@pytest.mark.parametrize("threads", [2, 5])
def test_torus_rings_overlap(M, threads):
    import torch

    t = M.PeriodicTriangulation(torus_points(3000, 9))
    first = torch.empty(t.n * 16, dtype=torch.int32, device="cuda")
    t.oneRing(16, first)  # works out the half-edges that later calls start from

    def job(i):
        s = torch.cuda.Stream()
        out = torch.empty(t.n * 16, dtype=torch.int32, device="cuda")
        return lambda: t.oneRing(6 + i, out, stream=s)

    jobs = [job(i) for i in range(threads)]
    torch.cuda.synchronize()
    alone = [j() for j in jobs]
    assert alone[0] > 0
    for i, got in enumerate(together(jobs, 200)):
        assert got == [alone[i]] * 200, i
    assert [j() for j in jobs] == alone
    t.close()
