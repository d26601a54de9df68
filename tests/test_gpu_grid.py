"""The grid build's tables against numpy's stable sort by cell: cell counts on both
sides of the scan's block of 4096 cells and of its quadruples, single cells, crowded
cells, points outside the domain, one point, and the velocities that go along."""
import numpy as np
import pytest

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


def ints(ptr, n):
    import torch

    class A:
        __cuda_array_interface__ = dict(shape=(n,), typestr="<i4", data=(ptr, False), version=3)

    return torch.as_tensor(A(), device="cuda").cpu().numpy()


@pytest.mark.parametrize("n,nx,ny,crowd", [(1, 1, 1, 0), (255, 1, 1, 0), (257, 3, 1, 0), (1000, 4095, 1, 0),
                                           (1000, 1024, 4, 0), (1025, 4097, 1, 0), (5000, 64, 65, 2000),
                                           (200000, 311, 313, 700), (30000, 2049, 2050, 0)])
@pytest.mark.parametrize("periodic", [False, True])
def test_tables(M, n, nx, ny, crowd, periodic):
    import torch

    rng = np.random.default_rng(n + nx)
    p = (rng.random((n, 2)) * (nx, ny)).astype(np.float32)
    p[: n // 50] += np.float32(3 * nx)  # outside the domain
    p[n - crowd:] = (0.5 * nx, 0.5 * ny)
    v = rng.standard_normal((n, 2)).astype(np.float32)
    k = np.floor(p).astype(np.int64)
    k = k % (nx, ny) if periodic else np.clip(k, 0, (nx - 1, ny - 1))
    cell = k[:, 1] * nx + k[:, 0]
    order = np.argsort(cell, kind="stable")
    count = np.bincount(cell, minlength=nx * ny)
    g = M.GridCount2d(n, (0.0, 0.0), (1.0, 1.0), (nx, ny), periodic=periodic)
    pos, vel = torch.from_numpy(p).cuda(), torch.from_numpy(v).cuda()
    for again in range(2):
        g.build(pos)
        t = g.tables()
        assert np.array_equal(ints(t["count"], nx * ny), count)
        assert np.array_equal(ints(t["start"], nx * ny), np.cumsum(count) - count)
        perm = ints(t["perm"], n)
        assert np.array_equal(perm[order], np.arange(n))
    g.update(pos, vel)
    assert np.array_equal(pos.cpu().numpy(), p[order])
    assert np.array_equal(vel.cpu().numpy(), v[order])
    g.close()


@pytest.mark.parametrize("periodic", [False, True])
def test_neighbours_far_apart_in_the_order(M, periodic):
    """More points than 16 bits count: rows met across the wrap, and one cell so
    crowded that its own points are that far apart."""
    import torch
    from scipy.spatial import cKDTree

    n, L, r, F = 90000, 300.0, np.float32(2.25), 32
    rng = np.random.default_rng(7)
    p = (rng.random((n, 2)) * L).astype(np.float32)
    g = M.GridCount2d(n, (0.0, 0.0), (1.5, 1.5), (200, 200), periodic=periodic)
    counts = torch.zeros(n, dtype=torch.int32, device="cuda")
    ids = torch.full((n, F), -1, dtype=torch.int32, device="cuda")
    g.build(torch.from_numpy(p).cuda())
    g.frnn_ids(float(r), F, counts, ids)
    got_c, got = counts.cpu().numpy(), ids.cpu().numpy()
    tree = cKDTree(p.astype(np.float64), boxsize=L if periodic else None)
    for i in np.concatenate([np.arange(40), rng.integers(0, n, 400), np.argsort(p[:, 1])[:200]]):
        near = np.array(sorted(set(tree.query_ball_point(p[i].astype(np.float64), float(r) + 0.01)) - {i}))
        d = (p[i] - p[near]).astype(np.float32)
        if periodic:
            d = np.where(np.abs(d) > np.float32(L / 2), (d - np.copysign(np.float32(L), d)).astype(np.float32), d)
        want = near[(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).astype(np.float32) <= r * r]
        assert got_c[i] == len(want)
        assert np.array_equal(np.sort(got[i, :got_c[i]]), want)
        assert (got[i, got_c[i]:] == -1).all()
    g.close()

    k = 40000
    p = np.full((k, 2), 10.0, np.float32)
    g = M.GridCount2d(k, (0.0, 0.0), (1.5, 1.5), (200, 200), periodic=periodic)
    counts = torch.zeros(k, dtype=torch.int32, device="cuda")
    ids = torch.full((k, 60), -1, dtype=torch.int32, device="cuda")
    g.build(torch.from_numpy(p).cuda())
    assert g.frnn_ids(1.0, 60, counts, ids) == k
    got = ids.cpu().numpy()
    assert (counts.cpu().numpy() == 60).all()
    for i in (0, 1, 47, 59, 60, 61, 32767, 32768, 32830, k - 1):
        want = np.arange(61)
        assert np.array_equal(got[i], want[want != i][:60])
    g.close()
