"""Imported meshes whose first four vertices are not the corners of a square around the
rest: their rings start at the smallest neighbour all the same."""
import numpy as np
import pytest

from helpers import csr_from_table
from oracle import oracle as O

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


def mesh_of(M, pos, tri, first):
    """HostTriangulation of counter-clockwise triangles; first[v] (optional): the end of
    the half-edge that vertex v names."""
    inner = {}
    for t, (a, b, c) in enumerate(tri):
        for k, (u, v) in enumerate([(a, b), (b, c), (c, a)]):
            inner[(u, v)] = (t, (a, b, c)[(k + 2) % 3])
    pairs = sorted({(min(e), max(e)) for e in inner})
    num = {}
    for e, (u, v) in enumerate(pairs):
        num[(u, v)], num[(v, u)] = 2 * e, 2 * e + 1
    out = {u: v for u, v in num if (u, v) not in inner}  # the border, one half-edge from each vertex
    he = np.zeros((len(num), 4), np.int32)
    for (u, v), h in num.items():
        if (u, v) in inner:
            t, apex = inner[(u, v)]
            he[h] = (num[(v, apex)], u, t, apex)
        else:
            he[h] = (num[(v, out[v])], u, -1, -1)
    host = M.HostTriangulation()
    host.m_pos = np.ascontiguousarray(pos, np.float32)
    host.m_he = he
    v = [[i, next(num[(i, j)] for j in ([first[i]] if i in first else range(len(pos))) if (i, j) in num)]
         for i in range(len(pos))]
    host.m_v = np.array(v, np.int32)
    host.m_t = np.array([[num[(a, b)]] for a, b, c in tri], np.int32)
    return host


def points():
    """Vertex 0 with vertices 1, 2 and 3 beside it, one after the other, all four in the
    middle of a disk of points."""
    rng = np.random.default_rng(4)
    mid = np.array([[0, 0], [9, 5], [0, 10], [-9, 5]], np.float64)
    a = rng.random(60) * 2 * np.pi
    far = 30 + 100 * np.sqrt(rng.random(60))
    return np.concatenate([mid, np.stack([far * np.cos(a), far * np.sin(a)], 1)]).astype(np.float32)


def delaunay(pos):
    from scipy.spatial import Delaunay

    tri = Delaunay(pos.astype(np.float64)).simplices
    p = pos.astype(np.float64)
    u, w = p[tri[:, 1]] - p[tri[:, 0]], p[tri[:, 2]] - p[tri[:, 0]]
    turned = u[:, 0] * w[:, 1] - u[:, 1] * w[:, 0] < 0
    tri[turned] = tri[turned][:, [0, 2, 1]]
    return [tuple(int(x) for x in t) for t in tri]


@pytest.mark.parametrize("start", [1, 2, 3])
def test_rings_of_an_inner_fixed_vertex(M, start):
    import torch

    pos = points()
    host = mesh_of(M, pos, delaunay(pos), {0: start})
    dt = M.DeviceTriangulation(host)
    V = len(pos)
    assert dt.step(torch.zeros((V, 2), device="cuda"))["status"] == 0  # Delaunay now
    assert not any(dt.validate().values())
    counts, ids = O.ring_sets_from_edges(host.edges(), V)
    offs = np.concatenate([[0], np.cumsum(counts)])
    assert {1, 2, 3} < set(ids[:counts[0]].tolist())
    for layout, size in [(0, 64), (1, 64), (0, 4), (1, 4)]:  # 4: rows cut off
        ring = torch.full((V * size,), -7, dtype=torch.int32, device="cuda")
        assert dt.oneRing(size, ring, layout=layout) == int((counts > size - 1).sum())
        c, rows = csr_from_table(ring.cpu().numpy(), layout, V, size)
        assert np.array_equal(c, np.minimum(counts, size - 1))
        for i in range(V):
            want = ids[offs[i]:offs[i + 1]].tolist()
            assert set(rows[i].tolist()) <= set(want) and rows[i][0] == min(want), (i, size)
    dt.close()
