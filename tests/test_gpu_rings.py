"""Ring and neighbour queries at the sizes where their forms meet, against the
mesh's edges and brute force: rings of more spokes than the registers' share, rows
cut off, row strides that are no multiple of four words, lists with vertices that
do not exist, and neighbour sets larger than a warp's list."""
import numpy as np
import pytest

from helpers import csr_from_table, uniform_points
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


def fan(n):
    """A hub with n points around it and a cluster that gives long corner rings."""
    a = np.linspace(0, 2 * np.pi, n, endpoint=False)
    rim = 4096 + 1500 * np.stack([np.cos(a), np.sin(a)], 1)
    side = np.stack([np.zeros(80), np.linspace(100, 8000, 80)], 1)
    return np.concatenate([[[4096, 4096]], rim, side]).astype(np.float32)


@pytest.mark.parametrize("max_ring", [4, 15, 16, 17, 32, 63])
@pytest.mark.parametrize("points", ["fan", "uniform", "one"])
def test_rings_rows_and_lists(M, points, max_ring):
    import torch

    pts = {"fan": fan(40), "uniform": uniform_points(777, 4), "one": np.float32([[4000, 5000]])}[points]
    host = M.HostTriangulation()
    host.addDelaunayPoints(pts.copy())
    dt = M.DeviceTriangulation(host)
    V = dt.m_pos_size
    dt.step(torch.zeros((V, 2), device="cuda"))  # Delaunay: the corners' short cut is open
    dt.transferToHost()
    counts, ids = O.ring_sets_from_edges(host.edges(), V)
    offs = np.concatenate([[0], np.cumsum(counts)])
    table = {}
    for layout in (0, 1):
        ring = torch.full((V * max_ring,), -7, dtype=torch.int32, device="cuda")
        cut = dt.oneRing(max_ring, ring, layout=layout)
        assert cut == int((counts > max_ring - 1).sum())
        assert dt.oneRing(max_ring, ring, layout=layout) == cut  # the count starts again
        c, rows = csr_from_table(ring.cpu().numpy(), layout, V, max_ring)
        assert np.array_equal(c, np.minimum(counts, max_ring - 1))
        for i in range(V):
            want = set(ids[offs[i]:offs[i + 1]].tolist())
            assert rows[i][0] == min(want) and set(rows[i].tolist()) <= want and len(set(rows[i].tolist())) == c[i]
        # slots past a ring stay as they were
        t = ring.cpu().numpy().reshape((max_ring, V) if layout == 0 else (V, max_ring))
        t = t if layout else t.T
        assert all((t[i, 1 + c[i]:] == -7).all() for i in range(V))
        table[layout] = t
    assert np.array_equal(table[0], table[1])
    b = M.MeshBatch(dt.handle)
    verts = np.concatenate([np.arange(V)[::-1], [V, -1, 3]]).astype(np.int32)
    out = torch.full((len(verts) * max_ring,), -7, dtype=torch.int32, device="cuda")
    b.one_ring_list(torch.from_numpy(verts).cuda(), max_ring, out)
    got = out.cpu().numpy().reshape(len(verts), max_ring)
    b.handle = type(b.handle)()  # the mesh is dt's
    for q, v in enumerate(verts):
        if 0 <= v < V:
            assert np.array_equal(got[q], table[1][v])
        else:
            assert got[q, 0] == 0 and (got[q, 1:] == -7).all()


@pytest.mark.parametrize("r", [0.0, 1.0, 2.0, 3.7, 6.0])
def test_mesh_neighbours_of_every_size(M, r):
    """r = 3.7 gives sets on either side of 64, r = 6 sets on either side of 113."""
    import torch

    n = 1200
    pts = uniform_points(n, 12)
    host = M.HostTriangulation()
    host.addDelaunayPoints(pts.copy())
    dt = M.DeviceTriangulation(host)
    V, F = dt.m_pos_size, 256
    rad = r * 8192.0 / np.sqrt(n)
    bc, bids = O.frnn_brute(host.m_pos, rad)
    offs = np.concatenate([[0], np.cumsum(bc)])
    for layout in (0, 1):
        out = torch.zeros(V * F, dtype=torch.int32, device="cuda")
        assert dt.getFRNN(F, rad, out, layout=layout) == 0
        c, rows = csr_from_table(out.cpu().numpy(), layout, V, F)
        assert np.array_equal(c, bc) and np.array_equal(np.concatenate(rows), bids)
    out = torch.zeros(V * 20, dtype=torch.int32, device="cuda")
    assert dt.getFRNN(20, rad, out, layout=1) == int((bc > 19).sum())
    t = out.cpu().numpy().reshape(V, 20)
    for i in range(V):
        assert t[i, 0] == min(bc[i], 19) and np.array_equal(t[i, 1:1 + t[i, 0]], bids[offs[i]:offs[i] + t[i, 0]])
