"""Rings longer than their rows and hubs of odd and even numbers of spokes: the first
neighbours, clockwise from the smallest, and how many rows were cut off."""
import numpy as np
import pytest

from helpers import uniform_points
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


def clockwise(pos, i, nb):
    d = pos[nb].astype(np.float64) - pos[i].astype(np.float64)
    r = nb[np.argsort(-np.arctan2(d[:, 1], d[:, 0]))]
    return np.roll(r, -int(np.argmin(r)))


@pytest.mark.parametrize("spokes", [14, 15, 16, 17, 30, 31, 100, 701])
@pytest.mark.parametrize("max_ring", [2, 3, 4, 6, 7, 8, 20, 702])
def test_hub(M, spokes, max_ring):
    import torch

    c = np.array([4096.0, 4096.0])
    p = uniform_points(600, spokes)
    p = p[np.hypot(*(p - c).T) > 1200]
    a = np.linspace(0, 2 * np.pi, spokes, endpoint=False) + 0.01
    p = np.concatenate([p, c[None], c + 1000 * np.stack([np.cos(a), np.sin(a)], 1)]).astype(np.float32)
    b = M.MeshBatch.from_points([p])
    pos = b.download(0)[0]
    counts, ids = O.ring_sets_from_edges(b.edges(0), b.V)
    offs = np.concatenate([[0], np.cumsum(counts)])
    assert counts.max() >= spokes
    rows = [clockwise(pos, i, ids[offs[i]:offs[i + 1]])[:max_ring - 1] for i in range(4, b.V)]
    verts = torch.arange(4, b.V, dtype=torch.int32, device="cuda")
    for layout in (0, 1):
        out = torch.full((b.V * max_ring,), -7, dtype=torch.int32, device="cuda")
        assert b.one_ring(max_ring, out, layout=layout) == (counts > max_ring - 1).sum()
        t = out.cpu().numpy().reshape((max_ring, b.V) if layout == 0 else (b.V, max_ring))
        t = (t.T if layout == 0 else t)[4:]
        part = torch.full((len(rows) * max_ring,), -7, dtype=torch.int32, device="cuda")
        assert b.one_ring_list(verts, max_ring, part, layout=layout) == (counts[4:] > max_ring - 1).sum()
        u = part.cpu().numpy().reshape((max_ring, len(rows)) if layout == 0 else (len(rows), max_ring))
        assert np.array_equal(t, u.T if layout == 0 else u)
        for r, want in zip(t, rows):
            assert r[0] == len(want) and np.array_equal(r[1:1 + r[0]], want) and (r[1 + r[0]:] == -7).all()
    b.close()
