"""Mesh neighbour searches where their forms meet: a thread's list, a part's list, a
thread alone, and the numbers of queries at which they change; whole meshes, lists with
vertices that do not exist, both layouts, and rows too short.  Against brute force."""
import numpy as np
import pytest

from helpers import uniform_points

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


def neighbours(pos, r):
    """Per vertex the sorted ids within r by the float formula (a tree finds a few more)."""
    from scipy.spatial import cKDTree

    t = cKDTree(pos.astype(np.float64))
    pairs = t.query_pairs(float(r) * 1.001, output_type="ndarray")
    d = pos[pairs[:, 0]] - pos[pairs[:, 1]]
    r2 = np.float32(r) * np.float32(r)
    pairs = pairs[(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).astype(np.float32) <= r2]
    both = np.concatenate([pairs, pairs[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    offs = np.searchsorted(both[:, 0], np.arange(len(pos) + 1))
    return offs, both[:, 1].astype(np.int32)


@pytest.mark.parametrize("n", [2040, 2045, 65530, 65540, 99994, 99998, 140003])
@pytest.mark.parametrize("far", [0.2, 0.8, 1.2, 1.6, 2.5, 3.9, 4.6])
def test_uniform(M, n, far):
    import torch

    b = M.MeshBatch.from_points([uniform_points(n, n)])
    pos = b.download(0)[0]
    r = np.float32(far * 8192 / np.sqrt(n))
    offs, ids = neighbours(pos, r)
    counts = np.diff(offs)
    rd = torch.full((1,), float(r), device="cuda")
    rng = np.random.default_rng(n)
    verts = rng.permutation(np.concatenate([np.arange(b.V), [-1, b.V, b.V + 7, 3]])).astype(np.int32)
    for layout, F in ((0, 160), (1, 160), (1, 6), (0, 2)):
        want = np.minimum(counts, F - 1)
        out = torch.full((b.V * F,), -7, dtype=torch.int32, device="cuda")
        assert b.frnn(rd, F, out, layout=layout) == (counts > F - 1).sum()
        t = out.view((F, b.V) if layout == 0 else (b.V, F)).cpu().numpy()
        t = t.T if layout == 0 else t
        assert np.array_equal(t[:, 0], want)
        k = np.arange(F - 1)[None] < want[:, None]
        rank = np.arange(len(ids)) - np.repeat(offs[:-1], counts)
        assert np.array_equal(t[:, 1:][k], ids[rank < F - 1])
        assert (t[:, 1:][~k] == -7).all()
        q = torch.full((len(verts) * F,), -7, dtype=torch.int32, device="cuda")
        real = (verts >= 0) & (verts < b.V)
        assert b.frnn_list(rd, torch.from_numpy(verts).cuda(), F, q, layout=layout) == (counts[verts[real]] > F - 1).sum()
        u = q.view((F, len(verts)) if layout == 0 else (len(verts), F)).cpu().numpy()
        u = u.T if layout == 0 else u
        assert np.array_equal(u[real], t[verts[real]])
        assert (u[~real, 0] == 0).all() and (u[~real, 1:] == -7).all()
    b.close()
