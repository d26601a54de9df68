"""Neighbour searches that share a warp two by two: odd numbers of queries, neighbours in
the list of very different size (none, a few, more than a list holds, more than a row
holds), ids with no vertex, both layouts, against brute force in the same floats."""
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


@pytest.mark.parametrize("layout", ["column", "row"])
@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 63, 129])
def test_pairs(M, n, layout):
    import torch

    from mcleap_gb300 import _lib as L

    rng = np.random.default_rng(n)
    sparse = rng.random((2000, 2)) * 8000
    dense = 4000 + rng.standard_normal((400, 2)) * 30
    p = np.concatenate([sparse, dense]).astype(np.float32)
    b = M.MeshBatch.from_points([p])
    pos = b.download(0)[0]
    F = 48
    r = np.array([25.0], np.float32)
    verts = rng.integers(4, b.V, n).astype(np.int32)
    crowd = np.nonzero(np.abs(pos - 4000).max(1) < 20)[0]
    verts[::3] = rng.choice(crowd, len(verts[::3]))
    verts[5::7] = -1
    if n > 2:
        verts[1] = 0  # a corner
    lay = L.LAYOUT_COLUMN if layout == "column" else L.LAYOUT_ROW
    out = torch.full((n * F,), -9, dtype=torch.int32, device="cuda")
    over = b.frnn_list(torch.from_numpy(r).cuda(), torch.from_numpy(verts).cuda(), F, out, layout=lay)
    got = out.view(F, n).cpu().numpy().T if layout == "column" else out.view(n, F).cpu().numpy()
    cut = 0
    r2 = r[0] * r[0]
    for k, v in enumerate(verts):
        want = np.zeros(0, np.int64)
        if v >= 0:
            d = pos - pos[v]
            near = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).astype(np.float32) <= r2
            near[v] = False
            want = np.nonzero(near)[0]
        cut += len(want) > F - 1
        assert got[k, 0] == min(len(want), F - 1)
        assert np.array_equal(got[k, 1:1 + got[k, 0]], want[:F - 1]), (k, v)
        assert (got[k, 1 + got[k, 0]:] == -9).all()
    assert over == cut
    b.close()
