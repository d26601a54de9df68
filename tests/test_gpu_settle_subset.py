"""Settling one mesh of a batch: the table holds as many slots as the active meshes
need, down to a mesh of a single point, with the same result as every mesh active."""
import numpy as np
import pytest

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


@pytest.mark.parametrize("active", [[0], [1], [2], [3], [0, 3], [1, 2, 3], [0, 1, 2, 3]])
def test_subset(M, active):
    import torch

    rng = np.random.default_rng(4)
    sets = [np.array([[5, 6]], np.float32), np.array([[1, 1], [2, 1], [1, 3]], np.float32)]
    sets += [np.unique(rng.integers(0, 60, (n, 2)), axis=0).astype(np.float32) for n in (300, 900)]
    b = M.MeshBatch.from_points([p.copy() for p in sets])
    pos = np.concatenate([b.download(i)[0] for i in range(b.count)])
    comp = np.repeat(np.arange(b.count), [len(s) + 4 for s in sets])
    fixed = np.concatenate([np.arange(len(s) + 4) < 4 for s in sets])
    d = rng.integers(-2, 3, pos.shape).astype(np.float32)
    d[fixed] = 0
    want = d.copy()
    for c in active:
        at = comp == c
        want[at] = O.settle_moves(pos[at], d[at], comp=None, fixed=fixed[at])
    if len(active) < b.count:
        b.set_active(active)
    t = torch.from_numpy(d.copy()).cuda()
    b.settle(t)
    assert np.array_equal(t.cpu().numpy(), want)
    b.close()
