"""Which meshes have a mover, found by blocks that hold many small meshes, parts of
several, or a share of one: coincident moves of batches against the same rule in numpy."""
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


def settled(pos, d, mesh):
    """Moved vertices of one mesh that would share a place go back, until none do."""
    d = d.copy()
    while True:
        key = np.concatenate([mesh[:, None].astype(np.float32), (pos + d).astype(np.float32)], 1)
        _, inv, counts = np.unique(key, axis=0, return_inverse=True, return_counts=True)
        back = (counts[inv.ravel()] > 1) & d.any(1)
        if not back.any():
            return d
        d[back] = 0


@pytest.mark.parametrize("sizes", [[9] * 300, [1, 2, 255, 256, 257, 1000, 5000], [60000], [40000, 3, 20000]])
@pytest.mark.parametrize("share", [0.02, 0.6, 1.0])
def test_batches(M, sizes, share):
    import torch

    rng = np.random.default_rng(len(sizes))
    sets = []
    for n in sizes:  # points of a lattice, so that moves by whole cells meet
        side = int(np.ceil(np.sqrt(2 * n)))
        at = rng.permutation(side * side)[:n]
        sets.append(np.stack([at % side, at // side], 1).astype(np.float32) + 100)
    b = M.MeshBatch.from_points([p.copy() for p in sets])
    pos = np.concatenate([b.download(i)[0] for i in range(b.count)])
    mesh = np.repeat(np.arange(b.count), b.nv)
    d = rng.integers(-1, 2, (b.V, 2)).astype(np.float32)
    d[rng.random(b.V) >= share] = 0
    d[mesh % 7 == 3] = 0  # whole meshes at rest
    free = np.ones(b.V, bool)
    for v0 in b.v0:
        free[v0:v0 + 4] = False
    d[~free] = 0
    want = settled(pos, d, mesh)
    got = torch.from_numpy(d).cuda()
    assert b.settle(got) == (d.any(1) & ~want.any(1)).sum()
    assert np.array_equal(got.cpu().numpy(), want)
    assert (d.any(1) & ~want.any(1)).any()
    b.close()
