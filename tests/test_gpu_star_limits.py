"""Stars that cannot be made, and what takes over: more wide stars than there are
overflow rows, found when the mesh is built, at once, or in a later round of many
vertices.  The result is the oracle's exact triangulation either way."""
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


def wheels(count, single, spokes, jitter, seed):
    """`count` hubs with their rims and `single` points beside them, on a lattice of
    cells: (the rims scattered by `jitter` cells, the rims round)."""
    rng = np.random.default_rng(seed)
    side = int(np.ceil(np.sqrt(count + single)))
    w = 8192.0 / side
    at = rng.permutation(side * side)[:count + single]
    c = (np.stack([at % side, at // side], 1) + 0.5) * w
    a = np.linspace(0, 2 * np.pi, spokes, endpoint=False)
    far = 0.4 * w * (1 + 0.01 * rng.standard_normal((count, spokes, 1)))
    rim = c[:count, None] + far * np.stack([np.cos(a), np.sin(a)], 1)
    rest = c[count:] + 0.2 * w * np.clip(rng.standard_normal((single, 2)), -1, 1)
    after = np.concatenate([c[:count], rim.reshape(-1, 2), rest]).astype(np.float32)
    before = after.copy()
    k = count * (spokes + 1)
    before[:k] += (jitter * w * rng.standard_normal((k, 2))).astype(np.float32)
    return np.clip(before, 0, 8191).astype(np.float32), after


def moved_to(b, before, after):
    """The displacement, in the batch's order, that takes each point to its place."""
    pos = b.download(0)[0]
    at = {p.tobytes(): i for i, p in enumerate(before)}
    d = np.zeros_like(pos)
    d[4:] = after[[at[p.tobytes()] for p in pos[4:]]] - pos[4:]
    return d


def same(b, pos):
    assert not b.validate().any()
    assert np.array_equal(b.download(0)[0], pos)
    assert np.array_equal(b.edges(0), O.Mesh.build(pos[4:], exact=True).edges())


# 24 hubs in 100 are wide after the first stars, 92 after the next (counted on the
# CPU): the overflow rows, one for 64 vertices, run out in the second of these rounds,
# which takes 100,000 of the 210,000 vertices
@pytest.mark.parametrize("count,single", [(4000, 126000), (300, 2000)])
def test_rows_run_out_in_a_later_round(M, count, single):
    import torch

    before, after = wheels(count, single, 20, 0.1, 1)
    b = M.MeshBatch.from_points([before.copy()])
    pos = b.download(0)[0]
    for d in (moved_to(b, before, after), None, None):
        if d is None:
            d = np.zeros_like(pos)
            d[4:] = np.random.default_rng(2).standard_normal((len(pos) - 4, 2)) * 1e-3 * 8192 / np.sqrt(len(pos))
        st = b.step(torch.from_numpy(d).cuda())
        assert st["status"] == 0, st
        pos = (pos + d).astype(np.float32)
        same(b, pos)
    b.close()


def test_rows_run_out_in_a_build(M):
    _, p = wheels(6000, 0, 20, 0.0, 3)
    b = M.MeshBatch.from_points([p.copy()])
    same(b, b.download(0)[0])
    b.close()
