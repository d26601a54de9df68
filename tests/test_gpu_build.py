"""The build against the oracle: the points' order bit for bit (the device's sort,
and the host's where Morton keys are equal), the exact triangulation's edges, and a
step on the built mesh.  Sizes sit where the forms meet: no point, fewer points than
a warp's candidates need, one block of the sort more or less, several warps' runs;
sets with equal keys, with so many that insertion takes over, on a lattice, on a
circle, in clusters, and at negative coordinates up to the square's border."""
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


def check(M, pts):
    import torch

    from mcleap_gb300.batch import build_mesh

    got = pts.copy()
    b = M.MeshBatch(build_mesh(got))
    want = O.morton_sort(pts) if len(pts) else pts
    assert np.array_equal(got, want)
    assert not b.validate().any()
    pos, _, he, t = b.download(0)
    c = np.float32(1e7)
    assert np.array_equal(pos[:4], np.array([[-c, -c], [c, -c], [c, c], [-c, c]]))
    assert np.array_equal(pos[4:], want)
    if len(pts):
        assert np.array_equal(b.edges(0), O.Mesh.build(want, exact=True).edges())
    d = np.zeros((b.V, 2), np.float32)
    if len(pts):
        gap = np.sqrt(np.prod(np.ptp(pts, axis=0) + 1.0) / len(pts))
        d[4::7] = np.random.default_rng(5).standard_normal(d[4::7].shape) * 0.2 * gap
        d[np.abs(pos).max(axis=1) > 9.9e6] = 0
    moved = (pos + d).astype(np.float32)
    st = b.step(torch.from_numpy(d).cuda())
    assert st["status"] == 0, st
    assert not b.validate().any()
    if len(pts):
        assert np.array_equal(b.edges(0), O.Mesh.build(moved[4:], exact=True).edges())
    b.close()


@pytest.mark.parametrize("n", [0, 1, 2, 3, 4, 31, 32, 33, 255, 256, 257, 2047, 2049, 30000, 117001])
def test_uniform(M, n):
    check(M, uniform_points(n, n + 1) if n else np.zeros((0, 2), np.float32))


@pytest.mark.parametrize("kind", ["some ties", "mostly ties", "lattice", "circle", "clusters", "negative", "border", "line"])
def test_sets(M, kind):
    rng = np.random.default_rng(len(kind))
    n = 6000
    if kind == "some ties":
        p = rng.random((n, 2)) * 400
    elif kind == "mostly ties":
        p = rng.random((n, 2)) * 8
    elif kind == "lattice":
        p = np.stack(np.meshgrid(np.arange(77), np.arange(77)), -1).reshape(-1, 2) * 16.0 + 1024
        p = rng.permutation(p)
    elif kind == "circle":
        a = np.linspace(0, 2 * np.pi, 700, endpoint=False)
        p = np.concatenate([[[4096, 4096]], 4096 + 3000 * np.stack([np.cos(a), np.sin(a)], 1)])
    elif kind == "clusters":
        p = 4096 + rng.standard_normal((n, 2)) * np.where(np.arange(n) % 3, 900, 30)[:, None]
    elif kind == "negative":
        p = (rng.random((n, 2)) - 0.5) * 8000
    elif kind == "border":
        p = np.concatenate([(rng.random((n, 2)) * 2 - 1) * 9.99e6, [[9999999, 0], [0, -9999999], [-9999999, 9999999]]])
    else:
        p = np.stack([rng.permutation(n) * 2.0, np.full(n, 77.0)], 1)
    p = p.astype(np.float32)
    check(M, p[np.sort(np.unique(p, axis=0, return_index=True)[1])])
