"""Untangling by stars against the oracle's exact triangulation, at the sizes
where its forms meet: the smallest meshes, a warp's share of vertices (a warp per
vertex up to it, a thread above), stars wider than a row and wider than a
thread's slots, moves far beyond the old neighbours, clamped collinear points,
and batches that hold meshes with no point.  Edge sets compare bit for bit."""
import numpy as np
import pytest

from helpers import gaussian_disp, spacing, uniform_points
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# the engine takes a warp per vertex up to 8 vertices per warp of the launch
WARP_SHARE = 8 * 8 * 3 * 152


@pytest.fixture(scope="module")
def M():
    import torch

    import mcleap_gb300 as M
    from mcleap_gb300 import build as B

    assert torch.cuda.is_available()
    B.build()
    M.lib()
    return M


def walk(M, sets, disp_of, steps):
    """Step a batch of the point sets; every mesh equals the oracle's rebuild."""
    import torch

    b = M.MeshBatch.from_points([p.copy() for p in sets])
    pos = [b.download(i)[0] for i in range(b.count)]
    made = 0
    for k in range(steps):
        d = np.concatenate([disp_of(i, pos[i], k) for i in range(b.count)]).astype(np.float32)
        st = b.step(torch.from_numpy(d).cuda())
        assert st["status"] == 0, st
        made += st["removed_vertices"]
        assert not b.validate().any()
        for i in range(b.count):
            v0 = int(b.v0[i])
            pos[i] = (pos[i] + d[v0:v0 + len(pos[i])]).astype(np.float32)
            got, _, he, _ = b.download(i)
            assert np.array_equal(got, pos[i])
            if len(pos[i]) > 4:
                assert np.array_equal(b.edges(i), O.Mesh.build(pos[i][4:], exact=True).edges()), (k, i, st)
    b.close()
    return made


@pytest.mark.parametrize("n,sigma", [(1, 1.0), (2, 1.0), (3, 1.0), (20, 0.5), (700, 3.0), (5000, 0.1),
                                     (WARP_SHARE - 4, 0.1), (WARP_SHARE - 3, 0.3), (120001, 0.15)])
def test_random_walks(M, n, sigma):
    made = walk(M, [uniform_points(n, n)],
                lambda i, pos, k: gaussian_disp(len(pos), sigma * spacing(n), 31 * k + n, clamp_pos=pos), 3)
    assert made > 0 or n < 20


def test_wide_stars_and_lattices(M):
    rng = np.random.default_rng(2)
    a = np.linspace(0, 2 * np.pi, 100, endpoint=False)
    wheel = np.concatenate([[[4096, 4096]], 4096 + 2000 * np.stack([np.cos(a), np.sin(a)], 1)]).astype(np.float32)
    g = np.arange(24)
    lattice = np.stack(np.meshgrid(g, g), -1).reshape(-1, 2).astype(np.float32) * 256 + 1024

    def disp(i, pos, k):
        d = np.zeros_like(pos)
        if i == 0:  # the hub keeps its hundred spokes, then the rim scatters
            d[4:] = rng.standard_normal((len(pos) - 4, 2)) * (5, 100, 300)[k % 3]
        elif i == 1 and k % 2 == 0:  # every other column passes its neighbour: collinear points change order
            d[4:, 0] = np.where(np.round(pos[4:, 0] / 256) % 2 == 0, 320, -320)
        return d

    assert walk(M, [wheel, lattice, np.zeros((0, 2), np.float32), uniform_points(40, 1)], disp, 4) > 0
