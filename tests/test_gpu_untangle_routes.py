"""Which way a step with turned faces goes: stars (no edge is flipped), removal and
reinsertion, removal after stars that could not be made, and stars after a send-back
that took most of the mesh.  Every mesh equals the oracle's exact triangulation."""
import numpy as np
import pytest

from helpers import gaussian_disp, spacing, uniform_points
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


def step(b, pos, d, meshes=(0,)):
    """One step of the batch; checks it against the oracle and returns (stats, positions)."""
    import torch

    st = b.step(torch.from_numpy(np.ascontiguousarray(d, np.float32)).cuda())
    assert st["status"] == 0, st
    assert not b.validate().any()
    pos = (pos + d).astype(np.float32)
    for i in meshes:
        v0, nv = int(b.v0[i]), int(b.nv[i])
        assert np.array_equal(b.download(i)[0], pos[v0:v0 + nv])
        assert np.array_equal(b.edges(i), O.Mesh.build(pos[v0 + 4:v0 + nv], exact=True).edges())
    return st, pos


def positions(b):
    return np.concatenate([b.download(i)[0] for i in range(b.count)])


@pytest.mark.parametrize("spokes", [127, 128, 129, 150])
def test_a_star_wider_than_the_lists(M, spokes):
    """A hub that stars have no room for, from 129 spokes on: each step goes by removal, the
    two after the first without trying stars (which test a circle for each vertex at
    least), and stars come back, within as many steps as they were left out for, once the
    hub has closed."""
    c = np.array([4096.0, 4096.0])
    p = uniform_points(3000, spokes)
    p = p[np.hypot(*(p - c).T) > 700]
    a = np.linspace(0, 2 * np.pi, spokes, endpoint=False) + 0.1
    p = np.concatenate([p, c[None], c + 600 * np.stack([np.cos(a), np.sin(a)], 1)]).astype(np.float32)
    b = M.MeshBatch.from_points([p])
    pos = positions(b)
    near = np.hypot(*(pos - c).T) < 650
    rng = np.random.default_rng(spokes)
    walk = gaussian_disp(b.V, 0.3 * spacing(3000), spokes, clamp_pos=pos)
    walk[np.hypot(*(pos - c).T) < 1000] = 0
    back = (pos - (pos + walk).astype(np.float32)).astype(np.float32)
    tests = []
    for k in range(9):  # there and back
        st, pos = step(b, pos, back if k % 2 else walk)
        assert st["inverted_faces"] > 0
        widest = np.bincount(b.edges(0).ravel()).max()
        assert widest >= spokes
        assert st["lawson_flips"] > 0 or widest <= 128
        tests.append(st["incircle_tests"])
    if spokes > 128:
        made = np.count_nonzero(walk.any(1))
        assert tests[2] + made // 2 < tests[0], tests
    d = np.zeros_like(pos)
    rim = near & (np.hypot(*(pos - c).T) > 1)
    d[rim] = rng.standard_normal((rim.sum(), 2)) * 40
    st, pos = step(b, pos, d)
    by_stars = []
    for k in range(9):
        st, pos = step(b, pos, gaussian_disp(b.V, 0.3 * spacing(3000), 71 * k + spokes, clamp_pos=pos))
        by_stars.append(st["lawson_flips"] == 0)
    assert by_stars[-1]
    b.close()


@pytest.mark.parametrize("tile", [0, 1, 32])
def test_few_movers_of_a_large_mesh(M, tile):
    """Above 200,000 vertices steps that move few of them go by removal; the mesh beside
    it is active in every other step."""
    b = M.MeshBatch.from_points([uniform_points(200500, 1), uniform_points(3000, 2)])
    b.set_tuning(removal_tile=tile)
    pos = positions(b)
    rng = np.random.default_rng(tile)
    for k in range(4):
        b.set_active([0] if k % 2 else None)
        d = np.zeros_like(pos)
        m = rng.integers(4, b.nv[0], 2000)
        d[m] = rng.standard_normal((2000, 2)) * 0.5 * spacing(200500)
        if k % 2 == 0:
            m = rng.integers(b.v0[1] + 4, b.V, 30)
            d[m] = rng.standard_normal((30, 2)) * 0.5 * spacing(3000)
        d[(pos + d < 0).any(1) | (pos + d >= 8192).any(1)] = 0
        st, pos = step(b, pos, d, (0, 1))
        assert st["inverted_faces"] > 0
        # the first step classifies every edge: whether few move is known from the last
        if k:
            assert st["lawson_flips"] > 0 and st["insert_rounds"] > 0
    b.close()


def test_few_turned_faces_of_a_large_mesh(M):
    """From 850,000 vertices on few open edges go by removal, many by stars."""
    n = 900000
    b = M.MeshBatch.from_points([uniform_points(n, 3)])
    pos = positions(b)
    st, pos = step(b, pos, gaussian_disp(b.V, 0.001 * spacing(n), 1, clamp_pos=pos))
    assert st["inverted_faces"] > 0 and st["lawson_flips"] > 0
    st, pos = step(b, pos, gaussian_disp(b.V, 0.1 * spacing(n), 2, clamp_pos=pos))
    assert st["inverted_faces"] > 0 and st["lawson_flips"] == 0
    b.close()


@pytest.mark.parametrize("n,far", [(900000, 3.0)])
def test_neighbours_that_move_together_far(M, n, far):
    """A swirl of several spacings a step turns few faces; sending their vertices back
    would send back their neighbours in turn."""
    b = M.MeshBatch.from_points([uniform_points(n, 4)])
    pos = positions(b)
    for k in range(2):
        u = (pos.astype(np.float64) / 8192 * 6.2 + 0.04) * (1 + 0.001 * k)
        d = np.stack([np.sin(u[:, 0]) * np.cos(u[:, 1]), -np.cos(u[:, 0]) * np.sin(u[:, 1])], 1) * far * spacing(n)
        d[:4] = 0
        st, pos = step(b, pos, d.astype(np.float32))
        assert st["inverted_faces"] > 0 and st["lawson_flips"] == 0, st
    b.close()


@pytest.mark.parametrize("n,movers,stars", [(3000, 20, True), (6000, 20, False), (40000, 400, False)])
def test_few_that_move_far(M, n, movers, stars):
    """A handful of vertices that jump several spacings go by removal, but in the smallest
    meshes; the rest of the mesh does not move."""
    b = M.MeshBatch.from_points([uniform_points(n, 5)])
    pos = positions(b)
    rng = np.random.default_rng(n)
    d = np.zeros_like(pos)
    m = rng.choice(np.arange(4, b.V), movers, replace=False)
    d[m] = rng.uniform(200, 8000, (movers, 2)) - pos[m]
    far = np.abs(d).max(1) > 8 * spacing(n)
    d[far] *= 8 * spacing(n) / np.abs(d[far]).max(1)[:, None]
    st, pos = step(b, pos, d)
    assert st["inverted_faces"] > 6 * movers
    assert (st["lawson_flips"] == 0) == stars
    b.close()


@pytest.mark.parametrize("n,part,far,stars", [
    (20000, 0.45, 3.0, True), (40000, 0.45, 1.0, True), (40000, 0.45, 4.0, False), (40000, 1.0, 2.0, True),
    (120000, 0.1, 3.0, False), (120000, 0.3, 1.0, True), (120000, 0.7, 4.0, False), (300000, 0.45, 2.0, False)])
def test_some_that_move_far(M, n, part, far, stars):
    """A part of the vertices moves several spacings while the rest stays: removal once
    most of the faces that have a mover are turned."""
    b = M.MeshBatch.from_points([uniform_points(n, 6)])
    pos = positions(b)
    d = gaussian_disp(len(pos), far * spacing(n), 7, pos)
    d[np.random.default_rng(8).random(len(d)) >= part] = 0
    st, pos = step(b, pos, d)
    assert (st["lawson_flips"] == 0) == stars, st
    b.close()
