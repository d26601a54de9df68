"""The thread forms of untangling by stars, run vertex by vertex on the CPU against the
oracle: random walks, moves far beyond the neighbours, lattices whose columns pass each
other, wheels wider than a row and than the lists, collinear and single points, and a
batch with an empty mesh."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from helpers import gaussian_disp, spacing, uniform_points
from mcleap_gb300 import build as B
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("star") / "libstar.so")
    r = subprocess.run([B.nvcc(), "-std=c++17", "-O1", "-w", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off",
                        "-gencode", "arch=compute_103a,code=sm_103a", "-I", os.path.join(ROOT, "mcleap_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "star_rounds.cu"), "-o", so], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(so)


def arrays(pts):
    """(pos, ev, en, vhe) of the oracle's triangulation of pts."""
    pos, v, he, _ = O.Mesh.build(pts, exact=True).aos()
    prev = np.zeros(len(he), np.int32)
    prev[he[:, 0]] = np.arange(len(he))
    a, b = he[0::2], he[1::2]
    ev = np.stack([a[:, 1], b[:, 1], np.where(a[:, 2] >= 0, a[:, 3], -1), np.where(b[:, 2] >= 0, b[:, 3], -1)], 1)
    en = np.stack([a[:, 0], prev[0::2], b[:, 0], prev[1::2]], 1)
    return np.asarray(pos, np.float32), ev.astype(np.int32), en.astype(np.int32), v[:, 1].astype(np.int32)


def valid(ev, en, vhe):
    h = np.arange(2 * len(ev))
    org, apex, nx, pv = ev[:, :2].ravel(), ev[:, 2:].ravel(), en[:, [0, 2]].ravel(), en[:, [1, 3]].ravel()
    inner = apex >= 0
    return ((pv[nx] == h).all() and (nx[pv] == h).all() and (org[nx] == org[h ^ 1]).all()
            and (nx[nx[nx]][inner] == h[inner]).all() and (apex[inner] == org[pv][inner]).all()
            and (org[vhe] == np.arange(len(vhe))).all())


class Meshes:
    """Point sets as one batch on the CPU."""

    def __init__(self, sets):
        parts = [arrays(p) for p in sets]
        nv, ne = [len(p[0]) for p in parts], [len(p[1]) for p in parts]
        self.v0 = np.concatenate([[0], np.cumsum(nv)]).astype(np.int32)
        self.e0 = np.concatenate([[0], np.cumsum(ne)]).astype(np.int32)
        self.pos = np.concatenate([p[0] for p in parts])
        self.ev = np.concatenate([np.where(p[1] >= 0, p[1] + v, -1) for p, v in zip(parts, self.v0)]).astype(np.int32)
        self.en = np.concatenate([p[2] + 2 * e for p, e in zip(parts, self.e0)]).astype(np.int32)
        self.vhe = np.concatenate([p[3] + 2 * e for p, e in zip(parts, self.e0)]).astype(np.int32)

    def step(self, lib, d):
        self.pos = np.ascontiguousarray((self.pos + d).astype(np.float32))
        info = np.zeros(5, np.int32)
        p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
        rc = lib.star_untangle(len(self.pos), len(self.ev), p(self.pos), p(self.ev), p(self.en), p(self.vhe),
                               len(self.v0) - 1, p(self.v0), p(self.e0), p(info))
        return rc, dict(zip(("rounds", "made", "rows", "turned", "wide"), info.tolist()))

    def check(self):
        assert valid(self.ev, self.en, self.vhe)
        for i in range(len(self.v0) - 1):
            e = np.sort(self.ev[self.e0[i]:self.e0[i + 1], :2] - self.v0[i], 1)
            pts = self.pos[self.v0[i] + 4:self.v0[i + 1]]
            if len(pts):
                assert np.array_equal(e[np.lexsort((e[:, 1], e[:, 0]))], O.Mesh.build(pts, exact=True).edges())


@pytest.mark.parametrize("n,sigma", [(1, 1.0), (2, 1.0), (3, 1.0), (20, 0.5), (700, 3.0), (1500, 1.0), (4000, 0.1)])
def test_random_walks(lib, n, sigma):
    m = Meshes([uniform_points(n, n)])
    turned = 0
    for k in range(3):
        rc, info = m.step(lib, gaussian_disp(n + 4, sigma * spacing(n), 31 * k + n, clamp_pos=m.pos))
        assert rc == 0, (rc, info)
        turned += info["turned"]
        m.check()
    assert turned > 0 or n < 20


def wheel(spokes):
    a = np.linspace(0, 2 * np.pi, spokes, endpoint=False)
    return np.concatenate([[[4096, 4096]], 4096 + 2000 * np.stack([np.cos(a), np.sin(a)], 1)]).astype(np.float32)


@pytest.mark.parametrize("spokes", [14, 15, 16, 100])
def test_wheels(lib, spokes):
    m = Meshes([wheel(spokes)])
    rng = np.random.default_rng(spokes)
    wide = 0
    for sigma in (5, 60, 300, 5):
        d = np.zeros_like(m.pos)
        d[4:] = rng.standard_normal((spokes + 1, 2)) * sigma
        rc, info = m.step(lib, d.astype(np.float32))
        assert rc == 0, (rc, info)
        wide += info["wide"]
        m.check()
    assert wide > 0 or spokes < 16


def test_lattice_batch(lib):
    g = np.arange(16)
    lattice = np.stack(np.meshgrid(g, g), -1).reshape(-1, 2).astype(np.float32) * 256 + 1024
    m = Meshes([lattice, np.zeros((0, 2), np.float32), uniform_points(40, 1)])
    for k in range(4):
        d = np.zeros_like(m.pos)
        at = slice(4, 4 + len(lattice))
        if k % 2 == 0:  # every other column passes its neighbour
            d[at, 0] = np.where(np.round(m.pos[at, 0] / 256) % 2 == 0, 320, -320)
        d[-40:] = np.random.default_rng(k).standard_normal((40, 2)) * 400
        rc, info = m.step(lib, d.astype(np.float32))
        assert rc == 0, (rc, info)
        m.check()


def test_what_stars_leave_to_removal(lib):
    """A star of more neighbours than the lists hold, coincident points, and a vertex outside
    the square end without a word written to the mesh."""
    m = Meshes([wheel(150)])
    before = m.ev.copy(), m.en.copy(), m.vhe.copy()
    d = np.zeros_like(m.pos)
    d[4 + 7] = 900, 700
    rc, _ = m.step(lib, d)
    assert rc in (1, 2)
    n = uniform_points(300, 3)
    for k in range(2):
        m2 = Meshes([n])
        start = m2.ev.copy()
        d = np.zeros_like(m2.pos)
        d[9] = m2.pos[200] - m2.pos[9] if k == 0 else (3e7, 100)
        rc, _ = m2.step(lib, d)
        assert rc != 0 and np.array_equal(m2.ev, start)
    assert all(np.array_equal(a, b) for a, b in zip(before, (m.ev, m.en, m.vhe)))
