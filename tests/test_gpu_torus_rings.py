"""Torus rings after steps that flip, that send vertices back and that remove and
reinsert them, against the rings read off the downloaded mesh: plain stars, one with
more spokes than a query keeps at hand, rows shorter than a star, both layouts, and
calls with neighbour searches in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = 1024.0


@pytest.fixture(scope="module")
def M():
    import torch

    import mcleap_gb300 as M
    from mcleap_gb300 import build as B

    assert torch.cuda.is_available()
    B.build()
    M.lib()
    return M


def rings(t):
    """Per vertex the clockwise (neighbour, offset byte) list from its smallest entry."""
    _, ev, en, eo = t.download()
    nib = lambda w, s: ((w >> s) & 15).astype(np.int64) - 8
    bx, by = nib(eo, 0), nib(eo, 4)
    org = ev[:, :2].reshape(-1)
    dst = ev[:, [1, 0]].reshape(-1)
    off = np.stack([(bx + 8) | ((by + 8) << 4), (8 - bx) | ((8 - by) << 4)], 1).reshape(-1)
    nxt = en[:, [0, 2]].reshape(-1)
    out = [None] * t.n
    for h in range(len(org)):
        v = int(org[h])
        if out[v] is not None:
            continue
        r, g = [], h
        while True:
            r.append((int(dst[g]), int(off[g])))
            g = int(nxt[g ^ 1])
            if g == h:
                break
        k = r.index(min(r))
        out[v] = r[k:] + r[:k]
    return out


def check(M, t, cap):
    import torch

    want = rings(t)
    ring = torch.full((t.n * cap,), -7, dtype=torch.int32, device="cuda")
    offs = torch.full((t.n * cap,), 77, dtype=torch.uint8, device="cuda")
    cut = t.oneRing(cap, ring, offs)
    got, go = ring.view(cap, t.n).cpu().numpy(), offs.view(cap, t.n).cpu().numpy()
    assert cut == sum(len(r) > cap - 1 for r in want)
    for v, r in enumerate(want):
        k = min(len(r), cap - 1)
        assert got[0, v] == k
        assert [(int(a), int(b)) for a, b in zip(got[1:k + 1, v], go[1:k + 1, v])] == r[:k], v
        assert (got[k + 1:, v] == -7).all()


@pytest.mark.parametrize("spokes", [0, 14, 15, 16, 17, 40])
def test_rings_follow_the_steps(M, spokes):
    import torch

    rng = np.random.default_rng(spokes)
    p = rng.random((1500, 2)) * L
    if spokes:
        c = np.array([0.5 * L, 0.5 * L])
        p = p[np.abs(p - c).max(1) > 140]
        a = np.linspace(0, 2 * np.pi, spokes, endpoint=False) + 0.1
        p = np.concatenate([p, c[None], c + 100 * np.stack([np.cos(a), np.sin(a)], 1)])
    p = (2 * L + p).astype(np.float32)
    t = M.PeriodicTriangulation(p, L)
    check(M, t, 48)
    near = torch.zeros(t.n * 32, dtype=torch.int32, device="cuda")
    for k, sigma in enumerate([1.0, 0.2, 3.0, 14.0, 1.0, 8.0, 0.5]):
        d = (rng.standard_normal((t.n, 2)) * sigma).astype(np.float32)
        if sigma < 2 and spokes:
            d[-spokes - 1:] = 0
        st = t.step(torch.from_numpy(d).cuda())
        assert st["status"] == 0
        if k % 3 == 2:
            t.getFRNN(32, 10.0, near)
        check(M, t, 48 if k % 2 else 6)
