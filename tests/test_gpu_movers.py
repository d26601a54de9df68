"""Steps that move few vertices: only the movers' stars are classified, sixteen spokes
at a time.  Hubs on both sides of that, moved alone, with others, so far that faces turn
over, and not at all, against the oracle's exact triangulation."""
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


@pytest.mark.parametrize("spokes", [3, 15, 16, 17, 31, 32, 33, 70])
def test_few_movers(M, spokes):
    import torch

    c = np.array([4096.0, 4096.0])
    p = uniform_points(4000, spokes)
    p = p[np.abs(p - c).max(1) > 700]
    a = np.linspace(0, 2 * np.pi, spokes, endpoint=False) + 0.1
    p = np.concatenate([p, c[None], c + 500 * np.stack([np.cos(a), np.sin(a)], 1)]).astype(np.float32)
    b = M.MeshBatch.from_points([p])
    pos = b.download(0)[0]
    hub = int(np.argmin(np.abs(pos - c).sum(1)))
    rng = np.random.default_rng(spokes)
    for k, (far, others) in enumerate([(0.0, 0), (30.0, 0), (-200.0, 3), (900.0, 0), (0.0, 5), (-800.0, 20), (1.0, 0)]):
        d = np.zeros((b.V, 2), np.float32)
        d[rng.integers(4, b.V, others)] = rng.standard_normal((others, 2)) * 20
        d[hub] = (far, 0.7 * far)
        st = b.step(torch.from_numpy(d).cuda())
        assert st["status"] == 0, st
        assert not b.validate().any()
        pos = (pos + d).astype(np.float32)
        assert np.array_equal(b.download(0)[0], pos)
        assert np.array_equal(b.edges(0), O.Mesh.build(pos[4:], exact=True).edges()), k
    b.close()
