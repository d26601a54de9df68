"""The launch shape a mesh reports is the one its steps use."""
import numpy as np
import pytest

from helpers import spacing, uniform_points

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


def test_reported_tail_is_the_one_used(M):
    """Setting what was read changes nothing, and 0 brings the default back."""
    b = M.MeshBatch.from_points([uniform_points(500, 1)])
    t = b.tuning()
    assert t["tail_items"] == 256 and t["blocks_per_sm"] == t["max_blocks_per_sm"]
    b.set_tuning(t["blocks_per_sm"], t["tail_items"])
    assert b.tuning() == t and b.clone().tuning() == t
    b.set_tuning(1, 2048)
    assert b.tuning()["tail_items"] == 2048 and b.tuning()["blocks_per_sm"] == 1
    assert b.clone().tuning()["tail_items"] == 2048
    b.set_tuning()
    assert b.tuning() == t
    b.close()
