"""The benchmark's record of an untangling step, from marks and counters as the kernel
leaves them after stars and after removal."""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402

STALE = 1_800_000_000_000_000_000  # a mark of an earlier launch


def test_stars():
    tl = np.full(48, STALE, np.int64)
    tl[0], tl[1], tl[43] = 1000, 81_000, 451_000
    tl[2:5] = [600_000, 700_000, 750_000]
    tl[44:48] = [900_000, 910_000, 1_050_000, 1_060_000]
    cn = np.zeros(32, np.int64)
    st = {"insert_rounds": 4, "lawson_rounds": 0, "lawson_flips": 0, "removal_flips": 0, "incircle_tests": 9_000_000}
    r = bench.untangle_record(tl, np.zeros(96, np.int64), np.zeros(64, np.int64), cn, st)
    assert r["by"] == "stars" and len(r["phases"]) == len(bench.PHASES["stars"])
    assert r["phases"].tolist() == [80.0, 370.0, 449.0, 10.0, 140.0, 10.0]
    assert r["rounds"] == {"stars": 3} and r["detail"] == {"round_us": [149.0, 100.0, 50.0]}
    # nothing is flipped: the tests of circles among candidates are no work-list items
    assert bench.untangle_bytes(10, 20, st, "stars") == 32 * 10 + 16 * 20


def test_removal():
    tl = np.full(48, STALE, np.int64)
    tl[0], tl[1] = 0, 80_000
    tl[43:48] = [100_000, 300_000, 500_000, 600_000, 610_000]
    trm, tin = np.zeros(96, np.int64), np.zeros(64, np.int64)
    trm[48:50] = [90_000, 99_000]
    trm[0:3], trm[4:7] = [110_000, 120_000, 200_000], [210_000, 220_000, 290_000]
    trm[64:66], trm[80] = [5000 << 16 | 7, 100 << 16 | 6], 1
    tin[0:4] = [320_000, 340_000, 400_000, 450_000]
    cn = np.zeros(32, np.int64)
    cn[14:16] = 2
    st = {"insert_rounds": 1, "lawson_rounds": 9, "lawson_flips": 3, "removal_flips": 2, "incircle_tests": 26}
    r = bench.untangle_record(tl, trm, tin, cn, st)
    assert r["by"] == "removal" and r["phases"].tolist() == [80.0, 20.0, 200.0, 200.0, 100.0, 10.0]
    assert r["rounds"] == {"fixpoint_passes": 2, "removal": 2, "insertion": 1, "flip": 9}
    assert r["detail"]["send_back_pass_us"] == [10.0, 9.0]
    assert r["detail"]["removal_round_us"] == [[10.0, 10.0, 80.0], [10.0, 10.0, 70.0]]
    assert r["detail"]["insertion_round_us"] == [[20.0, 20.0, 60.0]]
    assert r["detail"]["slowest_removal_cycles_spokes"] == [[5000, 7], [100, 6]]
    assert r["detail"]["uncached_removals"] == [1, 0]
    assert bench.untangle_bytes(10, 20, st, "removal") == 32 * 10 + 16 * 20 + 20 * 10 + 96 * 5
