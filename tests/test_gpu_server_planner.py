"""The server's planner: what it reports is the cut it uses."""
import numpy as np
import pytest

import mbcg
from gpu_util import written_nodes

pytestmark = pytest.mark.gpu

DEPTHS = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 512}


def planned(p, steps=3, **kw):
    """(depth reported, statistics, state) of a lattice served alone."""
    with mbcg.Server(arena_bytes=8 << 30, keep_results=1, **kw) as srv:
        rid = srv.submit(p, steps)
        info = srv.wait(rid)
        assert info.state == mbcg.REQ_DONE and info.status == 0
        st = srv.stats().as_dict()
        return -(-st["zchunk"] // st["zsplit"]), st, srv.fetch(rid, p.shape)[written_nodes(p)]


def test_reported_cut():
    # 9 tiles side by side: whole tiles of 8 planes (72) leave half of the SMs idle
    small = mbcg.bubble_params(64, q=27)
    depth, st, state = planned(small, calibrate=1)
    assert depth in DEPTHS and st["zsplit"] > 1 and depth < st["zchunk"], st
    # the depth reported, asked for: the same tiles
    again, st2, state2 = planned(small, calibrate=0, zchunk=depth)
    assert (again, st2["zchunk"], st2["zsplit"]) == (depth, depth, 1)
    np.testing.assert_array_equal(state, state2)
    # 63 tiles side by side, 192 planes: deep tiles fill the SMs, and a part more only adds its two planes
    depth, st, _ = planned(mbcg.bubble_params(192, q=27), calibrate=1)
    assert depth in DEPTHS and st["zsplit"] == 1 and st["zchunk"] == depth >= 8, st


def test_long_lattice_at_depth_one():
    """More planes than a tile's 16-bit index counts."""
    p = mbcg.bubble_params(8, q=19, radius=3.0)
    p.nx, p.ny, p.nz = 4, 4, 66005
    p.bubble_center[2] = 65990.0
    got = [planned(p, steps=3, calibrate=0, zchunk=z)[2] for z in (1, 64)]
    assert np.ptp(got[1][0]) > 0.1
    np.testing.assert_array_equal(got[0], got[1])
