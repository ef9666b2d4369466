"""The batch kernels on lattices whose non-periodic axis is x or y (and on z axes too short for end tiles).

There a CTA draws tiles that touch the boundary and tiles clear of it by turns, and the two kinds run
different bodies, which synchronise their warps differently: what one leaves behind must not reach the next.
So every lattice here has more tiles than the GPU has SMs, cut at an odd depth (an odd number of planes a
tile, depth + 2).

Gates: served alone and in the mix, the same bits (fetched fields and state hash); against the FP64 oracle
the FP32 parity gate; a server that cuts the tiles at an even depth stores the same bits as well."""
import numpy as np
import pytest

import mbcg
import oracle_lib as ol
from gpu_util import assert_fp32_parity, written_nodes
from test_gpu_step_tiles import make

pytestmark = pytest.mark.gpu

DEPTH = 7


def lattices(q):
    """(parameters, steps, what): inlets and walls along x and y, and z walls without end tiles (nz < 10).
    The jets run until the inlet's pressure wave has crossed most of the tiles clear of it."""
    out = []
    for kind, axis, size, steps in (("jet", 1, (118, 110, 63), 60), ("jet", 0, (121, 86, 63), 60),
                                    ("wall", 0, (118, 108, 63), 6), ("wall", 1, (90, 132, 84), 7),
                                    ("wall", 2, (360, 330, 7), 6)):
        p = make(kind, axis, q, size)
        p.jet_radius = 0.4 * min(size)
        if kind == "wall":  # (make()'s interface is that of a box of a few nodes)
            p.rti_amplitude = 0.2 * size[axis]
        out.append((p, steps, f"{kind} axis {axis} q{q} {size}"))
    return out


def serve(cases, depth, together):
    res = []
    with mbcg.Server(arena_bytes=6 << 30, keep_results=1, chunk_steps=3, calibrate=0, zchunk=depth) as srv:
        ids = [srv.submit(p, n) for p, n, _ in cases] if together else []
        for i, (p, n, what) in enumerate(cases):
            rid = ids[i] if together else srv.submit(p, n)
            info = srv.wait(rid)
            assert info.state == mbcg.REQ_DONE and info.status == 0 and info.diag.nonfinite == 0, what
            res.append((info.state_hash, srv.fetch(rid, p.shape)[written_nodes(p)]))
            srv.release(rid)
    return res


@pytest.mark.parametrize("q", [19, 27])
def test_boundaries_along_x_and_y_served(q):
    cases = lattices(q)
    alone = serve(cases, DEPTH, False)
    for (p, n, what), (_, got) in zip(cases, alone):
        a0 = ol.oracle_init(p, np.float64)
        o64 = ol.oracle_run(p, a0.copy(), n)[written_nodes(p)]
        o32 = ol.oracle_run(p, a0.astype(np.float32), n)[written_nodes(p)]
        assert_fp32_parity(got, o64, o32, None, what=what)
    for depth, together in ((DEPTH, True), (DEPTH, True), (DEPTH, False), (DEPTH + 1, True)):
        for (_, _, what), (h0, f0), (h, f) in zip(cases, alone, serve(cases, depth, together)):
            assert h == h0, (what, depth, together)
            np.testing.assert_array_equal(f, f0, err_msg=f"{what} depth {depth} together {together}")
