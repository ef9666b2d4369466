"""A lattice stores the same state whichever way it is stepped: through a case, through the server, and with
staging by plain loads instead of TMA.  Gate: the same bits.  (In the 16-bit forms nothing less holds for long:
the rounding of a stored slot turns a last bit of FP32 into a unit of the form.)"""
import numpy as np
import pytest

import mbcg
from gpu_util import written_nodes
from test_gpu_step_tiles import make

pytestmark = pytest.mark.gpu

STEPS = 12


def walls(axis, size, q):
    p = make("wall", axis, q, size)
    p.rti_amplitude = 0.2 * min(size)
    return p


def lattices(prec, q):
    two_tau = mbcg.rti_params(24, 90, q=q)
    two_tau.tau_b = 0.9
    out = [mbcg.bubble_params(30, q=q), mbcg.bubble_params(61, q=q), mbcg.bubble_params(64, q=q, radius=20.0),
           mbcg.rti_params(31, 64, q=q), two_tau, walls(0, (61, 45, 31), q), walls(1, (45, 61, 31), q),
           walls(2, (33, 47, 7), q), mbcg.jet_params(40, 36, 50, q=q, diameter=10.0), make("jet", 1, q, (35, 49, 31))]
    for p in out:
        p.precision = prec
    return out


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("prec", [mbcg.FP32, mbcg.FP16, mbcg.BF16])
def test_served_single_and_plain_load_states_agree(prec, q, monkeypatch):
    cases = lattices(prec, q)
    single = []
    for p in cases:
        with mbcg.Case(p) as c:
            c.init()
            c.step(STEPS)
            single.append(c.copy_out()[written_nodes(p)])
            assert c.status() == 0 and np.isfinite(single[-1]).all()
    for kw in ({"calibrate": 0}, {"calibrate": 0, "zchunk": 5, "max_live": 3}):
        with mbcg.Server(arena_bytes=1 << 30, keep_results=1, chunk_steps=5, **kw) as srv:
            ids = [srv.submit(p, STEPS) for p in cases]
            for rid, p, ref in zip(ids, cases, single):
                assert srv.wait(rid).state == mbcg.REQ_DONE
                np.testing.assert_array_equal(srv.fetch(rid, p.shape)[written_nodes(p)], ref, err_msg=str(p.describe()))
    monkeypatch.setenv("MBCG_NO_TMA", "1")
    for p, ref in zip(cases, single):
        with mbcg.Case(p) as c:
            c.init()
            c.step(STEPS)
            np.testing.assert_array_equal(c.copy_out()[written_nodes(p)], ref, err_msg=str(p.describe()))


@pytest.mark.parametrize("prec", [mbcg.FP16, mbcg.BF16])
def test_every_body_is_calibrated(prec):
    """The cost model has a rate for each body, and the planner serves 16-bit lattices with it."""
    with mbcg.Server(arena_bytes=2 << 30, calibrate=1, keep_results=1) as srv:
        ns = srv.stats().as_dict()["plane_ns"]
        assert all(v > 1 for v in ns.values()), ns
        for p in lattices(prec, 27):
            info = srv.wait(srv.submit(p, 3))
            assert info.state == mbcg.REQ_DONE and info.status == 0 and info.diag.nonfinite == 0
