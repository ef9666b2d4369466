"""Lattices whose layout TMA cannot describe (row pitch not a multiple of 16 bytes, or MBCG_NO_TMA): every
thread stages its own two nodes by plain copies, and next to an x or y boundary the colour gradient's rule
reads a neighbouring thread's.

Gates: the bits of the staging by TMA, on lattices with an interface across the boundary rows of every plane
and tiles cut at several depths; and the FP32 parity gate for the caller's own dense arrays with an odd row
length, as the reference lays them out."""
import numpy as np
import pytest

import mbcg
import oracle_lib as ol
from gpu_util import assert_fp32_parity, gpu_run, written_nodes
from test_gpu_step_tiles import make, state_of

pytestmark = pytest.mark.gpu

STEPS = 4
SIZES = [(30, 21, 8), (31, 23, 9), (95, 61, 45)]


def lattice(kind, axis, q, size):
    """A density field that mixes the colours everywhere, so that every node beside the boundary has a
    colour gradient that changes from plane to plane."""
    p = make(kind, axis, q, size)
    a = state_of(p)
    z, y, x = np.meshgrid(*(np.arange(k) for k in p.shape), indexing="ij")
    phi = 0.8 * np.sin(2 * np.pi * (x - 1) / (p.nx - 2)) * np.cos(2 * np.pi * (y - 1) / (p.ny - 2)) * \
        np.sin(1.9 * z + 0.3 * x + 0.2 * y)
    for ax in range(3):  # ghost layers of periodic axes hold the images
        if p.bc[ax] == mbcg.BC_PERIODIC:
            phi = np.moveaxis(phi, 2 - ax, 0)
            phi[0], phi[-1] = phi[-2], phi[1]
            phi = np.moveaxis(phi, 0, 2 - ax)
    a[0], a[1] = 0.5 * (1 + phi) * p.rho_r0, 0.5 * (1 - phi) * p.rho_b0
    return p, a.astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("kind,axis", [(k, a) for k in ("wall", "jet") for a in range(3)])
def test_plain_copies_stage_what_tma_stages(q, kind, axis):
    for size in SIZES:
        p, a = lattice(kind, axis, q, size)
        idx = written_nodes(p)
        tma = gpu_run(p, a, STEPS, env={"MBCG_ALL_FEATURES": "1"})[idx]  # (as the plain copies' kernel)
        assert np.isfinite(tma).all()
        for depth in (1, 2, 5, 64):
            plain = gpu_run(p, a, STEPS, env={"MBCG_NO_TMA": "1", "MBCG_ZCHUNK": str(depth)})[idx]
            np.testing.assert_array_equal(plain, tma, err_msg=f"{kind} axis {axis} {size} depth {depth}")


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("kind,axis", [("wall", 1), ("jet", 1), ("jet", 0)])
def test_odd_rows_of_the_caller(q, kind, axis):
    torch = pytest.importorskip("torch")
    lib = mbcg.Library.get()
    for size in ((31, 23, 9), (95, 61, 45)):
        p, a = lattice(kind, axis, q, size)
        assert p.nx % 4
        o64 = ol.oracle_run(p, a.copy(), STEPS)
        o32 = ol.oracle_run(p, a.astype(np.float32), STEPS)
        t = [torch.from_numpy(a.astype(np.float32)).cuda() for _ in range(2)]
        m = [mbcg.moments_from_tensors([s[f] for f in range(11)], p.nx) for s in t]
        for k in range(STEPS):
            src, dst = m[k & 1], m[1 - (k & 1)]
            lib.check(lib.mbcg_rcs_moments(p, src, dst, k + 1, None), "rcs")
            lib.check(lib.mbcg_bc_moments(p, dst, src, k + 1, None), "bc")
        torch.cuda.synchronize()
        got = t[STEPS & 1].cpu().numpy()
        assert_fp32_parity(got, o64, o32, written_nodes(p), what=f"{kind} axis {axis} {size}")
