"""The step kernel at the edges of its tiles, against the FP64 oracle.

A tile owns 30 columns and 22 (or 6) rows of a chunk of planes; on a non-periodic z axis the first and
the last two fluid planes are tiles of their own, and tiles clear of the non-periodic axis run a body
without its parts.  The sizes are the smallest lattice, one below, at and above a tile's extent on each
axis, and the plane counts at which the end tiles appear, with the non-periodic axis along x, y and z.

Gate: the FP32 parity gate (relative L2 1e-5 per group, or 3x the reference arithmetic's own distance
from the FP64 oracle)."""
import numpy as np
import pytest

import mbcg
import oracle_lib as ol
from gpu_util import assert_fp32_parity, written_nodes

pytestmark = pytest.mark.gpu

STEPS = 3
# fluid nodes (x, y, z)
SIZES = [(2, 2, 2), (29, 22, 7), (30, 21, 8), (31, 23, 9), (32, 6, 12), (61, 45, 5)]


def make(kind, axis, q, size):
    nx, ny, nz = (s + 2 for s in size)
    p = mbcg.reference_jet_params(nx, ny, nz, q=q, tau=0.7, sigma=0.05, beta=0.7, radius=0.3 * min(size) + 0.6)
    for a in range(3):
        p.bc[a] = mbcg.BC_PERIODIC
    n = (nx, ny, nz)
    if kind == "periodic":
        p.ic = mbcg.IC_BUBBLE
        p.bubble_radius, p.bubble_width, p.bubble_phase = 0.3 * min(size) + 0.6, 2.0, 1.0
    else:
        p.bc[axis] = mbcg.BC_WALL if kind == "wall" else mbcg.BC_INOUT
        t = [a for a in range(3) if a != axis]
        p.jet_center[0], p.jet_center[1] = (n[t[0]] - 1) / 2.0, (n[t[1]] - 1) / 2.0
        if kind == "wall":
            p.ic = mbcg.IC_RTI
            p.rho_r0, p.rho_b0 = 3.0, 1.0
            p.gravity[axis] = -1e-4
            p.rti_position, p.rti_amplitude, p.rti_width = n[axis] / 2.0, 0.5, 2.0
        else:
            p.inlet_noise = 0.01
    return p


def state_of(p):
    a = ol.oracle_init(p, np.float64)
    z, y, x = np.meshgrid(*(np.arange(k) for k in p.shape), indexing="ij")
    for c, (s, n) in enumerate(((y, p.ny), (z, p.nz), (x, p.nx))):
        a[2 + c] += 0.01 * (0.4 + np.sin(2 * np.pi * (s - 1) / (n - 2) + c))
    for ax in range(3):  # ghost layers of periodic axes hold the images; walls are at rest
        d, n = 3 - ax, p.shape[2 - ax]
        lo, hi = [slice(None)] * 4, [slice(None)] * 4
        lo[d], hi[d] = 0, n - 1
        src_lo, src_hi = list(lo), list(hi)
        src_lo[d], src_hi[d] = n - 2, 1
        if p.bc[ax] == mbcg.BC_PERIODIC:
            a[tuple(lo)], a[tuple(hi)] = a[tuple(src_lo)], a[tuple(src_hi)]
        elif p.bc[ax] == mbcg.BC_WALL:
            for s in (lo, hi):
                a[tuple([slice(2, 5)] + s[1:])] = 0.0
    return a.astype(np.float32).astype(np.float64)


CASES = [("periodic", 0)] + [(k, a) for k in ("wall", "jet") for a in range(3)]


@pytest.mark.parametrize("q", [19, 27])
@pytest.mark.parametrize("kind,axis", CASES)
def test_tile_edges(kind, axis, q):
    for size in SIZES:
        p = make(kind, axis, q, size)
        a = state_of(p)
        o64 = ol.oracle_run(p, a.copy(), STEPS)
        o32 = ol.oracle_run(p, a.astype(np.float32), STEPS)
        idx = written_nodes(p)
        first = None
        for shape in ((16, 5), (8, 2)):
            with mbcg.Case(p) as c:
                c.set_shape(*shape)
                c.copy_in(a.astype(np.float32))
                c.step(STEPS)
                got = c.copy_out()
                assert c.status() == 0
            assert_fp32_parity(got, o64, o32, idx, what=f"{kind} axis {axis} q{q} {size} shape {shape}")
            # the tiling never shows in the bits
            if first is None:
                first = got
            np.testing.assert_array_equal(got[idx], first[idx], err_msg=f"{kind} {axis} q{q} {size}")


@pytest.mark.parametrize("precision", [mbcg.FP16, mbcg.BF16])
def test_pure_nodes_keep_their_colour_in_16_bits(precision):
    """A minority density that rounds below zero must not turn the colour slot's sign: after a step of
    the density-ratio case from the same state, phi of the 16-bit form stays within the form's
    resolution of FP32's at every node (half of it stored, as much again read back: 2^-10 and 2^-7)."""
    p = mbcg.rti_params(64, 192, q=27)
    a = ol.oracle_init(p, np.float64).astype(np.float32)
    z, y, x = np.meshgrid(*(np.arange(k) for k in p.shape), indexing="ij")
    a[2] += 0.01 * np.sin(2 * np.pi * (y - 1) / (p.ny - 2)) * np.sin(np.pi * z / (p.nz - 1))
    phi = []
    for prec in (mbcg.FP32, precision):
        p.precision = prec
        with mbcg.Case(p) as c:
            c.copy_in(a)
            c.step(1)
            s = c.copy_out()[:, 1:-1, 1:-1, 1:-1].astype(np.float64)
        phi.append((s[0] - s[1]) / (s[0] + s[1]))
    assert np.abs(phi[0] - phi[1]).max() < 2.0 * (2.0 ** -10 if precision == mbcg.FP16 else 2.0 ** -7)


@pytest.mark.parametrize("precision", [mbcg.FP32, mbcg.FP16])
@pytest.mark.parametrize("size", [(30, 22, 12), (125, 90, 40), (61, 45, 300)])  # one, some, many tiles at once
def test_steps_in_a_row_are_the_steps_one_by_one(size, precision):
    """Steps queued behind each other start their set-up before the one in front is complete: the state
    has to be that of steps each waited for (bit for bit: the arithmetic is the same)."""
    p = make("inout", 2, 27, size)
    p.precision = precision
    got = []
    for alone in (False, True):
        with mbcg.Case(p) as c:
            c.init()
            for n in [1] * 24 if alone else [24]:
                c.step(n)
                if alone:
                    assert c.status() == 0  # (waits for the device)
            assert c.status() == 0
            got.append(c.copy_out())
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))


@pytest.mark.parametrize("kind,axis", [("periodic", 0), ("wall", 0), ("wall", 1), ("wall", 2)])
def test_tiling_does_not_show_in_bf16(kind, axis):
    """Lattices without an inlet in BF16 storage step by populations; tile shape and depth change no bit."""
    for size in SIZES:
        p = make(kind, axis, 27, size)
        p.precision = mbcg.BF16
        a = state_of(p).astype(np.float32)
        idx = written_nodes(p)
        first = None
        for shape in ((16, 5), (8, 2), (16, 64)):
            with mbcg.Case(p) as c:
                c.set_shape(*shape)
                c.copy_in(a)
                c.step(STEPS)
                got = c.copy_out()
                assert c.status() == 0
            assert np.isfinite(got[idx]).all()
            if first is None:
                first = got
            np.testing.assert_array_equal(got[idx], first[idx], err_msg=f"{kind} {axis} {size} {shape}")
