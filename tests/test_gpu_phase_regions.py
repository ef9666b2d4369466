"""Region counts of mbcg_phase_statistics where most warps hold several regions, lanes without any and (at
the end of the lattice) lanes without a node: random fields at odd sizes, against scipy's labelling."""
import numpy as np
import pytest

import mbcg

pytestmark = pytest.mark.gpu


def regions(p, red):
    """(count, largest, detached, detached volume) of the face-connected regions of red (z, y, x)."""
    ndimage = pytest.importorskip("scipy.ndimage")
    lab, n = ndimage.label(red)
    parent = np.arange(n + 1)

    def root(i):
        while parent[i] != i:
            i = parent[i]
        return i

    for a in range(3):  # regions joined across periodic ends
        if p.bc[a] == mbcg.BC_PERIODIC:
            lo, hi = np.take(lab, 0, 2 - a), np.take(lab, -1, 2 - a)
            for i, j in set(zip(lo[(lo > 0) & (hi > 0)], hi[(lo > 0) & (hi > 0)])):
                i, j = root(i), root(j)
                parent[max(i, j)] = min(i, j)
    lab = np.array([root(i) for i in range(n + 1)])[lab]
    ids, size = np.unique(lab[lab > 0], return_counts=True)
    ia = next((a for a in range(3) if p.bc[a] == mbcg.BC_INOUT), None)
    attached = set(np.unique(np.take(lab, 0, 2 - ia))) if ia is not None else set()
    detached = [s for i, s in zip(ids, size) if i not in attached]
    return len(ids), int(size.max()), len(detached), int(sum(detached))


@pytest.mark.parametrize("fill", [0.02, 0.25, 0.33, 0.7])
@pytest.mark.parametrize("size,axis", [((7, 5, 3), None), ((33, 31, 29), None), ((37, 41, 43), 1), ((97, 61, 53), 2),
                                       ((211, 97, 83), 0)])
def test_regions_of_random_fields(size, axis, fill):
    p = mbcg.bubble_params(8, q=19)
    p.nx, p.ny, p.nz = (s + 2 for s in size)
    p.ic = mbcg.IC_NONE
    if axis is not None:
        p.bc[axis] = mbcg.BC_INOUT
        p.jet_phase = 1.0  # red is tracked
    red = np.random.default_rng(hash((size, fill)) % 2 ** 32).random(size[::-1]) < fill
    red[0, 0, 0] = True
    s = np.zeros((11,) + p.shape, dtype=np.float32)
    s[1] = 1.0
    s[0, 1:-1, 1:-1, 1:-1], s[1, 1:-1, 1:-1, 1:-1] = red, ~red
    with mbcg.Case(p) as c:
        c.copy_in(s)
        st = c.phase_statistics(components=True)
    assert st["status"] == 0 and st["volume_tracked"] == red.sum()
    got = (st["components"], st["largest_component"], st["detached"], st["detached_volume"])
    assert got == regions(p, red)
