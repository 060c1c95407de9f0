"""Dual contouring's bit masks, ranks and work lists (csrc/dc.cu) against the
oracle, bit for bit, where they can go wrong: random values, so that almost
every edge crosses and a leaf's lists are near their longest (1,536 crossings,
512 cells); grids whose ends lie inside, on and one voxel past a leaf's end;
one leaf, a row of leaves, all 27 neighbours; holes (inactive voxels) cut on
whole planes, which leave every gradient a neighbour."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from oracle import binding as ob
from tests.gpu_common import context

pytestmark = pytest.mark.gpu


def multiset(t):
    u = np.ascontiguousarray(t, np.float32).reshape(-1, 9).view(np.uint32)
    return u[np.lexsort(u.T[::-1])]


@pytest.mark.parametrize("dims,lo", [((8, 8, 8), (0, 0, 0)), ((2, 2, 2), (7, 7, 7)), ((9, 8, 8), (0, 0, 0)),
                                     ((8, 9, 8), (0, 0, 0)), ((8, 8, 9), (0, 0, 0)), ((7, 16, 17), (-3, 5, -9)),
                                     ((24, 24, 24), (-8, -8, -8)), ((3, 40, 5), (6, -20, 100)), ((5, 3, 33), (-5, 7, 7))])
@pytest.mark.parametrize("holes", [False, True])
def test_random_values_match_oracle(dims, lo, holes):
    rng = np.random.default_rng(sum(dims) + 7 * holes)
    h, band = np.float32(0.5), 3
    vals = rng.uniform(-1.9, 1.9, dims).astype(np.float32)
    vals.flat[:: 17] = rng.choice(np.array([0.0, -0.0, 1.25, -1.25], np.float32), len(vals.flat[:: 17]))
    if holes:  # planes of far values are inactive; both sides keep two voxels or more
        for ax in range(3):
            if dims[ax] >= 5:
                np.moveaxis(vals, ax, 0)[dims[ax] // 2] = 9.0
    vmin = np.asarray(lo, np.float32) * h
    vmax = (np.asarray(lo) + np.asarray(dims) - 1).astype(np.float32) * h
    g = bs.Volume.from_fn(h, vmin, vmax, band, lambda p: vals.ravel(), ctx=context())
    o = ob.volume_from_samples(h, band, np.asarray(lo), vals)
    want, status, crossings, cells = o.dual_contour()
    if status == 0:
        got = bs.DualContouringMesher().with_voxel_size(float(h)).mesh(g)
        st = context().last_stats()
        assert (st["crossings"], st["cells"]) == (crossings, cells)
        assert got.shape == want.shape
        assert np.array_equal(multiset(got), multiset(want))
    else:
        with pytest.raises(bs.BsError):
            bs.DualContouringMesher().with_voxel_size(float(h)).mesh(g)
