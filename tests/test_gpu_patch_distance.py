"""The patch distance pass (csrc/m2v_patch.cuh) against the oracle, bit for
bit (distances, masks, leaf set), where its cell arithmetic can go wrong:
triangles cut into exactly n^2 sub-triangles for n at the edges of the patch
shapes (one triangle to n = 3, blocks of 2 x 2 cells beyond, odd n with ragged
last blocks), slender ones, degenerate ones beside them, wide bands (which
select the pass), single meshes and a batch."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import synthetic
from oracle import binding as ob
from tests.gpu_common import compare_volumes, context

pytestmark = pytest.mark.gpu


def cut_soup(n, h, count, seed, slender):
    """Triangles whose longest side is between n h and (n + 1) h: n^2 sub-triangles each."""
    rng = np.random.default_rng(seed)
    t = rng.normal(size=(count, 3, 3))
    if slender:
        t[:, 2] = t[:, 0] + rng.uniform(0.1, 0.9, (count, 1)) * (t[:, 1] - t[:, 0]) + \
            rng.normal(size=(count, 3)) * 10.0 ** rng.uniform(-2.5, -0.5, (count, 1))
    side = np.linalg.norm(t[:, [0, 0, 1]] - t[:, [1, 2, 2]], axis=2).max(axis=1)
    t *= (h * (n + rng.uniform(0.02, 0.98, count)) / side)[:, None, None]
    t += rng.uniform(-1, 1, (count, 1, 3)) * h * (n + 12)
    return t


def as_mesh(t):
    v = np.ascontiguousarray(t, np.float32).reshape(-1, 3)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


def check(vol, v, f, h, band):
    o, _, _ = ob.mesh_to_volume(v, f, h, band)
    rep = compare_volumes(vol.export(), o.export())
    assert rep["leaf_set_equal"] and rep["mask_mismatch_leaves"] == 0 and rep["value_mismatch"] == 0, rep
    assert rep["active"] > 0


def convert(v, f, h, band):
    return bs.MeshToVolume(context()).with_voxel_size(h).with_narrow_band_width(band).convert((v, f))


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8, 33])
@pytest.mark.parametrize("slender", [False, True])
def test_cut_triangles_match_oracle(n, slender):
    h, band = np.float32(0.01), 5
    t = cut_soup(n, float(h), 24 if n < 30 else 4, n + 100 * slender, slender)
    v, f = as_mesh(t)
    vol = convert(v, f, h, band)
    st = context().last_stats()
    assert st["subtris"] == n * n * len(f)
    # the rule's estimate must select the patches for this input
    area = 0.5 * np.linalg.norm(np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]), axis=1).sum() / float(h) ** 2
    assert 0.61 * (2 * band + 3.3) ** 2 * st["subtris"] / area > 140
    check(vol, v, f, h, band)


def test_degenerate_among_cut_triangles():
    h, band = np.float32(0.01), 5
    t = cut_soup(3, float(h), 30, 7, False)
    t[5:8, 2] = t[5:8, 1]                                     # zero area
    t[8:10] = t[8:10, :1]                                     # points
    t[10:14, 2] = 0.5 * (t[10:14, 0] + t[10:14, 1]) + 1e-9    # collinear up to rounding
    v, f = as_mesh(t + 5.0)
    check(convert(v, f, h, band), v, f, h, band)


def test_torus_and_batch():
    """The benchmark's slender torus cells at band 4, alone and beside an icosphere cut finely."""
    a = synthetic.torus(1.0, 0.3, 96, 48, 0.02, seed=2)
    b = synthetic.icosphere(2, 0.8, 0.03, seed=3)
    check(convert(*a, 0.01, 4), *a, 0.01, 4)
    for vol, m, h in zip(bs.convert_batch([a, b], [(0.012, 5), (0.015, 5)], ctx=context()), (a, b), (0.012, 0.015)):
        check(vol, *m, np.float32(h), 5)
