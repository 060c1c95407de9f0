"""The passes of dual contouring that compute values (csrc/dc.cu) give a leaf
more warps the fewer leaves there are.  A crowded block (almost every edge
crosses, most of 512 cells to a leaf) must have the same vertices, bit for bit,
alone and as a part of volumes on both sides of every change of that number;
and a few crowded leaves must not take longer than several times as many cells
spread over many leaves."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import synthetic
from tests.gpu_common import context
from tests.test_gpu_dual_contouring_masks import multiset

pytestmark = pytest.mark.gpu


def mesher(qef):
    m = bs.DualContouringMesher().with_voxel_size(0.5)
    return m.with_qef_vertices() if qef else m


def grid(vals):
    top = (np.asarray(vals.shape) - 1).astype(np.float32) * np.float32(0.5)
    return bs.Volume.from_fn(0.5, np.zeros(3, np.float32), top, 3, lambda p: vals.ravel(), ctx=context())


@pytest.mark.parametrize("qef", [False, True])
def test_same_vertices_in_volumes_of_every_size(qef):
    rows = (152, 153, 305, 609, 1217, 2433)  # 4 leaves each: around 4, 8, ... 64 per SM
    z = np.arange(8 * (rows[-1] + 2))
    xy = np.sin(0.9 * np.arange(16))
    vals = (xy[:, None, None] + xy[None, :, None] + 1.3 * np.sin(0.4 * z)).astype(np.float32)
    vals[:, :, :24] = np.random.default_rng(5).uniform(-1.4, 1.4, (16, 16, 24))
    vals[:, :, 24:40] = 9.0  # two rows of leaves that do not exist
    want = multiset(mesher(qef).mesh(grid(vals[:, :, :24])))
    assert len(want) > 6000
    for r in rows:
        got = mesher(qef).mesh(grid(vals[:, :, :8 * (r + 2)]))
        assert context().last_stats()["crossings"] > 3 * 64 * r
        block = got[got.reshape(-1, 9)[:, 2::3].max(axis=1) < 16.0].reshape(-1, 9)
        assert np.array_equal(multiset(block), want)


@pytest.mark.parametrize("qef", [False, True])
def test_few_crowded_leaves_do_not_wait_for_one_warp(qef):
    ctx, name = context(), "k_dc_cell_qef" if qef else "k_dc_cell_points"

    def cell_ms(vol):
        best = 1e9
        ctx.set_stage_timing(True)
        try:
            for _ in range(4):
                ctx.stage_times(reset=True)
                mesher(qef).mesh(vol.clone())  # a volume keeps its mesh
                best = min(best, ctx.stage_times(reset=True)[name][0])
        finally:
            ctx.set_stage_timing(False)
        return best, ctx.last_stats()["cells"]

    crowded, few = cell_ms(grid(np.random.default_rng(1).uniform(-1.4, 1.4, (16, 16, 16)).astype(np.float32)))
    v, f = synthetic.torus(30.0, 9.0, 200, 100, 0.6, seed=1)
    spread, many = cell_ms(bs.MeshToVolume(ctx).with_voxel_size(0.5).with_narrow_band_width(2).convert((v, f)))
    print("%s: %d cells on 8 leaves %.3f ms, %d cells spread %.3f ms" % (name, few, crowded, many, spread))
    assert 2500 < few and 4 * few < many
    assert crowded <= spread
