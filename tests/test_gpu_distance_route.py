"""Which distance pass a conversion takes (csrc/m2v.cu: on patches of
sub-triangles where a band voxel meets many of their boxes and they can be
culled, else on sub-triangles; the timed stages carry the kernels' names)."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import synthetic
from oracle import binding as ob
from tests.gpu_common import compare_volumes, context

pytestmark = pytest.mark.gpu


def needles(n, aspect, seed):
    """Random triangles about 0.4 long and `aspect` of that high."""
    rng = np.random.default_rng(seed)
    t = rng.uniform(-0.5, 0.5, (n, 1, 3)) + 0.2 * rng.normal(size=(n, 3, 3))
    x = t[:, 1] - t[:, 0]
    up = np.cross(x, rng.normal(size=(n, 3)))
    up *= (aspect * np.linalg.norm(x, axis=1) / np.linalg.norm(up, axis=1))[:, None]
    t[:, 2] = t[:, 0] + x * rng.uniform(0.2, 0.8, (n, 1)) + up
    v = t.astype(np.float32).reshape(-1, 3)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


def convert(mesh, h, band, ctx=None):
    """The volume, and whether the pass on patches made it."""
    ctx = ctx or context()
    ctx.set_stage_timing(True)
    try:
        ctx.stage_times(reset=True)
        vol = bs.MeshToVolume(ctx).with_voxel_size(h).with_narrow_band_width(band).convert(mesh)
        st = ctx.stage_times(reset=True)
        took = "k_patches" in st
        for sub, patch in (("k_brick_distance", "k_patch_distance"), ("k_count_pairs", "k_count_patches"),
                           ("k_fill_pairs", "k_fill_patches")):
            assert (patch in st) == took and (sub in st) != took
        return vol, took
    finally:
        ctx.set_stage_timing(False)


def assert_same(vol, mesh, h, band):
    o, _, _ = ob.mesh_to_volume(*mesh, h, band)
    rep = compare_volumes(vol.export(), o.export())
    assert rep["leaf_set_equal"] and rep["mask_mismatch_leaves"] == 0 and rep["value_mismatch"] == 0, rep
    assert rep["active"] > 0


@pytest.mark.parametrize("aspect,patches", [(0.7, True), (0.003, False)])
def test_slender_triangles_keep_the_pass_on_sub_triangles(aspect, patches):
    """Equally many boxes per voxel; the slender triangles' sub-triangles are never culled."""
    mesh, h, band = needles(100, aspect, 1), 0.02, 4
    vol, took = convert(mesh, h, band)
    assert took == patches
    st = context().last_stats()
    assert (st["voxel_pairs_evaluated"] < st["voxel_pairs"]) == patches
    assert_same(vol, mesh, h, band)


@pytest.mark.parametrize("tile", [8, 32])
def test_autotune_keeps_the_tile_on_patches(tile):
    """The pass on patches has no tile: what the context has must stay, and no
    more than the three shapes be timed."""
    ctx = bs.Context(0)
    mesh = synthetic.torus(1.0, 0.3, 96, 48, 0.02, seed=5)
    ctx.set_launch_shape(128, 4, tile)
    assert convert(mesh, 0.02, 4, ctx)[1]
    choice = ctx.autotune(mesh, 0.02, 4)
    t = choice["distance_ms"]
    assert choice["dist_tile"] == (min(tile, 16) if choice["dist_threads"] == 256 else tile)
    assert t[64, 8] == t[64, 16] == t[64, 32] > 0 and t[128, 8] == t[128, 16] == t[128, 32] > 0
    assert t[256, 8] == t[256, 16] > 0
    assert t[choice["dist_threads"], 16] == min(t.values())
    assert all(ms > 0 for ms in choice["sign_ms"].values())


@pytest.mark.parametrize("band,patches", [(1, False), (4, True)])
def test_every_launch_shape_of_both_passes_matches_oracle(band, patches):
    ctx = bs.Context(0)
    mesh, h = synthetic.torus(1.0, 0.3, 96, 48, 0.02, seed=5), 0.02
    o, _, _ = ob.mesh_to_volume(*mesh, h, band)
    o = o.export()
    for threads, tile in ((64, 8), (64, 16), (64, 32), (128, 8), (128, 16), (128, 32), (256, 8), (256, 16)):
        ctx.set_launch_shape(threads, 0, tile)
        vol, took = convert(mesh, h, band, ctx)
        assert took == patches
        rep = compare_volumes(vol.export(), o, check_inactive=True)
        assert rep["leaf_set_equal"] and rep["mask_mismatch_leaves"] == rep["value_mismatch"] == 0, rep
        assert rep["sign_mismatch"] == rep["inactive_mismatch"] == 0 and rep["active"] > 0, rep


def of_every_split():
    """Meshes whose patches' lists are filled by 32, 16, ... 1 threads per patch, with voxel size and band."""
    return {"80": (synthetic.icosphere(1, 1.0, 0.0, seed=1), 0.1625, 5),
            "1280": (synthetic.icosphere(3, 1.0, 0.0, seed=1), 0.03, 4),
            "5120": (synthetic.icosphere(4, 1.0, 0.005, seed=1), 0.015, 4),
            "9216": (synthetic.torus(1.0, 0.3, 96, 48, 0.02, seed=5), 0.02, 4),
            "65536": (synthetic.torus(1.0, 0.3, 256, 128, 0.02, seed=5), 0.0075, 4)}


@pytest.mark.parametrize("name", ["80", "1280", "5120", "9216", "65536"])
def test_lists_of_patches_are_complete_at_every_split(name):
    mesh, h, band = of_every_split()[name]
    vol, took = convert(mesh, h, band)
    assert took
    assert_same(vol, mesh, h, band)


def test_lists_of_few_large_patches_cost_less_than_the_pass():
    """80 triangles, dozens of bricks each: filling the lists must leave most of
    the time to the distances."""
    mesh, h, band = of_every_split()["80"]
    ctx = context()
    best = {}
    ctx.set_stage_timing(True)
    try:
        for _ in range(6):
            ctx.stage_times(reset=True)
            bs.MeshToVolume(ctx).with_voxel_size(h).with_narrow_band_width(band).convert(mesh)
            for k, (ms, _) in ctx.stage_times(reset=True).items():
                best[k] = min(best.get(k, 1e9), ms)
    finally:
        ctx.set_stage_timing(False)
    lists = best["k_count_patches"] + best["k_fill_patches"]
    print("lists %.3f ms, distances %.3f ms" % (lists, best["k_patch_distance"]))
    assert lists <= 0.75 * best["k_patch_distance"]
