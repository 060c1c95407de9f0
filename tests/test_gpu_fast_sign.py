"""The certified filter of the sign pass on the library's own tree
(csrc/fast_sign.cu) against the traversal that it stands for: WindingNumbers on
the same tree sums one cut per 32 consecutive points, so points given in the
order of the pass's voxels (bricks in turn, Morton order inside) have the
pass's cuts.  Every sign must be the one that traversal's float32 sum gives.
Equality, no tolerance: the filter settles a warp's voxels or hands them over."""
import ctypes as C

import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import _native as N
from tests.gpu_common import context, unpack_mask
from tests.test_gpu_sign_filter import shapes

pytestmark = pytest.mark.gpu

M = np.arange(512)
MORTON = ((((M >> 2) & 1) | ((M >> 4) & 2) | ((M >> 6) & 4)) << 6 | (((M >> 1) & 1) | ((M >> 3) & 2) | ((M >> 5) & 4)) << 3
          | (M & 1) | ((M >> 2) & 2) | ((M >> 4) & 4))


def convert(meshes, params, beta, thresh):
    """One call for all meshes (fast tree, order 2)."""
    ctx, K = context(), len(meshes)
    P, out = (N.M2VParams * K)(), (C.c_void_p * K)()
    for p, (h, band) in zip(P, params):
        N.load().bs_m2v_params_default(C.byref(p))
        p.voxel_size, p.band_width, p.wn_beta, p.wn_threshold, p.wn_tree = h, band, beta, thresh, 1
    xyz = np.concatenate([np.asarray(v, np.float32) for v, _ in meshes])
    tri = np.concatenate([np.asarray(f, np.uint32) for _, f in meshes])
    nv = np.array([len(v) for v, _ in meshes], np.uint64)
    nt = np.array([len(f) for _, f in meshes], np.uint64)
    N.check(N.load().bs_mesh_to_volume_batch(ctx.h, K, xyz.ctypes.data, nv.ctypes.data, tri.ctypes.data,
                                             nt.ctypes.data, P, out), ctx.h)
    return [bs.Volume(C.c_void_p(o), ctx) for o in out]


def check(vol, v, f, h, beta, thresh):
    o, val, m = vol.export()
    act = np.stack([unpack_mask(x) for x in m])[:, MORTON]
    li, k = np.nonzero(act)
    vi = MORTON[k]
    vox = o[li] + np.stack([vi >> 6, (vi >> 3) & 7, vi & 7], 1)
    pts = vox.astype(np.float32) * np.float32(h)
    wn = bs.WindingNumbers.from_mesh((v, f), ctx=context(), tree="fast")
    step = 1 << 19  # larger sets are reordered
    w = np.concatenate([wn.approximate(pts[i:i + step], beta) for i in range(0, len(pts), step)])
    assert len(pts) > 0
    assert np.array_equal(np.signbit(val[li, vi]), ~(w < np.float32(thresh)))


@pytest.mark.parametrize("name", sorted(shapes()))
@pytest.mark.parametrize("beta,thresh", [(2.0, 0.2), (1.0, 0.5), (3.5, 0.05)])
def test_signs_equal_the_traversal(name, beta, thresh):
    v, f, h, band = shapes()[name]
    check(convert([(v, f)], [(h, band)], beta, thresh)[0], v, f, h, beta, thresh)


def test_threshold_through_the_field():
    """Thresholds in the middle of an open sheet's smooth field: warps stay
    unsettled in both attempts."""
    v = np.array([[-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]], np.float32)
    f = np.array([[0, 1, 2], [0, 2, 3]], np.uint32)
    for thresh in (0.25, 0.37, -0.4, 0.5):
        check(convert([(v, f)], [(0.02, 12)], 2.0, thresh)[0], v, f, 0.02, 2.0, thresh)


def test_batch_of_all_shapes():
    s = [x for k, x in sorted(shapes().items()) if k not in ("out_of_range", "tiny")]
    vols = convert([(v, f) for v, f, _, _ in s], [(h, b) for _, _, h, b in s], 2.0, 0.2)
    for vol, (v, f, h, _) in zip(vols, s):
        check(vol, v, f, h, 2.0, 0.2)
