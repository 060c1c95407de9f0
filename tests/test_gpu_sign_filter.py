"""The sign pass's certified filter (csrc/sign_filter.cu) against the exact
traversal of the same tree (WindingNumbers on the reference's tree, one
traversal per point, csrc/ref_tree.cu): at every band voxel the sign must be
the one the traversal's float32 winding number gives, whatever the mesh, the
scale, the accuracy scale and the threshold.  Equality, no tolerance: the
filter's bound either settles a voxel or hands it to that traversal."""
import ctypes as C

import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import _native as N
from baby_shark_gb300 import synthetic
from tests.gpu_common import context, unpack_mask


def soup(tri):
    v = np.ascontiguousarray(tri, np.float32).reshape(-1, 3)
    return v, np.arange(len(v), dtype=np.uint32).reshape(-1, 3)


def cube(lo, hi):
    v = np.array([[x, y, z] for x in (lo, hi) for y in (lo, hi) for z in (lo, hi)], np.float32)
    q = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    return v, np.array([t for a, b, c, d in q for t in ((a, b, c), (a, c, d))], np.uint32)


def shapes():
    rng = np.random.default_rng(4)
    v, f = synthetic.icosphere(4, 1.0, 0.05, seed=1)
    holed = (v, synthetic.remove_faces(f, 0.3, seed=2))
    hedge = synthetic.icosphere(3, 1.0, 0.4, seed=3)
    few = [soup(rng.uniform(-1, 1, (n, 3, 3))) for n in (1, 2, 4, 7)]
    needles = rng.uniform(-1, 1, (300, 1, 3)) + rng.normal(size=(300, 3, 3)) * np.array([0.4, 0.01, 0.001])
    flat = np.concatenate([needles[:50], np.repeat(needles[50:100, :1], 3, axis=1),  # points
                           np.repeat(needles[100:101], 40, axis=0)])                 # coincident copies
    return {"noisy": (v, f, 0.03, 3), "holes": (*holed, 0.03, 3), "hedgehog": (*hedge, 0.04, 2),
            "torus": (*synthetic.torus(1.0, 0.3, 200, 100, 0.02, seed=3), 0.02, 3),
            "on_grid": (*cube(-1.0, 1.0), 0.125, 2),   # faces through grid points: solid angles at their branch cut
            "fine": (*cube(-0.3, 0.4), 0.01, 3),        # triangles of tens of voxels
            "needles": (*soup(needles), 0.05, 2), "degenerate": (*soup(flat), 0.05, 2),
            "coarse": (v, f, 0.4, 1),                    # many triangles in every voxel
            "far_away": (v + np.float32(3000.0), f, 0.05, 2),
            "out_of_range": (v * np.float32(3e6), f, 1e5, 2), "tiny": (v * np.float32(1e-7), f, 4e-9, 2),
            **{"few%d" % k: (*m, 0.1, 3) for k, m in enumerate(few)}}


def convert(v, f, h, band, beta, thresh):
    ctx, P, out = context(), N.M2VParams(), C.c_void_p()
    N.load().bs_m2v_params_default(C.byref(P))
    P.voxel_size, P.band_width, P.wn_beta, P.wn_threshold = h, band, beta, thresh
    v, f = np.ascontiguousarray(v, np.float32), np.ascontiguousarray(f, np.uint32)
    N.check(N.load().bs_mesh_to_volume(ctx.h, v.ctypes.data, len(v), f.ctypes.data, len(f), C.byref(P), C.byref(out)),
            ctx.h)
    return bs.Volume(out, ctx)


def check(vol, v, f, h, beta, thresh):
    o, val, m = vol.export()
    act = np.stack([unpack_mask(x) for x in m])
    li, vi = np.nonzero(act)
    vox = o[li] + np.stack([vi >> 6, (vi >> 3) & 7, vi & 7], 1)
    pts = vox.astype(np.float32) * np.float32(h)
    wn = bs.WindingNumbers.from_mesh((v, f), ctx=context(), tree="reference").approximate(pts, beta)
    assert len(pts) > 0
    assert np.array_equal(np.signbit(val[li, vi]), ~(wn < np.float32(thresh)))


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(shapes()))
@pytest.mark.parametrize("beta,thresh", [(2.0, 0.2), (1.0, 0.5), (3.5, 0.05)])
def test_signs_equal_the_exact_traversal(name, beta, thresh):
    v, f, h, band = shapes()[name]
    check(convert(v, f, h, band, beta, thresh), v, f, h, beta, thresh)


@pytest.mark.gpu
def test_threshold_through_the_field():
    """A threshold in the middle of an open sheet's smooth field: the filter
    leaves a shell of voxels undecided, in both of its attempts."""
    v = np.array([[-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]], np.float32)
    f = np.array([[0, 1, 2], [0, 2, 3]], np.uint32)
    for thresh in (0.25, 0.37, -0.4, 0.5):
        check(convert(v, f, 0.02, 12, 2.0, thresh), v, f, 0.02, 2.0, thresh)


@pytest.mark.gpu
def test_batch_of_all_shapes():
    """One call over every shape: undecided voxels of several meshes at once."""
    s = [x for k, x in shapes().items() if k not in ("out_of_range", "tiny")]
    vols = bs.convert_batch([(v, f) for v, f, _, _ in s], [(h, b) for _, _, h, b in s], ctx=context())
    for vol, (v, f, h, _) in zip(vols, s):
        check(vol, v, f, h, 2.0, 0.2)


def test_expansion_bound():
    """The polynomial of a node (dipole to degree 2, quadrupole to degree 1)
    stays within the truncation bound of the kernel, in float64, for random
    nodes and points up to the largest expansion ratio."""
    rng = np.random.default_rng(0)
    n = 100000
    a, B = rng.normal(size=(n, 3)), rng.normal(size=(n, 3, 3)) * 10.0 ** rng.uniform(-3, 1, (n, 1, 1))
    s, d = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
    s /= np.linalg.norm(s, axis=1, keepdims=True)
    x = rng.uniform(0.01, 0.5, n)
    d *= (x / np.linalg.norm(d, axis=1))[:, None]
    d[: n // 4] = s[: n // 4] * x[: n // 4, None]  # straight at the node, where the terms align
    r = s - d
    R = np.linalg.norm(r, axis=1)
    dot = lambda u, w: (u * w).sum(1)  # noqa: E731
    rBr, tr = np.einsum("ni,nij,nj->n", r, B, r), np.trace(B, axis1=1, axis2=2)
    field = dot(a, r) / R ** 3 + tr / R ** 3 - 3 * rBr / R ** 5
    S = (B + B.transpose(0, 2, 1)) / 2 - tr[:, None, None] / 3 * np.eye(3)
    Ss = np.einsum("nij,nj->ni", S, s)
    an, sSs, sd, ad, dd = dot(a, s), dot(s, Ss), dot(s, d), dot(a, d), dot(d, d)
    poly = an + 3 * sd * an - ad + (15 * sd * sd * an - 3 * an * dd - 6 * sd * ad) / 2
    poly += -3 * sSs - 15 * sd * sSs + 6 * dot(Ss, d)
    na, nb = np.linalg.norm(a, axis=1), np.sqrt((B * B).sum((1, 2)))
    bound = x ** 2 / (1 - x) ** 2 * (4 * na * x + 4.16 * 5 * nb / (1 - x))
    assert np.all(np.abs(poly - field) <= bound)
    assert (np.abs(poly - field) / bound).max() > 0.3  # the bound is not slack by construction
