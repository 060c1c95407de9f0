"""A batch on the library's tree with meshes of both far-field orders
(csrc/m2v.cu k_wn_sign_batch): each mesh takes its own order's traversal, so
its volume is the one that it has alone (order 2 alone goes through the
certified filter, which gives the traversal's signs)."""
import ctypes as C

import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import _native as N
from baby_shark_gb300 import synthetic
from tests.gpu_common import context

pytestmark = pytest.mark.gpu


def convert(meshes, orders, h, band):
    ctx, K = context(), len(meshes)
    P, out = (N.M2VParams * K)(), (C.c_void_p * K)()
    for p, order in zip(P, orders):
        N.load().bs_m2v_params_default(C.byref(p))
        p.voxel_size, p.band_width, p.wn_order, p.wn_tree = h, band, order, 1
    xyz = np.concatenate([np.asarray(v, np.float32) for v, _ in meshes])
    tri = np.concatenate([np.asarray(f, np.uint32) for _, f in meshes])
    nv = np.array([len(v) for v, _ in meshes], np.uint64)
    nt = np.array([len(f) for _, f in meshes], np.uint64)
    N.check(N.load().bs_mesh_to_volume_batch(ctx.h, K, xyz.ctypes.data, nv.ctypes.data, tri.ctypes.data,
                                             nt.ctypes.data, P, out), ctx.h)
    return [bs.Volume(C.c_void_p(o), ctx) for o in out]


@pytest.mark.parametrize("orders", [(2, 3, 2), (3, 3, 2), (3, 2, 3)])
def test_each_mesh_takes_its_order(orders):
    v, f = synthetic.icosphere(4, 1.0, 0.05, seed=1)
    meshes = [(v, synthetic.remove_faces(f, 0.3, seed=2)), synthetic.torus(1.0, 0.3, 96, 48, 0.02, seed=3),
              (v, synthetic.remove_faces(f, 0.5, seed=4))]
    for vol, m, order in zip(convert(meshes, orders, 0.03, 2), meshes, orders):
        for a, b in zip(vol.export(), convert([m], [order], 0.03, 2)[0].export()):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
