"""The passes over large nodes of the reference's tree build go by chunks of
2048 positions from 4 M triangles on (csrc/ref_tree.cu), 512 below.  Meshes of
one batch are built together, so a batch of more than 4 M triangles builds each
mesh's tree with the larger chunks: the work of the signs' traversal, which
depends on every node, and the volumes equal those of the meshes alone."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import synthetic
from tests.gpu_common import context

pytestmark = pytest.mark.gpu


def test_large_chunks_build_the_same_trees():
    sphere = synthetic.icosphere(8, 1.0, 0.02, seed=1)  # 1.3 M triangles
    meshes = [sphere, (sphere[0], synthetic.remove_faces(sphere[1], 0.2, seed=2)),
              synthetic.torus(1.0, 0.3, 1024, 512, 0.02, seed=3), synthetic.torus(1.0, 0.3, 800, 601, 0.02, seed=4)]
    assert all(len(f) < 1 << 22 for _, f in meshes) and sum(len(f) for _, f in meshes) > 1 << 22
    one = bs.MeshToVolume(context()).with_voxel_size(0.05).with_narrow_band_width(1)
    alone, work = [], {"wn_far": 0, "wn_exact": 0}
    for m in meshes:
        alone.append(one.convert(m).export())
        for k in work:
            work[k] += context().last_stats()[k]
    vols = bs.convert_batch(meshes, [(0.05, 1)] * len(meshes), ctx=context())
    assert {k: context().last_stats()[k] for k in work} == work
    for vol, (o, v, m) in zip(vols, alone):
        a, b, c = vol.export()
        assert np.array_equal(a, o) and np.array_equal(c, m) and np.array_equal(b.view(np.uint32), v.view(np.uint32))
