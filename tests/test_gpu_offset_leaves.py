"""The offset's leaf sweeps evaluate only the voxels that can change, found on
masks in the sweep's order (csrc/offset.cu): a few triangles in every
orientation put them anywhere in the leaves, at faces, edges and corners, for
all eight directions; thin bands leave most voxels free and wide ones whole
leaves frozen; offsets of less than a voxel to several leaves change nothing,
little or all.  Bit for bit the oracle."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from oracle import binding as ob
from tests.gpu_common import context
from tests.test_gpu_offset import assert_same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 9])
@pytest.mark.parametrize("band", [0, 2, 6])
@pytest.mark.parametrize("d", [0.01, -0.01, 0.13, -0.13, 1.3, -1.3])
def test_triangles_match_oracle(n, band, d):
    h = 0.1
    rng = np.random.default_rng(1000 * n + 10 * band)
    v = (rng.uniform(-1.5, 1.5, (n, 1, 3)) + rng.normal(size=(n, 3, 3)) * 0.8).astype(np.float32).reshape(-1, 3)
    f = np.arange(len(v), dtype=np.uint32).reshape(-1, 3)
    g = bs.MeshToVolume(context()).with_voxel_size(h).with_narrow_band_width(band).convert((v, f))
    o, _, _ = ob.mesh_to_volume(v, f, h, band)
    g.offset(d)
    o.offset(d)
    assert_same(g, o)
