"""The offset of volumes that hold NaN voxels (from_fn keeps a point unless
|value| > band, volume/mod.rs:60-62, so a NaN sample becomes an active voxel):
the sweeps meet NaN among the three neighbour distances in every position of
the sort (csrc/offset.cu compute_distance).  Against the oracle: leaves, masks
and every value, NaN where it has NaN (payload and sign of a NaN that went
through an addition are the hardware's)."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from oracle import binding as ob
from tests.gpu_common import as_dict, context, unpack_mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.001, 0.02, 0.3])
@pytest.mark.parametrize("d", [0.13, -0.13, 0.4])
def test_nan_voxels_match_oracle(share, d):
    h, n = np.float32(0.1), 24
    rng = np.random.default_rng(int(1000 * share))
    x = (np.stack(np.meshgrid(*3 * [np.arange(n)], indexing="ij"), -1) - 11.4) * float(h)
    val = (np.linalg.norm(x, axis=-1) - 0.6).astype(np.float32)
    nan = rng.random(val.shape) < share
    val[nan] = np.copysign(np.float32("nan"), rng.choice([-1, 1], nan.sum()))
    o = ob.volume_from_samples(h, 1, [-12, -12, -12], val)

    def field(points):
        assert len(points) == val.size
        return val.reshape(-1)

    g = bs.Volume.from_fn(h, -12 * h * np.ones(3), 11 * h * np.ones(3), 1, field, ctx=context())
    g.offset(d)
    o.offset(d)
    a, b = as_dict(*g.export()), as_dict(*o.export())
    assert set(a) == set(b) and len(a) > 0
    for k in a:
        (v1, m1), (v2, m2) = a[k], b[k]
        assert np.array_equal(m1, m2)
        on = unpack_mask(m1)
        v1, v2 = v1[on], v2[on]
        assert np.array_equal(np.isnan(v1), np.isnan(v2))
        ok = ~np.isnan(v1)
        assert np.array_equal(v1[ok].view(np.uint32), v2[ok].view(np.uint32))
