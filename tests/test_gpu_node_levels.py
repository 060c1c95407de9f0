"""The internal levels of a volume (csrc/volume_ops.cu: a directory over the
nodes' bounding box, or sorting where the box has too many cells) and their
flood fill, against the oracle through booleans, bit for bit with tiles: one
leaf, one node, a dozen top-level nodes along each axis (gaps between them
filled along z), and a volume so wide that the box has more cells than the
directory takes."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from oracle import binding as ob
from tests.gpu_common import context
from tests.test_gpu_csg import assert_same

pytestmark = pytest.mark.gpu


def boxes(at, half):
    """Closed boxes around the given centres."""
    v, f = [], []
    for c in at:
        p = np.array([[x, y, z] for x in (-half, half) for y in (-half, half) for z in (-half, half)]) + c
        q = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
        f += [[len(v) + i for i in t] for a, b, c, d in q for t in ((a, b, c), (a, c, d))]
        v += list(p)
    return np.array(v, np.float32), np.array(f, np.uint32)


def places():
    rng = np.random.default_rng(3)
    out = {"leaf": np.array([[4.3, 4.2, 4.1]]), "node": rng.uniform(20, 100, (3, 3)),
           "corner": np.array([[0.3, -0.2, 0.1], [4096.2, 4095.7, 4096.4]])}
    for k, ax in enumerate("xyz"):
        p = rng.uniform(-30, 30, (12, 3))
        p[:, k] = 5200.0 * np.arange(12) - 20000
        out["line_" + ax] = p
    p = rng.uniform(0, 260, (40, 3))
    p[:, 0] = np.linspace(-600e3, 600e3, 40)
    p[0, 1:], p[1, 1:] = 0, 260  # 9375 x 3 x 3 nodes
    out["wide"] = p
    return out


def convert(v, f):
    g = bs.MeshToVolume(context()).with_voxel_size(1.0).with_narrow_band_width(1).convert((v, f))
    return g, ob.mesh_to_volume(v, f, 1.0, 1)[0]


@pytest.mark.parametrize("name", sorted(places()))
@pytest.mark.parametrize("op", ["union", "subtract", "intersect"])
def test_levels_match_oracle(name, op):
    at = places()[name]
    ga, oa = convert(*boxes(at, 3.4 if name == "leaf" else 12.4))
    gb, ob_ = convert(*boxes(at[::2] + np.array([2.2, 1.1, -1.6]), 3.4 if name == "leaf" else 11.3))
    g, o = getattr(ga, op)(gb), getattr(oa, op)(ob_)
    assert_same(g, o)
