"""The work counters of a conversion's sign pass (bs_ctx_last_counters [10],
[11], and on the library's tree [6]) count every voxel's cut once, whoever
walks it: the certified filter, or the traversal where the filter has no room
for the cut or is not used.  They equal the counters of WindingNumbers on the
same tree at the same points (on the library's tree in the pass's order, 32
points per cut), and so do the signs."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from baby_shark_gb300 import synthetic
from tests.gpu_common import context, unpack_mask
from tests.test_gpu_fast_sign import MORTON
from tests.test_gpu_fast_sign import convert as convert_fast
from tests.test_gpu_sign_filter import convert as convert_reference
from tests.test_gpu_sign_filter import shapes, soup

pytestmark = pytest.mark.gpu
KEYS = {"fast": ("wn_warp_visits", "wn_far", "wn_exact"), "reference": ("wn_far", "wn_exact")}


def cases():
    s = shapes()
    out = {k: (*s[k], 2.0, 0.2) for k in ("torus", "on_grid", "degenerate", "tiny", "out_of_range", "coarse", "few2")}
    # every node near: the pending nodes of 32 voxels outgrow the filter's stacks
    out["all_near"] = (*synthetic.torus(1.0, 0.3, 400, 200, 0.02, seed=3), 0.2, 1, 500.0, 0.2)
    # random triangles: values on either side of the threshold and close to it
    rng = np.random.default_rng(0)
    out["heap"] = (*soup(rng.normal(size=(20000, 1, 3)) * 0.3 + rng.normal(size=(20000, 3, 3)) * 0.02), 0.03, 2, 2.0, 0.2)
    # a threshold at the outside's value: half of the groups cannot be settled,
    # and after the first ones the filter gives the mesh up
    out["outside_value"] = (*synthetic.torus(1.0, 0.3, 256, 128, 0.02, seed=3), 0.006, 3, 2.0, 0.0)
    return out


@pytest.mark.parametrize("tree", ["reference", "fast"])
@pytest.mark.parametrize("name", sorted(cases()))
def test_counters_equal_the_traversal(name, tree):
    v, f, h, band, beta, thresh = cases()[name]
    vol = convert_fast([(v, f)], [(h, band)], beta, thresh)[0] if tree == "fast" else \
        convert_reference(v, f, h, band, beta, thresh)
    st = context().last_stats()
    o, val, m = vol.export()
    li, k = np.nonzero(np.stack([unpack_mask(x) for x in m])[:, MORTON])
    vi = MORTON[k]
    pts = (o[li] + np.stack([vi >> 6, (vi >> 3) & 7, vi & 7], 1)).astype(np.float32) * np.float32(h)
    wn = bs.WindingNumbers.from_mesh((v, f), ctx=context(), tree=tree)
    want, w = dict.fromkeys(KEYS[tree], 0), []
    for i in range(0, len(pts), 1 << 19):  # larger sets are reordered
        w.append(wn.approximate(pts[i:i + (1 << 19)], beta))
        got = context().last_stats()
        for key in want:
            want[key] += got[key]
    assert len(pts) > 0 and want["wn_far"] + want["wn_exact"] > 0
    assert {key: st[key] for key in want} == want
    assert np.array_equal(np.signbit(val[li, vi]), ~(np.concatenate(w) < np.float32(thresh)))
