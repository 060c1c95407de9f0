"""How much a conversion's sign filter leaves to the traversal
(bs_ctx_last_counters [15]; voxels on the reference's tree, warps of 32 on the
library's): nothing on a closed surface, some on
a heap of random triangles and where the threshold is the outside's value,
everything out of the filter's range.  The signs
at these inputs are compared in test_gpu_sign_filter.py, test_gpu_fast_sign.py
and test_gpu_sign_counters.py; here that the fallbacks are what gives them."""
import numpy as np
import pytest

from tests.gpu_common import context
from tests.test_gpu_fast_sign import convert as convert_fast
from tests.test_gpu_sign_filter import convert as convert_reference
from tests.test_gpu_sign_filter import shapes, soup

pytestmark = pytest.mark.gpu

def left(tree, v, f, h, band, thresh):
    """Voxels or warps left, and of how many."""
    if tree == "fast":
        convert_fast([(v, f)], [(h, band)], 2.0, thresh)
    else:
        convert_reference(v, f, h, band, 2.0, thresh)
    st = context().last_stats()
    assert st["wn_tree"] == tree
    return st["wn_left_to_traversal"], st["active_voxels"] if tree == "reference" else -(-st["active_voxels"] // 32)


@pytest.mark.parametrize("tree", ["reference", "fast"])
def test_what_is_left(tree):
    v, f, h, band = shapes()["torus"]
    assert left(tree, v, f, h, band, 0.2)[0] == 0
    rng = np.random.default_rng(0)
    heap = soup(rng.normal(size=(20000, 1, 3)) * 0.3 + rng.normal(size=(20000, 3, 3)) * 0.02)
    for n, of in (left(tree, v, f, h, band, 0.0), left(tree, *heap, 0.03, 2, 0.2)):
        assert 0 < n < of
    n, of = left(tree, *shapes()["out_of_range"], 0.2)
    assert n == of > 0
