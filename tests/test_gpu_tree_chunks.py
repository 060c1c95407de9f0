"""The passes over large nodes of the reference's tree build go by chunks of
512 positions that the device lists itself (csrc/ref_tree.cu): node sizes
around whole chunks, one short last chunk, and several levels of them.  The
same work as the oracle's tree (see tests/test_gpu_reference_tree.py)."""
import numpy as np
import pytest

from tests.test_gpu_reference_tree import check_against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 513, 1023, 1024, 1025, 1537, 4097, 9000])
def test_chunk_edges_match_oracle(n):
    rng = np.random.default_rng(n)
    v = (rng.uniform(-1, 1, (n, 1, 3)) + 0.05 * rng.normal(size=(n, 3, 3))).astype(np.float32).reshape(-1, 3)
    f = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    check_against_oracle(v, f, rng.uniform(-1.3, 1.3, (4000, 3)).astype(np.float32))
