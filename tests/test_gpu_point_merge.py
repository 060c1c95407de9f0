"""The corner table's point merge by hash table (csrc/corner_table.cu): from one
triangle to enough points to fill blocks and the table to half, all points
equal, none equal, zeros of both signs, and NaN points, which equal nothing.
Every table entry is the oracle's builder's on the reference's merge."""
import numpy as np
import pytest

import baby_shark_gb300 as bs
from tests.gpu_common import context
from tests.test_gpu_corner_table import assert_same_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("faces", [1, 10, 11, 86, 1366, 40000])
@pytest.mark.parametrize("kind", ["distinct", "clustered", "zeros"])
def test_merge_matches_oracle(faces, kind):
    rng = np.random.default_rng(faces)
    if kind == "distinct":
        soup = rng.normal(size=(faces, 3, 3))
    elif kind == "clustered":
        soup = rng.normal(size=(max(4, faces // 4), 3))[rng.integers(0, max(4, faces // 4), (faces, 3))]
    else:
        soup = rng.choice([0.0, -0.0, 1.0, -1.0, 1e-42], (faces, 3, 3))
        soup[:, :, 0] += np.arange(faces)[:, None] // 7  # keeps runs of equal edges short
    assert_same_tables(soup.astype(np.float32))


def test_all_equal_and_nan():
    same = np.full((50, 3, 3), 2.5, np.float32)
    same[:, 1, 0], same[:, 2, 1] = 3.5, 4.5
    assert_same_tables(same)
    soup = np.random.default_rng(1).normal(size=(20, 3, 3)).astype(np.float32)
    soup[:, 0] = soup[0, 0]
    soup[5:9, 0, 1] = np.nan  # each of the four is a vertex of its own
    c = bs.CornerTable.from_triangles_soup(soup, context()).counts()
    assert c["faces"] == 20
    base = assert_same_tables(np.delete(soup, range(5, 9), axis=0))
    ex = bs.CornerTable.from_triangles_soup(soup, context()).export()
    assert len(np.unique(ex["corner_vertex"][0::3][5:9])) == 4 and base["faces"] == 16
