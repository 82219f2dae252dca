"""The pair sort at the sizes where it can go wrong: one thread block's share and one past it, tiles of
pairs that are full, short by one and over by one, and odd and even numbers of passes. Sparse cells come
sorted by their first triangle, so with a triangle a cell their order is known."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 31, 33, 1023, 1025, 8191, 8192, 8193, 10239, 10241, 65537, 300001])
def test_cells_sorted_by_triangle(ctx, n):
    res = 128
    cell = np.random.default_rng(n).permutation(res ** 3)[:n]
    xyz = np.stack([cell % res, (cell // res) % res, cell // (res * res)], 1).astype(np.int32)
    corner = np.array([[-0.25, -0.25, 0.0], [0.25, 0.0, 0.125], [0.0, 0.25, -0.125]])
    soup = ((xyz[:, None, :] + 0.5 + corner[None]) / res).astype(np.float32)
    cells, org, vox = ctx.voxelize_sparse(soup.reshape(-1, 3), (0, 0, 0), (1, 1, 1), res)
    assert tuple(org) == (0.0, 0.0, 0.0) and vox == 1.0 / res
    assert np.array_equal(np.asarray(cells).reshape(-1, 3), xyz)
