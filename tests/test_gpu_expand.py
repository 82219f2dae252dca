"""The expansion of triangles into candidate cells and columns where it can go wrong: triangles of no
item, of a few, of more than a thread block's share and of enough for the whole grid, and crossings
above, below and exactly at cell centres, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = np.array([[0, 2, 1], [0, 3, 2], [4, 5, 6], [4, 6, 7], [0, 1, 5], [0, 5, 4], [1, 2, 6], [1, 6, 5], [2, 3, 7],
                [2, 7, 6], [3, 0, 4], [3, 4, 7]], np.uint32)


def _scene(dims, voxel):
    """Over the grid [0, dims * voxel): a box that is wider than the grid, its faces at cell centres, a
    tilted slab, and a sphere far finer than the grid."""
    from sdfb import meshgen as mg
    ext = np.asarray(dims, np.float64) * voxel
    unit = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]], np.float64)
    lo, hi = -0.1 * ext, 1.1 * ext
    lo[2], hi[2] = (dims[2] // 4 + 0.5) * voxel, (dims[2] // 2 + 0.5) * voxel
    box = lo + unit * (hi - lo)
    slab = ext * (0.07 + 0.83 * unit)
    slab[:, 2] = ext[2] * (0.55 + 0.1 * unit[:, 2] + 0.2 * unit[:, 0] + 0.1 * unit[:, 1])
    v, f = mg.icosphere(4)
    ball = (v * 0.3 * ext.min() + ext * (0.45, 0.55, 0.4), f)
    v, f = mg.concat([(box, BOX), ball, (slab, BOX)])
    return np.asarray(v, np.float32), f


@pytest.mark.parametrize("dims", [(1, 1, 1), (5, 3, 31), (20, 17, 70), (70, 71, 33), (601, 530, 9)])
def test_candidates(ctx, oracle, dims):
    import sdfb
    voxel = 1.0 / 64  # cell centres are exact
    v, f = _scene(dims, voxel)
    g = sdfb.make_grid((0, 0, 0), voxel, dims)
    d, occ = ctx.bake(v, f, g, sdfb.make_opts(sign_mode=sdfb.SIGN_PARITY))
    assert np.array_equal(occ.reshape(-1), oracle.occupancy(v, f, (0, 0, 0), voxel, dims))
    s = oracle.sign_parity(v, f, (0, 0, 0), voxel, dims)
    away = d.reshape(-1) != 0
    assert np.array_equal((d.reshape(-1) < 0)[away], (np.asarray(s).reshape(-1) < 0)[away])


def test_candidates_of_a_batch(ctx):
    """Meshes of a batch share the passes: each grid equals its lone bake."""
    import sdfb
    dims = [(20, 17, 70), (1, 1, 1), (601, 530, 9), (70, 71, 33)]
    meshes = [_scene(n, 1.0 / 64) for n in dims]
    grids = [sdfb.make_grid((0, 0, 0), 1.0 / 64, n) for n in dims]
    modes = (sdfb.SIGN_PARITY, sdfb.SIGN_GWN)
    for mode in modes:
        opts = sdfb.make_opts(sign_mode=mode)
        dists, occs = ctx.bake_batch(meshes, grids, opts)
        for (v, f), g, d, o in zip(meshes, grids, dists, occs):
            d1, o1 = ctx.bake(v, f, g, opts)
            assert np.array_equal(d, d1) and np.array_equal(o, o1)


def test_more_grid_wide_triangles_than_listed(ctx):
    """1100 copies of a triangle of 320k candidate columns and cells (1024 are kept for the whole grid):
    the occupancy of one."""
    import sdfb
    dims, voxel = (601, 530, 9), 1.0 / 64
    tri = np.array([[-1.0, -1.0, 0.03], [12.0, -2.0, 0.08], [-2.0, 11.0, 0.11]], np.float32)
    g = sdfb.make_grid((0, 0, 0), voxel, dims)
    occ = []
    for n in (1, 1100):
        v = np.tile(tri, (n, 1))
        _, o = ctx.bake(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), g, sdfb.make_opts(), want_dist=False)
        occ.append(o)
    assert occ[0].any() and np.array_equal(*occ)


@pytest.mark.parametrize("T", [1, 12, 150, 700, 1500])
def test_few_large_triangles(ctx, oracle, T):
    """Triangles of 513 to some 100k candidate cells, each by several thread blocks, by one, or more of them than
    blocks: occupancy and parity of the oracle, and all cells tested once."""
    import sdfb
    rng = np.random.default_rng(T)
    dims, voxel = (75, 61, 66), 1.0 / 64
    v = (rng.uniform(0.1, 0.9, (T, 1, 3)) + rng.normal(0, 0.25, (T, 3, 3))).astype(np.float32).reshape(-1, 3)
    f = np.arange(3 * T, dtype=np.uint32).reshape(-1, 3)
    st = sdfb.Stats()
    d, occ = ctx.bake(v, f, sdfb.make_grid((0, 0, 0), voxel, dims), sdfb.make_opts(sign_mode=sdfb.SIGN_PARITY), stats=st)
    p = v.reshape(-1, 3, 3) * 64
    lo = np.clip(np.floor(p.min(axis=1)), 0, np.array(dims) - 1)
    hi = np.clip(np.floor(p.max(axis=1)), 0, np.array(dims) - 1)
    assert st.sat_tests == int((hi - lo + 1).prod(axis=1).sum())
    assert np.array_equal(occ.reshape(-1), oracle.occupancy(v, f, (0, 0, 0), voxel, dims))
    s = np.asarray(oracle.sign_parity(v, f, (0, 0, 0), voxel, dims)).reshape(-1)
    away = d.reshape(-1) > 1e-5 if T == 1 else np.abs(d.reshape(-1)) > 1e-5
    assert np.array_equal((d.reshape(-1) < 0)[away], (s < 0)[away])
