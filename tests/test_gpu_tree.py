"""The packed tree and the distance walk at the sizes where they can go wrong: partial blocks, nodes
and levels, every block size, tile shape and the block-per-tile pass, against the FP64 oracle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# A point's coordinates in a triangle's frame carry a few roundings (2^-24 each) of its distance to
# the frame's origin, at most the diagonal; the distance adds about as many.
TOL = 16 * 2.0 ** -24


def soup(T, seed):
    """T triangles: small ones, slivers, repeated points and every hundredth as large as the box."""
    rng = np.random.default_rng(seed)
    size = np.where(np.arange(T) % 100 == 7, 1.0, 0.05)
    v = rng.uniform(-0.4, 0.4, (T, 1, 3)) + rng.normal(0.0, 0.3, (T, 3, 3)) * size[:, None, None]
    k = np.arange(T) % 10
    v[k == 3, 2] = v[k == 3, 1] + 1e-6 * rng.normal(size=((k == 3).sum(), 3))
    v[k == 5, 2] = v[k == 5, 0]
    v = np.clip(v, -0.5, 0.5).astype(np.float32).reshape(-1, 3)
    return v, np.arange(3 * T, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("T", [1, 2, 3, 63, 64, 65, 255, 257, 2047, 2049, 8193, 65537])
def test_tree_sizes(ctx, oracle, T):
    """Every block size, tile and pass gives the same bits: the walk drops a triangle only when its
    computed distance cannot be the minimum, so the order and the grouping do not matter."""
    import sdfb
    v, i = soup(T, T)
    n = (19, 13, 22)
    origin, voxel = (-0.5, -0.35, -0.55), 1.0 / 20
    g = sdfb.make_grid(origin, voxel, n)
    d64 = oracle.distance(v, i, origin, voxel, n)
    ref = None
    for leaf in (2, 4, 8):
        for tile, budget in ((1, -1), (2, 64), (3, -1), (4, 64), (5, -1), (5, 64), (6, -1)):
            d, _ = ctx.bake(v, i, g, sdfb.make_opts(sign_mode=sdfb.SIGN_NONE, leaf_size=leaf, tile=tile,
                                                    step_budget=budget, no_occupancy=True), want_occ=False)
            if ref is None:
                ref = d
                diag = np.linalg.norm(np.asarray(n) * voxel)
                assert np.abs(d.reshape(-1) - d64).max() <= TOL * diag
            assert np.array_equal(d, ref), (leaf, tile, budget)


def test_tree_batch_of_unequal_meshes(ctx):
    """Meshes of a batch own separate trees: each grid equals its lone bake, bit for bit."""
    import sdfb
    meshes = [soup(T, 50 + T) for T in (1, 700, 33, 4097)]
    grids = [sdfb.make_grid((-0.5,) * 3, 1.0 / n, (n, n + 1, n + 2)) for n in (9, 24, 16, 31)]
    opts = sdfb.make_opts(sign_mode=sdfb.SIGN_NONE)
    dists, _ = ctx.bake_batch(meshes, grids, opts)
    for (v, i), g, d in zip(meshes, grids, dists):
        assert np.array_equal(d, ctx.bake(v, i, g, opts)[0])


@pytest.mark.parametrize("leaf", [2, 8])
def test_block_pass_with_more_nodes_than_it_keeps(ctx, oracle, leaf):
    """Cells about the centre of a sphere: every node of every level may hold the nearest triangle, at
    blocks of two 5120 nodes on the last level (the pass keeps 2048 and walks the others' subtrees)."""
    import sdfb
    from sdfb import meshgen as mg
    v, f = mg.icosphere(7)
    v, n, voxel = (v * 0.4).astype(np.float32), (3, 4, 5), 1e-3
    origin = tuple(-0.5 * voxel * k for k in n)
    g = sdfb.make_grid(origin, voxel, n)
    d64 = oracle.distance(v, f, origin, voxel, n)
    ref = None
    for tile, budget in ((1, -1), (1, 64), (4, 64), (5, 64), (6, 64)):
        d, _ = ctx.bake(v, f, g, sdfb.make_opts(sign_mode=sdfb.SIGN_NONE, leaf_size=leaf, tile=tile, step_budget=budget,
                                                no_occupancy=True), want_occ=False)
        if ref is None:
            ref = d
            assert np.abs(d.reshape(-1) - d64).max() <= TOL * 0.8  # the sphere's diameter, not the grid's
        assert np.array_equal(d, ref), (tile, budget)


@pytest.mark.parametrize("T, leaf, blocks", [(1, 2, 1), (5, 2, 3), (5, 4, 2), (9, 8, 2), (64, 2, 32)])
def test_counted_work(ctx, T, leaf, blocks):
    """The counts are of tests that a lane had work for: one node with fewer than 32 blocks, seen by one tile."""
    import sdfb
    v, i = soup(T, T)
    st = sdfb.Stats()
    g = sdfb.make_grid((-0.5,) * 3, 0.25, (4, 4, 2))
    ctx.bake(v, i, g, sdfb.make_opts(sign_mode=sdfb.SIGN_NONE, leaf_size=leaf, tile=1, step_budget=-1, count_work=True,
                                     no_occupancy=True), want_occ=False, stats=st)
    assert (st.box_tests, st.plane_tests) == (0, blocks)
    assert st.rect_tests <= 32 * blocks and st.rect_tests % 32 == 0
    assert 32 * leaf <= st.tri_tests <= 32 * leaf * (1 + blocks) and st.tri_tests % leaf == 0


@pytest.mark.parametrize("T", [2, 12, 70, 600])
def test_large_triangles(ctx, oracle, T):
    """Triangles as large as the grid: most of a tile's cells want the blocks that survive, and are measured
    against them directly. Every block size, tile and pass gives the same bits."""
    import sdfb
    rng = np.random.default_rng(T)
    v = rng.uniform(-0.6, 0.6, (3 * T, 3)).astype(np.float32)
    i = np.arange(3 * T, dtype=np.uint32).reshape(-1, 3)
    n, origin, voxel = (30, 17, 26), (-0.5, -0.3, -0.45), 1.0 / 30
    g = sdfb.make_grid(origin, voxel, n)
    d64 = oracle.distance(v, i, origin, voxel, n)
    ref = None
    for leaf in (2, 4, 8):
        for tile, budget in [(t, b) for t in range(1, 7) for b in (-1, 64)]:
            d, _ = ctx.bake(v, i, g, sdfb.make_opts(sign_mode=sdfb.SIGN_NONE, leaf_size=leaf, tile=tile,
                                                    step_budget=budget, no_occupancy=True), want_occ=False)
            if ref is None:
                ref = d
                assert np.abs(d.reshape(-1) - d64).max() <= TOL * 1.2 * 3 ** 0.5  # the triangles' box
            assert np.array_equal(d, ref), (leaf, tile, budget)
