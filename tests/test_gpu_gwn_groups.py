"""Winding-number signs where the grouped walk can go wrong: grids smaller than a tile and just past
one, single triangles, one wide opening (large caps beside the cells) and overlapping shells, against
the FP64 sum over every triangle."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(kind):
    from sdfb import meshgen as mg
    if kind == "triangle":
        return np.array([[-0.3, -0.2, 0.1], [0.35, -0.1, -0.2], [0.0, 0.4, 0.15]], np.float32), np.array([[0, 1, 2]], np.uint32)
    v, f = mg.displaced_icosphere(3, 0.33, 3)
    if kind == "bowl":  # a wide opening: its fan of caps crosses the whole mesh
        return v, np.ascontiguousarray(f[v[f].mean(axis=1)[:, 2] < 0.12])
    w, g = mg.displaced_icosphere(3, 0.25, 4, center=(0.12, 0.05, -0.1))
    return mg.delete_faces(*mg.concat([(v, f), (w, g[:, ::-1])]), 0.03, 5)  # opposite orientations


@pytest.mark.parametrize("kind", ["triangle", "bowl", "shells"])
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 5, 2), (4, 4, 8), (5, 9, 17), (33, 31, 30)])
def test_group_walk_signs(ctx, oracle, kind, dims):
    """Every cell whose FP64 winding number is not on the level set, in and out of the band; a cell
    within 1e-6 of the surface or a cap has no robust side."""
    import sdfb
    v, f = _mesh(kind)
    voxel = 0.9 / max(dims)
    origin = tuple(-0.5 * voxel * d + 0.003 for d in dims)
    g = sdfb.make_grid(origin, voxel, dims)
    d, _ = ctx.bake(v, f, g, sdfb.make_opts(sign_mode=sdfb.SIGN_GWN))
    w = oracle.gwn(v, f, origin, voxel, dims)
    d64 = oracle.distance(v, f, origin, voxel, dims)
    sure = (np.abs(np.abs(w) - 0.5) > 1e-6) & (d64 > 1e-6)
    assert np.array_equal(d.reshape(-1)[sure] < 0, np.abs(w[sure]) > 0.5)


@pytest.mark.parametrize("level, direct", [(3, True), (7, False)])
def test_cells_left_by_the_coarse_pass(ctx, oracle, level, direct):
    """A bowl's opening, where many cells lie near the level set: with a short rim they are summed
    directly, with a long one walked again, and both give the FP64 sum's sides."""
    import sdfb
    from sdfb import meshgen as mg
    v, f = mg.displaced_icosphere(level, 0.33, 3)
    f = np.ascontiguousarray(f[v[f].mean(axis=1)[:, 2] < 0.12])
    dims = (130, 131, 40)
    voxel, origin = 0.7 / 130, (-0.351, -0.352, 0.0)
    st = sdfb.Stats()
    d, _ = ctx.bake(v, f, sdfb.make_grid(origin, voxel, dims), sdfb.make_opts(sign_mode=sdfb.SIGN_GWN), stats=st)
    assert st.gwn_fp64_cells > 0 and (st.gwn_direct_cells > 100) == direct
    samples = np.sort(np.random.default_rng(level).choice(np.prod(dims), 3000, replace=False)).astype(np.int64)
    w = oracle.gwn(v, f, origin, voxel, dims, samples=samples)
    d64 = oracle.distance(v, f, origin, voxel, dims, samples=samples)
    sure = (np.abs(np.abs(w) - 0.5) > 1e-6) & (d64 > 1e-6)
    assert np.array_equal(d.reshape(-1)[samples][sure] < 0, np.abs(w[sure]) > 0.5)


def test_more_crossings_than_the_lists_hold(oracle):
    """Many large triangles on a small grid: the first pass over the columns finds far more crossings than the lists
    were made for. The winding number then reads what they hold, and the bake is repeated with longer ones."""
    import sdfb
    rng = np.random.default_rng(3)
    T, n, voxel, origin = 3000, (24, 22, 20), 0.05, (-0.6, -0.55, -0.5)
    v = rng.uniform(-0.7, 0.7, (3 * T, 3)).astype(np.float32)
    f = np.arange(3 * T, dtype=np.uint32).reshape(-1, 3)
    g = sdfb.make_grid(origin, voxel, n)
    opts = sdfb.make_opts(sign_mode=sdfb.SIGN_GWN)
    with sdfb.Context(0) as ctx:  # a fresh one: lists at their least
        d, _ = ctx.bake(v, f, g, opts)
        st = sdfb.Stats()
        again, _ = ctx.bake(v, f, g, opts, stats=st)
    assert st.crossings > 4 * (4 * n[0] * n[1] + 2 * 4 * T)  # mesh and caps: the least, several times over
    assert np.array_equal(d, again)
    w = oracle.gwn(v, f, origin, voxel, n)
    d64 = oracle.distance(v, f, origin, voxel, n)
    sure = (np.abs(np.abs(w) - 0.5) > 1e-5) & (d64 > 1e-5)
    assert sure.mean() > 0.9 and np.array_equal(d.reshape(-1)[sure] < 0, np.abs(w[sure]) > 0.5)
