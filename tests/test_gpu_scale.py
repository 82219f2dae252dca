"""Bakes far from the unit box: a mesh and its grid scaled together by a power of two change no rounding,
so distances scale with them and signs stay, as long as the squares of lengths fit FP32."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-40, 30, 45, 50, 55, 61, 63])
def test_distance_at_scale(ctx, exponent):
    """63: the largest squares are just below FP32's largest value, and cells up to 1.2e19 away."""
    import sdfb
    from sdfb import meshgen as mg
    v, f = mg.displaced_icosphere(4, 0.35, 3)
    n, origin, voxel = (29, 22, 35), (-0.9, -0.5, -0.6), 1.0 / 24
    s = np.float32(2.0) ** exponent

    def bake(k, **opts):
        g = sdfb.make_grid(tuple(float(np.float32(o) * k) for o in origin), float(np.float32(voxel) * k), n)
        return ctx.bake(v * k, f, g, sdfb.make_opts(sign_mode=sdfb.SIGN_NONE, no_occupancy=True, **opts),
                        want_occ=False)[0]

    ref = bake(np.float32(1.0))
    for opts in ({}, {"tile": 1, "leaf_size": 2}, {"tile": 6, "step_budget": 64}):
        d = bake(s, **opts)
        if exponent > 0:
            assert np.array_equal(d, ref * s), opts
        else:  # squares of the smallest distances lose bits below 2^-126
            assert np.abs(d / s - ref).max() <= 16 * 2.0 ** -24 * 2.0, opts


@pytest.mark.parametrize("exponent", [-20, 24, 40])
@pytest.mark.parametrize("kind", ["bowl", "shells"])
@pytest.mark.parametrize("band", [1.0, 1000.0])
def test_signs_at_scale(ctx, kind, band, exponent):
    """The signs, and the cells that the bounds leave to FP64 and to the direct sum, do not depend on the scale."""
    import sdfb
    from sdfb import meshgen as mg
    v, f = mg.displaced_icosphere(4, 0.33, 3)
    if kind == "bowl":  # a wide opening: its fan of caps crosses the whole mesh
        f = np.ascontiguousarray(f[v[f].mean(axis=1)[:, 2] < 0.12])
    else:
        w, g = mg.displaced_icosphere(4, 0.25, 4, center=(0.12, 0.05, -0.1))
        v, f = mg.delete_faces(*mg.concat([(v, f), (w, g[:, ::-1])]), 0.03, 5)
    n, origin, voxel = (65, 62, 59), (-0.42, -0.4, -0.38), 0.8 / 62

    def bake(k):
        g = sdfb.make_grid(tuple(float(np.float32(o) * k) for o in origin), float(np.float32(voxel) * k), n)
        st = sdfb.Stats()
        d = ctx.bake(v * k, f, g, sdfb.make_opts(sign_mode=sdfb.SIGN_GWN, band_voxels=band, no_occupancy=True),
                     want_occ=False, stats=st)[0]
        return d, (st.gwn_fp64_cells, st.gwn_direct_cells)

    (d0, left0), (d1, left1) = bake(np.float32(1.0)), bake(np.float32(2.0) ** exponent)
    assert left0 == left1
    assert np.array_equal(np.signbit(d0), np.signbit(d1))
