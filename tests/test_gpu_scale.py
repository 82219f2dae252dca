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
