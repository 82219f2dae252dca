"""Winding-number signs of cells in the plane of an opening, within a few 1e-8 of its cap, where FP32 can put a
cap's solid angle on the other side of it, 4 pi off."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 128


def _tube(direction, seed):
    """A square tube open at both ends, and a grid with many cell centres in the first opening's plane but for
    rounding. The plane is vertical, so that the columns' crossings are exact there: its xy line runs along
    `direction` through a lattice point, and the corners are chosen so that their mean, the centre of the cap's
    fan, lies on it exactly."""
    rng = np.random.default_rng(seed)
    voxel = np.float32(rng.uniform(0.9, 1.1) / N)
    origin = rng.uniform(-0.55, -0.45, 3).astype(np.float32)
    base = origin[:2].astype(np.float64) + 64.5 * float(voxel)
    step = np.array(direction) * float(voxel) / np.abs(direction).max()
    p = (base - step * rng.uniform(35, 45)).astype(np.float32).astype(np.float64)
    while True:
        q = (base + step * rng.uniform(35, 45)).astype(np.float32).astype(np.float64)
        if np.array_equal(((p + q) / 2).astype(np.float32), (p + q) / 2):
            break
    while True:
        z = np.array([rng.uniform(-0.33, -0.27), rng.uniform(0.27, 0.33)]).astype(np.float32)
        if np.float32(z.astype(np.float64).mean()) == z.astype(np.float64).mean():
            break
    back = np.array([q[1] - p[1], p[0] - q[0]]) * 0.35  # the tube's length
    v = np.array([[*r, h] for h in z for r in (p, q, q + back, p + back)]).astype(np.float32)
    quads = [(0, 1, 2, 3), (7, 6, 5, 4), (1, 5, 6, 2), (0, 3, 7, 4)]  # bottom, top and the two sides
    f = [t for a, b, c, d in quads for t in ((a, b, c), (a, c, d))]
    return v, np.array(f, np.uint32), origin, float(voxel)


@pytest.mark.parametrize("band", [1.0, 1000.0])
@pytest.mark.parametrize("direction, seed", [((3, -4), 3), ((2, -5), 2), ((1, -3), 3), ((2, -3), 0)])
def test_cells_in_the_plane_of_an_opening(ctx, oracle, direction, seed, band):
    import sdfb
    v, f, origin, voxel = _tube(direction, seed)
    d, _ = ctx.bake(v, f, sdfb.make_grid(origin, voxel, (N, N, N)),
                    sdfb.make_opts(sign_mode=sdfb.SIGN_GWN, band_voxels=band, no_occupancy=True), want_occ=False)
    c = [(origin[a] + (np.arange(N, dtype=np.float32) + np.float32(0.5)) * np.float32(voxel)).astype(np.float64)
         for a in range(3)]
    a, t = v[0, :2].astype(np.float64), v[1, :2].astype(np.float64) - v[0, :2]
    y, x = np.meshgrid(c[1], c[0], indexing="ij")
    off = ((x - a[0]) * t[1] - (y - a[1]) * t[0]) / np.hypot(*t)
    along = ((x - a[0]) * t[0] + (y - a[1]) * t[1]) / (t @ t)
    columns = np.flatnonzero((np.abs(off) < 1e-7) & (off != 0) & (along > 0.03) & (along < 0.97))
    layers = np.flatnonzero((c[2] > v[0, 2] + 0.02) & (c[2] < v[4, 2] - 0.02))
    cells = (columns[None, :] + N * N * layers[:, None]).reshape(-1).astype(np.int64)
    assert len(cells) > 1000
    w = oracle.gwn(v, f, origin, voxel, (N, N, N), samples=cells)
    assert (np.abs(np.abs(w) - 0.5) > 1e-3).all()
    assert np.array_equal(d.reshape(-1)[cells] < 0, np.abs(w) > 0.5)
