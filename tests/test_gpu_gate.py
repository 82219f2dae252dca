"""The hashed weld and watertight gate of indexed meshes at block edges and in awkward meshes, against
the host weld and census of the de-indexed soup."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(kind, tris):
    from sdfb import meshgen as mg
    nv = max(3, int(round((tris / 6.0) ** 0.5)))
    v, f = mg.displaced_torus(max(3, int(round(tris / (2.0 * nv)))), nv, 0.28, 0.1, tris)
    if kind == "hole":
        f = f[:-1]
    elif kind == "doubled":
        f = np.concatenate([f, f[:1]])
    elif kind == "split":  # every triangle its own vertices: closed only through the weld
        v, f = v[f.reshape(-1)], np.arange(f.size, dtype=np.uint32).reshape(-1, 3)
    elif kind == "jitter":  # the same, moved within the lattice cell now and then
        v = v[f.reshape(-1)]
        v = (v + np.random.default_rng(3).normal(0.0, 3e-7, v.shape)).astype(np.float32)
        f = np.arange(f.size, dtype=np.uint32).reshape(-1, 3)
    elif kind == "point":  # all vertices equal: every triangle is degenerate
        v = np.full_like(v, 0.25)
    return np.ascontiguousarray(v, np.float32), np.ascontiguousarray(f, np.uint32)


@pytest.mark.parametrize("tris", [18, 510, 1026, 2100, 20000])
def test_gate_verdicts(ctx, tris):
    """One mesh at a time and all in one batch."""
    import sdfb
    g = sdfb.make_grid((-0.5,) * 3, 1.0 / 8, (8, 8, 8))
    st = sdfb.Stats()
    meshes, want = [], []
    for kind in ("closed", "hole", "doubled", "split", "jitter", "point"):
        v, f = _mesh(kind, tris)
        w, _ = sdfb.weld(v, v.min(0), v.max(0))
        ok = sdfb.is_watertight(w[f.reshape(-1)])[0]
        st.struct_size = sdfb.C.sizeof(sdfb.Stats)
        ctx.bake(v, f, g, sdfb.make_opts(no_distance=True), want_dist=False, stats=st)
        assert st.watertight == int(ok), kind
        meshes.append((v, f))
        want.append(ok)
    assert want[0] and not want[1] and not want[2] and want[3]
    dists, _ = ctx.bake_batch(meshes, [g] * len(meshes), sdfb.make_opts())
    for (v, f), d, ok in zip(meshes, dists, want):
        mode = sdfb.SIGN_PARITY if ok else sdfb.SIGN_GWN
        assert np.array_equal(d < 0, ctx.bake(v, f, g, sdfb.make_opts(sign_mode=mode))[0] < 0)


def test_gate_bad_index(ctx):
    import sdfb
    g = sdfb.make_grid((-0.5,) * 3, 1.0 / 8, (8, 8, 8))
    v, f = _mesh("closed", 1026)
    bad = f.copy()
    bad[700, 1] = len(v)
    assert ctx.bake_status(v, bad, g)[0] == sdfb.ERR_BAD_MESH
    with pytest.raises(sdfb.SdfbError) as e:
        ctx.bake_batch([(v, f), (v, bad)], [g, g], sdfb.make_opts())
    assert e.value.status == sdfb.ERR_BAD_MESH and "mesh 1" in str(e.value)


def test_batch_gate_in_runs():
    """A batch whose tables do not fit the gate's share of memory together: the meshes go through it in runs,
    which reuse one buffer, and every mesh gets its own verdict (a closed mesh's sign would be wrong for the
    open one, in the columns below its hole)."""
    import sdfb
    import torch
    from sdfb import meshgen as mg
    v, f = mg.displaced_torus(1025, 512, 0.28, 0.1, 3)  # just past 2^20 triangles: 111 MB of tables
    c = v[f].mean(axis=1)
    g = np.ascontiguousarray(f[~((c[:, 2] > 0.0) & (np.abs(c[:, 1]) < 0.15) & (c[:, 0] > 0))])
    dv = torch.as_tensor(v).cuda()
    df, dg = torch.as_tensor(f.astype(np.int32)).cuda(), torch.as_tensor(g.astype(np.int32)).cuda()
    closed = (dv.data_ptr(), len(v), df.data_ptr(), len(f))
    opened = (dv.data_ptr(), len(v), dg.data_ptr(), len(g))
    meshes = [opened if k % 5 == 2 else closed for k in range(24)]
    grid = sdfb.make_grid((-0.5,) * 3, 1.0 / 24, (24,) * 3)
    dist = torch.empty(24, *grid.shape, device="cuda")
    occ = torch.empty(24, *grid.shape, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    at = [d.data_ptr() for d in dist], [o.data_ptr() for o in occ]
    with sdfb.Context(0) as ctx:
        # Occupancy with statistics: the gate's tables are nearly all that the call allocates.
        ctx.bake_batch_device(meshes, [grid] * 24, None, None, at[1], stats=sdfb.Stats())
        assert ctx.device_bytes() < 1.6 * 2 ** 30
        ctx.bake_batch_device(meshes, [grid] * 24, None, *at)
        lone = {m: ctx.bake(v, i, grid)[0] for m, i in ((closed, f), (opened, g))}
        wrong = ctx.bake(v, g, grid, sdfb.make_opts(sign_mode=sdfb.SIGN_PARITY))[0]
    assert (np.signbit(wrong) != np.signbit(lone[opened])).sum() > 10
    for d, m in zip(dist.cpu().numpy(), meshes):
        assert np.array_equal(np.signbit(d), np.signbit(lone[m]))
