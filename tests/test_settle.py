"""A call that fails half way waits for what it has enqueued before it returns, since that reads and writes the
caller's buffers. The library's host code runs on a fake CUDA runtime (tests/fake_cudart.c) whose n-th call fails."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(lib, tmp_path_factory):
    import build as pkg_build
    import sdfb
    tmp = tmp_path_factory.mktemp("fake")
    obj, so = str(tmp / "fake.o"), str(tmp / "libsdfb_fake.so")
    subprocess.run(["gcc", "-O1", "-fPIC", "-I", "/usr/local/cuda/include", "-c", os.path.join(HERE, "fake_cudart.c"),
                    "-o", obj], check=True)
    objs = [os.path.join(pkg_build.BUILD, s + ".o") for s in pkg_build.CU_SOURCES + pkg_build.CPP_SOURCES]
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so, *objs, obj, "-lpthread", "-ldl"], check=True)
    return sdfb.load(so)


CALLS = ["bake", "bake_open", "bake_stats", "bake_device", "bake_occupancy", "soup", "soup_stats", "batch", "batch_device",
         "sparse", "materials"]


@pytest.mark.parametrize("call", CALLS)
def test_nothing_in_flight_after_an_error(fake, call):
    import sdfb
    from sdfb import meshgen as mg
    v, f = mg.icosphere(1)
    v, f = np.ascontiguousarray(v, np.float32), np.ascontiguousarray(f, np.uint32)
    p, T = v[f].reshape(-1, 3).copy(), len(f)
    g = sdfb.make_grid((-1.0,) * 3, 0.25, (8, 8, 8))
    dist, occ = np.zeros(4096, np.float32), np.zeros(4096, np.uint8)
    P = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    lo, hi = np.full(3, -1, np.float32), np.full(3, 1, np.float32)
    mats, keep = sdfb.make_materials(mg.random_materials(T, 1))
    out, n, u = np.zeros((4096, 3), np.float32), C.c_uint64(), sdfb.GridDesc()
    descs, grids = (sdfb.MeshDesc * 2)(), (sdfb.GridDesc * 2)(g, g)
    for d in descs:
        d.verts, d.idx, d.num_verts, d.num_tris = v.ctypes.data, f.ctypes.data, len(v), T
    dp, op = (C.c_void_p * 2)(*[dist.ctypes.data] * 2), (C.c_void_p * 2)(*[occ.ctypes.data] * 2)
    gwn = C.byref(sdfb.make_opts(sign_mode=sdfb.SIGN_GWN))
    st = sdfb.Stats()

    def run(h):
        if call == "bake_device":
            return fake.sdfb_bake_device(h, P(v), len(v), P(f), T, C.byref(g), None, P(dist), P(occ), None, None)
        if call.startswith("bake"):
            return fake.sdfb_bake(h, P(v), len(v), P(f), T, C.byref(g), gwn if call == "bake_open" else None,
                                  None if call == "bake_occupancy" else P(dist), P(occ),
                                  C.byref(st) if call == "bake_stats" else None)
        if call.startswith("soup"):
            return fake.sdfb_bake_soup(h, P(p), T, P(lo), P(hi), 8, None, C.byref(u), P(dist), P(occ),
                                       C.byref(st) if call == "soup_stats" else None)
        if call.startswith("batch"):
            # a fake GPU captures no graph: its refusal stands for an error as good as any
            return (fake.sdfb_bake_batch(h, 2, descs, grids, None, dp, op, None) if call == "batch" else
                    fake.sdfb_bake_batch_device(h, 2, descs, grids, None, dp, op, None, None))
        if call == "sparse":
            return fake.sdfb_voxelize_sparse(h, P(p), T, P(lo), P(hi), 8, P(out), 64, C.byref(n), None, None)
        return fake.sdfb_bake_materials(h, P(p), T, C.byref(g), C.byref(mats), P(out), None, None)

    fake.fake_fail_at.argtypes = [C.c_long]
    fake.fake_calls.restype = C.c_long
    failed = 0
    for k in range(1, 400):
        h = C.c_void_p()
        fake.fake_fail_at(0)
        fake.fake_reset()
        assert fake.sdfb_ctx_create(0, C.byref(h)) == 0
        fake.fake_fail_at(k)
        status = run(h)
        reached = fake.fake_calls() >= k
        assert fake.fake_pending() == 0, (k, status, fake.sdfb_last_error(h))
        assert not reached or status != 0 or call.startswith("batch")
        failed += status != 0
        fake.sdfb_ctx_destroy(h)
        if not reached:
            break
    assert failed > 10 and not reached
