"""The tree built beside the gate, which a bake without statistics takes: the same grids as stage by
stage, and the same refusals."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(kind):
    from sdfb import meshgen as mg
    v, f = mg.displaced_icosphere(3, 0.35, 5)
    if kind == "open":
        v, f = mg.delete_faces(v, f, 0.03, 7)
    return (v, f) if kind != "one" else (v, f[:1])


@pytest.mark.parametrize("kind", ["closed", "open", "one"])
@pytest.mark.parametrize("call", ["host", "device", "soup"])
def test_same_grids(ctx, kind, call):
    import sdfb
    import torch
    v, f = _mesh(kind)
    g = sdfb.make_grid((-0.5,) * 3, 1.0 / 21, (21, 22, 23))

    def bake(stats):
        if call == "host":
            return ctx.bake(v, f, g, stats=stats)
        if call == "soup":
            _, d, o = ctx.bake_soup(v[f].reshape(-1, 3), v.min(0), v.max(0), 17, stats=stats)
            return d, o
        dv, df = torch.as_tensor(v).cuda(), torch.as_tensor(f.astype(np.int32)).cuda()
        d, o = torch.empty(23, 22, 21, device="cuda"), torch.empty(23, 22, 21, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        ctx.bake_device(dv.data_ptr(), len(v), df.data_ptr(), len(f), g, sdfb.make_opts(), d.data_ptr(), o.data_ptr(),
                        stats=stats)
        return d.cpu().numpy(), o.cpu().numpy()

    d0, o0 = bake(sdfb.Stats())
    for _ in range(2):
        d1, o1 = bake(None)
        assert np.array_equal(d0, d1) and np.array_equal(o0, o1)


@pytest.mark.parametrize("want_occ", [True, False])
@pytest.mark.parametrize("fault", ["index", "nan"])
def test_same_refusals(ctx, fault, want_occ):
    import sdfb
    v, f = _mesh("closed")
    w, h = v.copy(), f.copy()
    if fault == "index":
        h[17, 1] = len(v)
    else:
        w[f[17, 1], 2] = np.nan
    g = sdfb.make_grid((-0.5,) * 3, 1.0 / 16, (16, 16, 16))
    for stats in (None, sdfb.Stats()):
        with pytest.raises(sdfb.SdfbError) as e:
            ctx.bake(w, h, g, want_occ=want_occ, stats=stats)
        assert e.value.status == sdfb.ERR_BAD_MESH
        assert np.array_equal(*(ctx.bake(v, f, g, stats=s)[0] for s in (None, sdfb.Stats())))  # nothing is left behind


@pytest.mark.parametrize("sign", ["auto", "parity"])
def test_stream_under_capture(ctx, sign):
    """A bake on a stream that is being captured is refused, and leaves the context to other streams meanwhile."""
    import sdfb
    import torch
    v, f = _mesh("closed")
    g = sdfb.make_grid((-0.5,) * 3, 1.0 / 21, (21, 22, 23))
    dv, df = torch.as_tensor(v).cuda(), torch.as_tensor(f.astype(np.int32)).cuda()
    d, o = torch.zeros(g.shape, device="cuda"), torch.zeros(g.shape, dtype=torch.uint8, device="cuda")
    opts = sdfb.make_opts(sign_mode=sdfb.SIGN_AUTO if sign == "auto" else sdfb.SIGN_PARITY)

    def bake(stream):
        ctx.bake_device(dv.data_ptr(), len(v), df.data_ptr(), len(f), g, opts, d.data_ptr(), o.data_ptr(), stream)

    torch.cuda.synchronize()
    bake(0)
    want = d.cpu().numpy()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="relaxed")
        with pytest.raises(sdfb.SdfbError) as e:
            bake(stream.cuda_stream)
        assert e.value.status == sdfb.ERR_CUDA
        bake(0)  # on the context's own stream
        try:
            graph.capture_end()
        except RuntimeError:
            pass  # a wait inside the capture ended it
    assert np.array_equal(d.cpu().numpy(), want)
