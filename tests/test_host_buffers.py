"""Host buffers that kernels may address themselves on a coherent host (aligned for their words) give
the results of buffers that are copied: unaligned ones, results that overlap their inputs, inputs in a
read-only file mapping, and the sizes at which device queries are binned."""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


def _shifted(a, by):
    """A copy of `a` that starts `by` bytes past a 64-byte boundary."""
    raw = np.empty(a.nbytes + 128, np.uint8)
    start = -raw.ctypes.data % 64 + by
    out = raw[start:start + a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


def _f(a):
    return a.ctypes.data_as(C.POINTER(C.c_float))   # holds on to the array


def _queries(n):
    r = np.random.default_rng(3)
    q = np.zeros((n, 16), np.float32)
    q[:, 0:3] = r.random((n, 3))
    for k in (3, 6, 9):
        d = r.standard_normal((n, 3))
        q[:, k:k + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    q[:, 12] = 1.0
    return q


@pytest.mark.parametrize("n", [7945, 100003, (1 << 19) - 1, 1 << 19])
def test_ray_queries(n, tmp_path):
    ctx = lf.Context(0)
    ds = ctx.upload(lf.HostScene().gen_room(60, 4).build())
    q = lf.gen_rays([0, 0, 0], [10, 4, 10], n, 3, tmax=6.0)
    q.tofile(tmp_path / "rays")
    mapped = np.memmap(tmp_path / "rays", np.float32, "r", shape=(n, 8))
    for name, elem in (("lf_trace_closest", 16), ("lf_trace_any", 1)):
        def call(src, dst, flags=0):
            ctx._c(getattr(lf.lib(), name)(ctx.h, ds.h, _f(src), n, C.c_void_p(dst.ctypes.data), flags))
            return dst.reshape(-1).view(np.uint8)[:n * elem].tobytes()

        ctx.set_host_chunks(2)   # pieces are copied
        ref = call(_shifted(q, 0), np.zeros(n * elem, np.uint8))
        ctx.set_host_chunks(0)
        for flags in (0, lf.TRACE_UNSORTED, lf.TRACE_SIMPLE):
            for by, to in ((0, 0), (4, 0), (16, 1), (16, 16)):
                assert call(_shifted(q, by), _shifted(np.zeros(n * elem, np.uint8), to), flags) == ref
        both = _shifted(q, 0)
        assert call(both, both) == ref
        assert call(mapped, np.zeros(n * elem, np.uint8)) == ref
    ds.close()
    ctx.close()


def test_queries_of_a_large_scene():
    """More triangles than host queries are traced in input order for."""
    ctx = lf.Context(0)
    ds = ctx.upload(lf.HostScene().gen_soup(151000, 10, 1).build())
    q = lf.gen_rays([0, 0, 0], [1, 1, 1], 1 << 19, 3, tmax=1.0e6)
    for trace in (ctx.trace_closest, ctx.trace_any):
        assert trace(ds, q).tobytes() == trace(ds, q, flags=lf.TRACE_UNSORTED).tobytes()
    ds.close()
    ctx.close()


@pytest.mark.parametrize("by", [1, 4, 8, 16])
def test_display_pass(by):
    ctx = lf.Context(0)
    s = lf.HostScene().gen_cornell(64, 64).build()
    p = s.render_params()
    p.width, p.height = 257, 3
    ds = ctx.upload(s)
    f = lf.Frame(ctx, ds, p)
    f.render(0, 1)
    post = lf.PostParams.defaults(2)
    want8, wantf = f.postprocess(1, post)
    got8 = _shifted(np.zeros_like(want8), by)
    gotf = _shifted(np.zeros_like(wantf), by & ~3)
    ctx._c(lf.lib().lf_frame_postprocess(f.h, C.byref(post), 1, C.c_void_p(got8.ctypes.data), _f(gotf)))
    f.close()
    ds.close()
    ctx.close()
    assert got8.tobytes() == want8.tobytes() and gotf.tobytes() == wantf.tobytes()


@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("by", [4, 8, 16])
def test_guide(by, tensor):
    n = 2003
    q = _queries(n)
    L = lf.lib()
    with lf.Context(0) as ctx:
        g = lf.Guide(ctx, [0, 0, 0], [1, 1, 1], seed=3)
        g.set_tensor_path(tensor)
        w, t = g.params()
        mix, pdf = g.eval(q)
        m, d = _shifted(np.zeros_like(mix), by), _shifted(np.zeros_like(pdf), by)
        ctx._c(L.lf_guide_eval(g.h, _f(_shifted(q, by)), n, _f(m), _f(d)))
        assert m.tobytes() == mix.tobytes() and d.tobytes() == pdf.tobytes()
        over = _shifted(q, 0)
        ctx._c(L.lf_guide_eval(g.h, _f(over), n, None, _f(over)))
        assert over.reshape(-1)[:n].tobytes() == pdf.tobytes()
        loss, dw, dt = g.gradients(q)
        ew, et, el = np.zeros_like(dw), _shifted(np.zeros_like(dt), by), C.c_float()
        ctx._c(L.lf_guide_gradients(g.h, _f(_shifted(q, by)), n, _f(ew), _f(et), C.byref(el)))
        g.close()
    # the sums are FP32 atomics in any order: n terms of up to the largest one's size
    for x, y in ((dw, ew), (dt, et), (np.float32(loss), np.float32(el.value))):
        assert np.abs(x - y).max() <= n * 2.0 ** -24 * max(np.abs(x).max(), 1e-6) * 8
