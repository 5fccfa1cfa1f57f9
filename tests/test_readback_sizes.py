"""Readbacks packed on the device (accumulation, display pass, guide gradients) at sizes that do not
divide their words and blocks."""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (2, 1), (3, 1), (5, 3), (85, 3), (256, 1), (257, 3), (512, 2)])
def test_accumulation_and_display_pass(size):
    with lf.Context(0) as ctx:
        s = lf.HostScene().gen_cornell(64, 64).build()
        p = s.render_params()
        p.width, p.height = size
        ds = ctx.upload(s)
        f = lf.Frame(ctx, ds, p)
        f.render(0, 3)
        acc = f.accum()
        paths = f.paths(3)
        assert acc.tobytes() == ((paths[0] + paths[1]) + paths[2]).tobytes()
        post = lf.PostParams.defaults(2)
        rgb8, rgbf = f.postprocess(3, post)
        want8, wantf = oracle.postprocess(acc, post, 3)
        assert rgb8.tobytes() == want8.tobytes()
        assert rgbf.tobytes() == np.ascontiguousarray(wantf[..., :3]).tobytes()
        # either output alone
        only8, onlyf = np.empty_like(rgb8), np.empty_like(rgbf)
        L = lf.lib()
        ctx._c(L.lf_frame_postprocess(f.h, C.byref(post), 3, only8.ctypes.data_as(C.c_void_p), None))
        ctx._c(L.lf_frame_postprocess(f.h, C.byref(post), 3, None, onlyf.ctypes.data_as(C.POINTER(C.c_float))))
        assert only8.tobytes() == rgb8.tobytes() and onlyf.tobytes() == rgbf.tobytes()
        f.close()
        ds.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
def test_gradients_leave_the_accumulators_clear(n):
    """Two calls in a row, and one after a training step, give the same gradients."""
    with lf.Context(0) as ctx:
        r = np.random.default_rng(2)
        q = r.standard_normal((n, 16)).astype(np.float32)
        for k in (3, 6, 9):
            q[:, k:k + 3] /= np.linalg.norm(q[:, k:k + 3], axis=1, keepdims=True)
        q[:, 12] = 1.0
        g = lf.Guide(ctx, [-3, -3, -3], [3, 3, 3], seed=4)
        w, t = g.params()
        first = g.gradients(q)
        again = g.gradients(q)
        g.train(q)
        g.set_params(w, t)
        after = g.gradients(q)
        g.close()
    for a in (again, after):
        # the sums are FP32 atomics in any order: n terms of up to the largest one's size
        for x, y in zip(first, a):
            x, y = np.asarray(x), np.asarray(y)
            assert np.abs(x - y).max() <= n * 2.0 ** -24 * max(np.abs(x).max(), 1e-6) * 8
