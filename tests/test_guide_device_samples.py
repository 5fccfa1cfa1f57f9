"""A training step on device samples that are aligned for floats only gives the weights of the same step on
aligned ones. One tile of 128 samples is one CTA, which adds each weight's gradient once, so the
weights are the same bits; the grid's are sums of atomics in any order, of one sample the same bits."""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128])
def test_shifted_samples(n):
    r = np.random.default_rng(n)
    q = np.zeros((n, 16), np.float32)
    q[:, 0:3] = r.random((n, 3))
    for k in (3, 6, 9):
        d = r.standard_normal((n, 3))
        q[:, k:k + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    q[:, 12] = r.random(n) + 0.1
    L, out = lf.lib(), []
    with lf.Context(0) as ctx:
        buf = C.c_void_p()
        ctx._c(L.lf_device_alloc(ctx.h, q.nbytes + 16, C.byref(buf)))
        for by in (0, 4, 8, 12):
            g = lf.Guide(ctx, [0, 0, 0], [1, 1, 1], seed=3)
            ctx._c(L.lf_copy_to_device(ctx.h, C.c_void_p(buf.value + by), q.ctypes.data_as(C.c_void_p), q.nbytes))
            ctx._c(L.lf_guide_train_device(g.h, C.c_void_p(buf.value + by), n, 1e-2))
            ctx.sync()
            out.append(g.params())
            g.close()
        ctx._c(L.lf_device_free(ctx.h, buf))
    for w, t in out[1:]:
        assert w.tobytes() == out[0][0].tobytes()
        assert n > 1 or t.tobytes() == out[0][1].tobytes()
