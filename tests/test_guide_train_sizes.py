"""Guide gradients on tcgen05 at the edges of its 128-sample tiles and of its one-tile-per-SM grid,
against the warp-level kernel on the same samples. Both round activations and gradients to FP16 at
the same places and differ in the order of FP32 sums, so a weight's gradient differs by flips of
single FP16 roundings: 2^-11 of a term each, over four layers in each direction, so by less than
8 x 2^-11 of the gradients' norm."""
import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu

BOUND = 8 * 2.0 ** -11


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 5000, 128 * 152, 128 * 152 + 1, 128 * 152 * 2 + 77])
def test_gradients_equal_the_warp_level_kernel(n):
    r = np.random.default_rng(n)
    q = np.zeros((n, 16), np.float32)
    q[:, 0:3] = r.random((n, 3))
    for k in (3, 6, 9):
        d = r.standard_normal((n, 3))
        q[:, k:k + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    q[:, 12] = r.random(n) + 0.1
    with lf.Context(0) as ctx:
        g = lf.Guide(ctx, [0, 0, 0], [1, 1, 1], seed=3)
        w, t = g.params()
        g.set_params(w, t * 2000.0)
        out = []
        for tensor in (False, True):
            g.set_tensor_path(tensor)
            out.append(g.gradients(q))
        assert ctx.device_errors() == 0
        g.close()
    (l0, w0, t0), (l1, w1, t1) = out
    assert abs(l0 - l1) <= BOUND * max(1.0, abs(l0))
    for a, b in ((w0, w1), (t0, t1)):
        assert np.linalg.norm(a - b) <= BOUND * np.linalg.norm(a)
