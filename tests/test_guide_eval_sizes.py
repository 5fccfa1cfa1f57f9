"""Guide evaluation at the edges of its tiles and of its page-locked staging (1,149 queries at most):
every query's mixture and density are the ones it has in a larger batch, bit for bit."""
import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("n", [1, 15, 16, 127, 128, 129, 257, 1149, 1150, 3000])
def test_queries_do_not_depend_on_the_batch(n, tensor):
    r = np.random.default_rng(3)
    q = np.zeros((4000, 16), np.float32)
    q[:, 0:3] = r.random((4000, 3))
    for k in (3, 6, 9):
        d = r.standard_normal((4000, 3))
        q[:, k:k + 3] = d / np.linalg.norm(d, axis=1, keepdims=True)
    with lf.Context(0) as ctx:
        g = lf.Guide(ctx, [0, 0, 0], [1, 1, 1], seed=3)
        w, t = g.params()
        g.set_params(2.0 * w, t * 2000.0)
        g.set_tensor_path(tensor)
        mix, pdf = g.eval(q)
        m, p = g.eval(q[:n])
        assert ctx.device_errors() == 0
        g.close()
    assert m.tobytes() == mix[:n].tobytes()
    assert p.tobytes() == pdf[:n].tobytes()
    assert (p > 0).all()
