"""Instances whose meshes have nodes or triangles in common are not merged into the instance level: hits,
instance ids, ties and occlusion are the oracle's."""
import numpy as np
import pytest

import lavaframe_gb300 as lf
import oracle
from tests import shared_meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", shared_meshes.KINDS)
def test_hits_equal_the_oracle(kind):
    v = shared_meshes.View(kind)
    q = lf.gen_rays([-1, -1, -1], [4, 2, 2], 4096, 5)
    with lf.Context(0) as ctx:
        ds = shared_meshes.upload(ctx, v)
        ref, _ = oracle.trace_closest(v.view, q)
        occ, _ = oracle.trace_any(v.view, q)
        assert ctx.trace_closest(ds, q).tobytes() == ref.tobytes() and np.array_equal(ctx.trace_any(ds, q), occ)
        assert (ref["prim"] >= 0).sum() > 50   # 125 to 400 of the rays hit
        ds.close()
