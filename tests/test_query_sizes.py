"""Ray queries at the sizes where their dispatch changes: rays per warp, first chunk and counter,
page-locked staging of small host queries, binning, cells per axis. All equal the plain
one-thread-per-ray kernel."""
import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    ctx = lf.Context(0)
    s = lf.HostScene().gen_room(60, 4).build()
    ds = ctx.upload(s)
    rays = lf.gen_rays([0, 0, 0], [10, 4, 10], (1 << 23) + 1, 3, tmax=6.0)
    yield ctx, ds, rays
    ds.close()
    ctx.close()


# 4256 warps hold the GPU at 7 blocks of 4 warps on 152 SMs; 5461 and 7943 are the most rays whose
# rays and results fit the staging block (closest, any)
@pytest.mark.parametrize("n", [1, 2, 31, 33, 4255, 4256, 4257, 5461, 5462, 7943, 7944, 68096, 68097, 136192, 136193,
                               (1 << 19) - 1, 1 << 19, (1 << 19) + 1])
def test_sizes_equal_the_plain_kernel(world, n):
    ctx, ds, rays = world
    q = rays[:n]
    for trace in (ctx.trace_closest, ctx.trace_any):
        ref = trace(ds, q, flags=lf.TRACE_SIMPLE | lf.TRACE_LIGHTS)
        for flags in (0, lf.TRACE_UNSORTED):
            assert trace(ds, q, flags=flags | lf.TRACE_LIGHTS).tobytes() == ref.tobytes()


@pytest.mark.parametrize("n", [(1 << 23) - 1, 1 << 23, (1 << 23) + 1])
def test_binned_occlusion_and_fine_cells(world, n):
    ctx, ds, rays = world
    q = rays[:n]
    for trace in (ctx.trace_closest, ctx.trace_any):
        assert trace(ds, q).tobytes() == trace(ds, q, flags=lf.TRACE_UNSORTED).tobytes()
