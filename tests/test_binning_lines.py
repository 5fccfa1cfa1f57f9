"""Device queries on both sides of the sizes from which scenes of three sizes are binned: the results are those
of input order."""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


def _device(ctx, nbytes):
    p = C.c_void_p()
    ctx._c(lf.lib().lf_device_alloc(ctx.h, nbytes, C.byref(p)))
    return p


# 200 x 10, 900 x 10 and 121,000 x 10 triangles
@pytest.mark.parametrize("meshes, line", [(200, 1 << 21), (900, 1 << 19), (121000, 1 << 18)])
def test_lines(meshes, line):
    L = lf.lib()
    ctx = lf.Context(0)
    ds = ctx.upload(lf.HostScene().gen_soup(meshes, 10, 1).build())
    rays = lf.gen_rays([0, 0, 0], [100, 100, 100], line + 1, 3, tmax=1.0e6)
    dr, dh = _device(ctx, rays.nbytes), _device(ctx, rays.nbytes // 2)
    ctx._c(L.lf_copy_to_device(ctx.h, dr, rays.ctypes.data_as(C.c_void_p), rays.nbytes))
    for n in (line - 1, line, line + 1):
        got = []
        for flags in (0, lf.TRACE_UNSORTED):
            out = np.zeros((n, 4), np.int32)
            ctx._c(L.lf_copy_to_device(ctx.h, dh, out.ctypes.data_as(C.c_void_p), out.nbytes))
            ctx._c(L.lf_trace_closest_device(ctx.h, ds.h, dr, n, dh, flags))
            ctx.sync()
            ctx._c(L.lf_copy_to_host(ctx.h, out.ctypes.data_as(C.c_void_p), dh, out.nbytes))
            got.append(out)
        assert got[0].tobytes() == got[1].tobytes()
        assert (got[0][:, 2] >= 0).any()
    for p in (dr, dh):
        ctx._c(L.lf_device_free(ctx.h, p))
    ds.close()
    ctx.close()
