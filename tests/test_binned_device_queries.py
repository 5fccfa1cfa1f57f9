"""Binned queries of device buffers at the sizes where occlusion starts to be binned and 64 cells per
axis take the place of 32: the results are those of input order, where no ray is binned. (Host
queries of such a scene are traced in input order anyway.)"""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


def test_binned_occlusion_and_fine_cells():
    L, line = lf.lib(), 1 << 23
    rays = lf.gen_rays([0, 0, 0], [10, 4, 10], line + 1, 3, tmax=2.0)
    with lf.Context(0) as ctx:
        ds = ctx.upload(lf.HostScene().gen_room(60, 4).build())
        dr, dh = C.c_void_p(), C.c_void_p()
        ctx._c(L.lf_device_alloc(ctx.h, rays.nbytes, C.byref(dr)))
        ctx._c(L.lf_device_alloc(ctx.h, rays.nbytes // 2, C.byref(dh)))
        ctx._c(L.lf_copy_to_device(ctx.h, dr, rays.ctypes.data_as(C.c_void_p), rays.nbytes))
        for name, elem in (("lf_trace_closest_device", 16), ("lf_trace_any_device", 1)):
            for n in (line - 1, line, line + 1):
                got = []
                for flags in (0, lf.TRACE_UNSORTED, lf.TRACE_SIMPLE):
                    out = np.full(n * elem, 7, np.uint8)
                    ctx._c(L.lf_copy_to_device(ctx.h, dh, out.ctypes.data_as(C.c_void_p), out.nbytes))
                    ctx._c(getattr(L, name)(ctx.h, ds.h, dr, n, dh, flags))
                    ctx.sync()
                    ctx._c(L.lf_copy_to_host(ctx.h, out.ctypes.data_as(C.c_void_p), dh, out.nbytes))
                    got.append(out)
                assert got[0].tobytes() == got[1].tobytes() == got[2].tobytes()
                if elem == 1:
                    assert 0 < got[0].sum() < n
        for p in (dr, dh):
            ctx._c(L.lf_device_free(ctx.h, p))
        ds.close()
