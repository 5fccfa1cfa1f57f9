"""Paths of more than 4096 bounces - the most that one thread takes a path through in one launch - in a
closed box of mirrors that emit a little, without Russian roulette: every bounce counts."""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf
import oracle

pytestmark = pytest.mark.gpu


def mirrors():
    s = lf.HostScene()
    m = np.zeros(28, np.float32)
    m[0:3], m[4:7], m[8], m[17], m[18], m[20:23], m[24:28] = 1.0, 1e-3, 1.0, 1.45, 1.0, 1.0, -1.0
    mat = s.add_material(m)
    v, n = [], []
    for axis in range(3):
        for side in (-1, 1):
            u, w, c = np.eye(3)[(axis + 1) % 3], np.eye(3)[(axis + 2) % 3], np.eye(3)[axis] * side
            p = [c - u - w, c + u - w, c + u + w, c - u + w]
            for k in (0, 1, 2, 0, 2, 3):
                v.append([*p[k], 0])
                n.append([*(-c), 0])
    mesh = s.add_mesh(np.array(v, np.float32), np.array(n, np.float32))
    s.add_instance(mesh, np.eye(4, dtype=np.float32).ravel(), mat)
    s.set_camera([0.1, 0.2, -0.3], [0.3, 0.1, 0.9], 60.0)
    return s.build()


@pytest.mark.parametrize("depth,tile", [(4095, 0), (4096, 0), (4097, 0), (5000, 0), (5000, 7)])
def test_every_bounce_counts(depth, tile):
    s = mirrors()
    p = s.render_params()
    p.width, p.height, p.enable_rr, p.max_depth = 16, 8, 0, depth
    p.tile_width = p.tile_height = tile
    want, _, _ = oracle.render(s.view(), p, 0, 1)
    L = lf.lib()
    with lf.Context(0) as ctx:
        ds = ctx.upload(s)
        for flags in (0, lf.FRAME_PER_BATCH):
            f = lf.Frame(ctx, ds, p, flags)
            f.render(0, 1)
            assert f.accum().tobytes() == want.tobytes()
            f.close()
        d = C.c_void_p()
        out = np.zeros((8, 16, 4), np.float32)
        ctx._c(L.lf_device_alloc(ctx.h, out.nbytes, C.byref(d)))
        ctx._c(L.lf_copy_to_device(ctx.h, d, out.ctypes.data_as(C.c_void_p), out.nbytes))
        ctx._c(L.lf_render_noalloc(ds.h, C.byref(p), 0, 1, d))
        ctx._c(L.lf_copy_to_host(ctx.h, out.ctypes.data_as(C.c_void_p), d, out.nbytes))
        ctx._c(L.lf_device_free(ctx.h, d))
        assert np.ascontiguousarray(out[..., :3]).tobytes() == want.tobytes()
        ds.close()
