"""A scene of more than 2^26 triangles, the runs of which fill the upper bits of a wide node's leaf codes:
two instances of their own meshes at both ends of the triangle array. (Such an index is a float in
the scene's nodes, exact where it is a multiple of eight.)"""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu

_F, _I = C.POINTER(C.c_float), C.POINTER(C.c_int32)
FAR = 1 << 26


def test_hits_at_both_ends_of_the_array():
    n = FAR + 3
    v = np.zeros((6, 4), np.float32)
    v[0:3, :3] = [[0, 0, 0], [1, 0, 0], [0, 1, 0]]
    v[3:6, :3] = v[0:3, :3] + [4, 0, 0]
    index = np.zeros((n, 3), np.int32)
    index[:] = [0, 1, 2]
    index[FAR:] = [3, 4, 5]
    nodes = np.zeros((5, 9), np.float32)
    nodes[0] = [0, 0, 0, 1, 1, 0, 0, 3, 1]        # mesh leaves
    nodes[1] = [4, 0, 0, 5, 1, 0, FAR, 3, 1]
    nodes[2] = [0, 0, 0, 1, 1, 0, 0, 0, -1]       # instances
    nodes[3] = [4, 0, 0, 5, 1, 0, 1, 0, -2]
    nodes[4] = [0, 0, 0, 5, 1, 0, 2, 3, 0]
    norms = np.tile(np.array([[0, 0, 1, 0]], np.float32), (6, 1))
    mats = np.full((1, 28), -1.0, np.float32)
    for moved in (0.0, 2.0):   # the second instance merged into the instance level, and entered
        xf = np.tile(np.eye(4, dtype=np.float32), (2, 1, 1))
        xf[1, 3, 1] = moved
        nodes[3, [1, 4]] = [moved, moved + 1]
        nodes[4, 4] = moved + 1

        def f(a):
            return a.ctypes.data_as(_F)

        view = lf.SceneView(nodes=f(nodes), num_nodes=5, top_level_index=4, vert_indices=index.ctypes.data_as(_I),
                            num_tris=n, vertices_uvx=f(v), normals_uvy=f(norms), num_vertices=6, materials=f(mats),
                            num_materials=1, transforms=f(xf), num_instances=2)
        rays = np.zeros((3, 8), np.float32)
        rays[:, 0:3] = [[0.25, 0.25, -1], [4.25, moved + 0.25, -1], [2.5, 0.25, -1]]
        rays[:, 6], rays[:, 7] = 1.0, 1.0e6
        with lf.Context(0) as ctx:
            h = C.c_void_p()
            ctx._c(lf.lib().lf_scene_upload(ctx.h, C.byref(view), C.byref(h)))
            hits = np.zeros(3, lf.HIT_DTYPE)
            ctx._c(lf.lib().lf_trace_closest(ctx.h, h, f(rays), 3, hits.ctypes.data_as(C.c_void_p), 0))
            ctx._c(lf.lib().lf_scene_release(h))
        assert hits["instance"].tolist() == [0, 1, -1] and hits["prim"].tolist() == [0, FAR, -1]
        assert hits["t"][:2].tolist() == [1.0, 1.0]
