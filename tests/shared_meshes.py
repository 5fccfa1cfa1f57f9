"""Scene views whose instances' meshes have nodes or triangles in common, made by hand (the library's
own builder gives every mesh a tree of its own)."""
import ctypes as C

import numpy as np

import lavaframe_gb300 as lf

# the second mesh is a subtree of the first (moved or in place), a leaf of it, or a leaf of its own over
# the first one's triangles; "chain" has a third instance on a subtree of the second's
KINDS = ["subtree moved", "subtree", "leaf moved", "leaf", "same triangles", "chain"]
_F, _I = C.POINTER(C.c_float), C.POINTER(C.c_int32)


class View:
    """Twelve triangles in four leaves under three inner nodes, and two or three instances of parts of
    that tree; holds the arrays of its lf_scene_view."""

    def __init__(self, kind):
        r = np.random.default_rng(7)
        n = 12
        self.verts = np.zeros((3 * n, 4), np.float32)
        c = np.repeat(np.arange(n)[:, None] % 3 + np.array([[0.0, 0.5, 0.25]]), 3, 0)
        self.verts[:, :3] = c + 0.7 * r.standard_normal((3 * n, 3))
        self.norms = np.tile(np.array([[0, 0, 1, 0]], np.float32), (3 * n, 1))
        self.index = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
        # mesh nodes: 0 root (1, 2); 1 inner (3, 4); 2 inner (5, 6); 3..6 leaves of three triangles; 7 a
        # second leaf over the triangles of node 3
        self.nodes = np.zeros((13, 9), np.float32)

        def box(k, tris):
            v = self.verts[np.concatenate([self.index[t] for t in tris]), :3]
            self.nodes[k, 0:3], self.nodes[k, 3:6] = v.min(0), v.max(0)

        for k, (left, right) in {0: (1, 2), 1: (3, 4), 2: (5, 6)}.items():
            self.nodes[k, 6:9] = left, right, 0
        for k in range(3, 8):
            first = 3 * (k - 3) if k < 7 else 0
            self.nodes[k, 6:9] = first, 3, 1
            box(k, range(first, first + 3))
        box(0, range(12)), box(1, range(6)), box(2, range(6, 12))
        moved = kind in ("subtree moved", "leaf moved", "chain")
        roots = {"subtree moved": [0, 1], "subtree": [0, 2], "leaf moved": [0, 4], "leaf": [0, 4],
                 "same triangles": [3, 7], "chain": [0, 2, 5]}[kind]
        self.xf = np.tile(np.eye(4, dtype=np.float32), (len(roots), 1, 1))
        for i in range(1, len(roots)):
            self.xf[i, 3, 0] = 0.75 * i if moved else 0.0
        # instance level: leaves 8.., then inner nodes, the last one on top
        for i, root in enumerate(roots):
            k = 8 + i
            self.nodes[k, 0:6] = self.nodes[root, 0:6]
            self.nodes[k, [0, 3]] += self.xf[i, 3, 0]
            self.nodes[k, 6:9] = root, 0, -(i + 1)
        top = 8
        for i in range(1, len(roots)):
            k = 10 + i
            self.nodes[k, 0:3] = np.minimum(self.nodes[top, 0:3], self.nodes[8 + i, 0:3])
            self.nodes[k, 3:6] = np.maximum(self.nodes[top, 3:6], self.nodes[8 + i, 3:6])
            self.nodes[k, 6:9] = top, 8 + i, 0
            top = k
        self.mats = np.zeros((1, 28), np.float32)
        self.mats[:, 24:] = -1.0

        def f(a):
            return a.ctypes.data_as(_F)

        self.view = lf.SceneView(nodes=f(self.nodes), num_nodes=len(self.nodes), top_level_index=top,
                                 vert_indices=self.index.ctypes.data_as(_I), num_tris=n, vertices_uvx=f(self.verts),
                                 normals_uvy=f(self.norms), num_vertices=3 * n, materials=f(self.mats), num_materials=1,
                                 transforms=f(self.xf), num_instances=len(roots))


class _Scene:
    def __init__(self, ctx, h):
        self.ctx, self.h = ctx, h

    def close(self):
        self.ctx._c(lf.lib().lf_scene_release(self.h))


def upload(ctx, v):
    h = C.c_void_p()
    ctx._c(lf.lib().lf_scene_upload(ctx.h, C.byref(v.view), C.byref(h)))
    return _Scene(ctx, h)
