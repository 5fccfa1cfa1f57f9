"""The triangle test decides most triangles without the barycentric quotients: rays through
vertices, along edges and next to both, triangles without area and coordinates near the ends of the
float range give the oracle's hits bit for bit. Distance culling is off, as in the oracle: a triangle
without area can be hit at a distance that has nothing to do with its box."""
import numpy as np
import pytest

import lavaframe_gb300 as lf
import oracle

pytestmark = pytest.mark.gpu


def grid(scale, jitter, seed):
    """A 12 x 12 sheet of triangles, some without area, around the origin."""
    r = np.random.default_rng(seed)
    n = 12
    x, y = np.meshgrid(np.linspace(-1, 1, n + 1), np.linspace(-1, 1, n + 1), indexing="ij")
    z = jitter * r.standard_normal(x.shape)
    pts = np.stack([x, y, z], -1).astype(np.float32) * np.float32(scale)
    tris = []
    for i in range(n):
        for j in range(n):
            a, b, c, d = pts[i, j], pts[i + 1, j], pts[i + 1, j + 1], pts[i, j + 1]
            tris += [(a, b, c), (a, c, d)]
    tris += [(pts[0, 0], pts[0, 0], pts[1, 1]), (pts[0, 0], pts[1, 1], pts[2, 2]), (pts[3, 3],) * 3]
    return np.array(tris, np.float32)


@pytest.mark.parametrize("scale", [1.0, 1.0e-3, 1.0e-12, 1.0e5, 1.0e12, 3.0e18])
@pytest.mark.parametrize("jitter", [0.0, 0.1])
@pytest.mark.parametrize("flip", [False, True])
def test_edges_and_vertices(scale, jitter, flip):
    tris = grid(scale, jitter, 5)
    if flip:
        tris = tris[:, ::-1]
    s = lf.HostScene()
    v = np.zeros((3 * len(tris), 4), np.float32)
    v[:, :3] = tris.reshape(-1, 3)
    nrm = np.tile(np.array([[0, 0, 1, 0]], np.float32), (len(v), 1))
    mid = s.add_mesh(v, nrm)
    s.add_instance(mid, np.eye(4, dtype=np.float32).ravel(), s.add_material(np.zeros(28, np.float32)))
    s.set_camera([0, 0, 2], [0, 0, 0], 45.0)
    s.build()
    r = np.random.default_rng(9)
    w = r.random((6000, 3)).astype(np.float32)
    w[::3, 2] = 0                                   # on edges
    w[1::9] = [1, 0, 0]                             # at vertices
    w[4::9, 0] = -np.float32(1e-7)                  # just outside
    w /= w.sum(1, keepdims=True)
    t = tris[r.integers(len(tris), size=len(w))]
    at = (w[:, :, None] * t).sum(1)
    d = r.standard_normal((len(w), 3)).astype(np.float32)
    d[::5] = [0.0, 1e-3, -1.0]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros((len(w), 8), np.float32)
    dist = np.float32(scale) * np.float32(1.5)
    rays[:, 0:3], rays[:, 4:7], rays[:, 7] = at - d * dist, d, 1.0e6
    rays[::7, 7] = dist                             # limits at the hit itself
    with lf.Context(0) as ctx:
        ds = ctx.upload(s)
        ds.set_culling(-1.0)
        ref, _ = oracle.trace_closest(s.view(), rays)
        assert ctx.trace_closest(ds, rays).tobytes() == ref.tobytes()
        occ, _ = oracle.trace_any(s.view(), rays)
        assert np.array_equal(ctx.trace_any(ds, rays), occ)
        ds.close()
