"""Instances with an identity transform and a mesh of their own are merged into the instance
level of the wide tree at upload: hits, instance ids, ties and occlusion stay those of the
oracle's two-level traversal, whatever mix of merged and entered instances a scene has and
however an update changes it."""
import numpy as np
import pytest

import lavaframe_gb300 as lf
import oracle

pytestmark = pytest.mark.gpu


def scene(meshes, tris, moved, shared, seed):
    """`meshes` random meshes of `tris` triangles in the unit cube; every `moved`-th instance has a
    rotation, and with `shared` every mesh also has a second, identity instance."""
    r = np.random.default_rng(seed)
    s = lf.HostScene()
    mat = s.add_material(np.zeros(28, np.float32))
    eye = np.eye(4, dtype=np.float32)
    for i in range(meshes):
        c = r.random(3)
        v = np.zeros((3 * tris, 4), np.float32)
        v[:, :3] = c + 0.2 * r.standard_normal((3 * tris, 3))
        mid = s.add_mesh(v, np.tile(np.array([[0, 0, 1, 0]], np.float32), (3 * tris, 1)))
        xf = eye.copy()
        if moved and i % moved == 0:
            a = 0.3 + 0.1 * i
            xf[0, 0], xf[0, 2], xf[2, 0], xf[2, 2] = np.cos(a), -np.sin(a), np.sin(a), np.cos(a)
            xf[3, :3] = 0.1
        s.add_instance(mid, xf.ravel(), mat)
        if shared:
            s.add_instance(mid, eye.ravel(), mat)
    s.set_camera([0.5, 0.5, 4.0], [0.5, 0.5, 0.0], 45.0)
    return s.build()


def rays(n, seed):
    """Random rays, and rays whose origin or direction has zeros of either sign or values that are
    not finite."""
    out = lf.gen_rays([-1, -1, -1], [2, 2, 2], n, seed)
    out[0:40:4, 0:3] = -0.0
    out[1:40:4, 0] = -0.0
    out[2:40:4, 4] = 0.0
    out[3:40:4, 5] = -0.0
    out[40, 0], out[41, 1], out[42, 2], out[43, 0] = np.inf, -np.inf, np.nan, 2.0e38
    return out


def check(ctx, ds, s, seed):
    q = rays(4096, seed)
    ref, _ = oracle.trace_closest(s.view(), q)
    assert ctx.trace_closest(ds, q).tobytes() == ref.tobytes()
    occ, _ = oracle.trace_any(s.view(), q)
    assert np.array_equal(ctx.trace_any(ds, q), occ)


@pytest.mark.parametrize("meshes,tris,moved,shared", [(1, 1, 0, False), (1, 3, 0, False), (1, 40, 0, False),
                                                      (2, 4, 0, False), (37, 1, 0, False), (64, 10, 0, False),
                                                      (64, 10, 3, False), (33, 9, 1, False), (16, 7, 2, True)])
def test_merged_instances_equal_the_oracle(meshes, tris, moved, shared):
    with lf.Context(0) as ctx:
        s = scene(meshes, tris, moved, shared, 11)
        ds = ctx.upload(s)
        check(ctx, ds, s, 3)
        ds.close()


def test_updates_between_merged_and_entered_instances():
    """Moving instances off and back onto the identity changes which meshes are merged (and the
    size of the wide tree)."""
    with lf.Context(0) as ctx:
        s = scene(48, 11, 0, False, 5)
        ds = ctx.upload(s)
        eye = np.eye(4, dtype=np.float32)
        _, _, mats = s.layout()
        for shift in (0.25, 0.0, 0.5):
            for i in range(0, 48, 1 if shift == 0.25 else 2):
                xf = eye.copy()
                xf[3, 0] = shift
                s.set_instance(i, xf.ravel(), int(mats[i]))
            s.rebuild_instances()
            ds.update_instances(s)
            check(ctx, ds, s, 7)
        ds.close()
