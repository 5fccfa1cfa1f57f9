"""Host code of the library when allocations or launches fail and while copies are still waiting, on
a CUDA runtime in host memory (tests/fake_cuda.cpp)."""
import ctypes as C

import numpy as np
import pytest

import lavaframe_gb300 as lf
from tests import shared_meshes
from tests.fakecuda import HOOK, PINNED, POOL, fake, fake_lib  # noqa: F401 (fixtures)


def _frame(ctx, width=16, height=8, batch=2):
    scene = ctx.upload(lf.HostScene().gen_cornell(width, height).build())
    p = lf.HostScene().gen_cornell(width, height).build().render_params()
    f = lf.Frame(ctx, scene, p)
    f.set_batch(batch)
    return scene, f


def test_no_room_for_the_last_pass(fake):  # noqa: F811
    """A run of several passes keeps the last one's radiance: without memory for a copy of it the frame
    holds on to the whole run's, and frees it once."""
    with lf.Context(0) as ctx:
        scene, f = _frame(ctx)
        f.render(0, 5)            # makes the engine
        fake.fake_fail_alloc(1)   # after the run's radiance
        f.render(5, 5)
        assert f.paths(1).shape[1:] == (8, 16, 3)
        f.render(10, 5)
        assert fake.fake_block(16 * 8 * 16, 1)
        f.close()
        assert fake.fake_bad_frees() == 0 and fake.fake_pool_blocks(0) == 0
        scene.close()


def test_no_copy_from_memory_that_is_gone(fake):  # noqa: F811
    """A render of several passes returns before its work has run: what its copies still have to read is
    page-locked memory of the engine, which is written again only after they have."""
    with lf.Context(0) as ctx:
        scene, f = _frame(ctx)
        f.render(0, 5)
        assert fake.fake_pending() > 0 and fake.fake_pending_pageable() == 0
        f.render(5, 5)
        assert fake.fake_changed_sources() == 0
        f.close()
        scene.close()


@pytest.mark.parametrize("by", [0, 4, 8, 12, 16])
def test_device_samples_reach_the_kernel_aligned(fake, by):  # noqa: F811
    """The tcgen05 training kernel loads its records 16 bytes at a time; a device pointer may be aligned
    for floats only."""
    n, seen = 200, []
    want = np.arange(n * 16, dtype=np.float32)

    def launched(name, args):
        if b"guide_train_tc_kernel" in name:
            fake.fake_flush()
            seen.append((args[1][0] % 16, bytes((C.c_char * want.nbytes).from_address(args[1][0])) == want.tobytes()))

    with lf.Context(0) as ctx:
        g = lf.Guide(ctx, [0, 0, 0], [1, 1, 1], seed=3)
        d = C.c_void_p()
        ctx._c(fake.lf_device_alloc(ctx.h, want.nbytes + 16, C.byref(d)))
        C.memmove(d.value + by, want.ctypes.data, want.nbytes)
        hook = HOOK(launched)
        fake.fake_hook(hook)
        ctx._c(fake.lf_guide_train_device(g.h, C.c_void_p(d.value + by), n, 1e-2))
        fake.fake_hook(HOOK())
        assert seen == [(0, True)]
        ctx._c(fake.lf_device_free(ctx.h, d))
        g.close()


@pytest.mark.parametrize("kind", shared_meshes.KINDS)
def test_meshes_that_share_nodes_are_accepted(fake, kind):  # noqa: F811
    """A mesh may be a part of another one's tree."""
    with lf.Context(0) as ctx:
        shared_meshes.upload(ctx, shared_meshes.View(kind)).close()


def test_noalloc_reports_its_own_errors(fake):  # noqa: F811
    """A render without allocation whose launch fails returns once its earlier passes are done, and their
    error bits are not the next call's."""
    p = lf.HostScene().gen_cornell(64, 32).build().render_params()
    p.tile_width, p.tile_height = 32, 32
    with lf.Context(0) as ctx:
        scene = ctx.upload(lf.HostScene().gen_cornell(64, 32).build())
        d = C.c_void_p()
        ctx._c(fake.lf_device_alloc(ctx.h, 64 * 32 * 16, C.byref(d)))
        status = C.cast(fake.fake_block(8, PINNED), C.POINTER(C.c_uint32))

        def launched(name, args):
            if b"engine_direct_kernel" in name:
                status[1] = 1

        hook = HOOK(launched)
        fake.fake_hook(hook)
        assert fake.lf_render_noalloc(scene.h, C.byref(p), 0, 1, d) == 4   # the bit is reported
        assert fake.lf_render_noalloc(scene.h, C.byref(p), 0, 1, d) == 4 and status[1] == 0
        fake.fake_fail_launch(2)   # the second tile's first kernel
        assert fake.lf_render_noalloc(scene.h, C.byref(p), 0, 1, d) == 2
        assert fake.fake_pending() == 0
        fake.fake_hook(HOOK())
        assert fake.lf_render_noalloc(scene.h, C.byref(p), 0, 1, d) == 0
        assert ctx.device_errors() == 1
        ctx._c(fake.lf_device_free(ctx.h, d))
        scene.close()


def test_a_failed_allocation_is_reported_once(fake):  # noqa: F811
    with lf.Context(0) as ctx:
        scene, f = _frame(ctx)
        f.render(0, 1)
        fake.fake_fail_alloc(0)
        with pytest.raises(lf.LFError) as err:
            f.render(0, 1)
        assert err.value.status == 3
        f.render(0, 1)   # its launches do not find the earlier call's error
        f.close()
        scene.close()


@pytest.mark.parametrize("width,height", [(13, 7), (256, 256), (256, 257)])   # 2^16 pixels are one piece
def test_readback_without_device_memory(fake, width, height):  # noqa: F811
    """A rendered image can be read when nothing is left to allocate on the device."""
    n = width * height
    a = np.arange(4 * n, dtype=np.float32)
    with lf.Context(0) as ctx:
        scene, f = _frame(ctx, width, height)
        ctx.sync()
        C.memmove(fake.fake_block(16 * n, POOL), a.ctypes.data, a.nbytes)
        fake.fake_fail_alloc(0)
        assert np.array_equal(f.accum().reshape(-1, 3), a.reshape(-1, 4)[:, :3])
        f.close()
        scene.close()


def test_the_default_memory_pool_is_left_alone(fake):  # noqa: F811
    """Contexts of a device share a pool of the library's own, which goes with the last of them."""
    with lf.Context(0) as a, lf.Context(0) as b:
        for ctx in (a, b):
            scene, f = _frame(ctx)
            f.render(0, 5)
            f.accum()
            assert fake.fake_pool_blocks(0) > 0 and fake.fake_pool_blocks(1) == 0
            f.close()
            scene.close()
        assert fake.fake_pools() == 1
    assert fake.fake_pools() == 0 and fake.fake_default_pool_changes() == 0


@pytest.mark.parametrize("n", [100, 20000])   # over the staging block and over copies
def test_results_beside_a_device_error(fake, n):  # noqa: F811
    """An error bit of one ray's traversal leaves the other rays' results: they are returned with the
    error, whatever way they came."""
    want = np.arange(4 * n, dtype=np.int32)
    with lf.Context(0) as ctx:
        scene, f = _frame(ctx)
        status = C.cast(fake.fake_block(8, PINNED), C.POINTER(C.c_uint32))

        def launched(name, args):
            if b"trace_fetch_wide" in name:
                fake.fake_flush()
                C.memmove(C.cast(args[4], C.POINTER(C.c_void_p))[0], want.ctypes.data, want.nbytes)
                status[0] = 1

        hook = HOOK(launched)
        fake.fake_hook(hook)
        rays, out = np.zeros((n, 8), np.float32), np.zeros((n, 4), np.int32)
        st = fake.lf_trace_closest(ctx.h, scene.h, rays.ctypes.data_as(C.POINTER(C.c_float)), n,
                                   out.ctypes.data_as(C.c_void_p), 0)
        fake.fake_hook(HOOK())
        assert st == 4 and ctx.device_errors() == 1 and out.reshape(-1).tobytes() == want.tobytes()
        f.close()
        scene.close()


@pytest.mark.parametrize("coherent", [0, 1])
@pytest.mark.parametrize("locked", [True, False])
def test_gradients_without_page_locked_memory(fake, locked, coherent):  # noqa: F811
    """The small results of a gradient call go over page-locked memory if there is some."""
    n, nW = 200, lf.GUIDE_WEIGHTS
    want = np.arange(nW + 1, dtype=np.float32)
    grid = np.arange(lf.GUIDE_GRID_PARAMS, dtype=np.float32)
    fake.fake_coherent(coherent)
    with lf.Context(0) as ctx:
        g = lf.Guide(ctx, [0, 0, 0], [1, 1, 1], seed=3)

        def launched(name, args):
            if b"guide_scale_kernel" in name:
                fake.fake_flush()
                at = [C.cast(args[k], C.POINTER(C.c_void_p))[0] for k in (4, 5, 6)]
                C.memmove(at[0], want.ctypes.data, 4 * nW)
                C.memmove(at[1], grid.ctypes.data, grid.nbytes)
                C.memmove(at[2], want.ctypes.data + 4 * nW, 4)

        hook = HOOK(launched)
        fake.fake_hook(hook)
        if not locked:
            fake.fake_fail_alloc_kind(PINNED)
        loss, dw, dg = g.gradients(np.zeros((n, 16), np.float32))
        fake.fake_hook(HOOK())
        assert dw.tobytes() == want[:nW].tobytes() and dg.tobytes() == grid.tobytes() and loss == nW
        g.close()
