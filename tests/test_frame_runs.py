"""Frame runs on the idle engine pool at the sizes and depths where their form changes (one launch,
kernel by kernel, drained after a bounce, split into passes and tiles), against the per-batch
pipeline: radiance, accumulation and ray counts bit for bit."""
import numpy as np
import pytest

import lavaframe_gb300 as lf

pytestmark = pytest.mark.gpu


def render(ctx, ds, p, spp, flags, batch=0, first=0):
    f = lf.Frame(ctx, ds, p, flags | lf.FRAME_FP64_ACCUM)
    if batch:
        f.set_batch(batch)
    f.render(first, spp)
    f.render(first + spp, 1)
    f.sync()
    out = [f.accum(), f.accum64(), np.array(f.counters())]
    if not p.tile_width:
        out.append(f.paths(1))
    f.close()
    return out


SCENES = {"cornell": lambda: lf.HostScene().gen_cornell(64, 64), "spheres": lambda: lf.HostScene().gen_icospheres(4, 3, 5, 64, 32)}


@pytest.mark.parametrize("scene", list(SCENES))
@pytest.mark.parametrize("size,spp,depth,tile,batch,flags", [
    ((1, 1), 1, 4, 0, 0, 0),
    ((33, 7), 3, 3, 0, 2, 0),          # one launch over two passes
    ((251, 67), 2, 5, 0, 0, 0),        # one launch, chunks that do not divide
    ((512, 256), 1, 4, 0, 0, 0),       # the largest one-launch run
    ((513, 256), 1, 4, 0, 0, 0),       # the smallest run in steps
    ((300, 120), 4, 1, 0, 0, 0),       # a single bounce
    ((300, 120), 4, 20, 0, 0, 0),      # deeper than the bounces in steps
    ((300, 120), 5, 20, 0, 0, 0),
    ((300, 120), 5, 5, 0, 3, 0),       # passes in steps
    ((300, 120), 5, 6, (64, 50), 2, 0),
    ((300, 120), 5, 6, (64, 50), 2, lf.FRAME_TILED_FRAMES),
    ((90, 60), 2, 6, (32, 32), 0, lf.FRAME_TILED_FRAMES),
    ((90, 60), 2, 0, (32, 32), 0, 0),  # depth 0
])
def test_runs_equal_the_per_batch_pipeline(scene, size, spp, depth, tile, batch, flags):
    with lf.Context(0) as ctx:
        s = SCENES[scene]().build()
        p = s.render_params()
        p.width, p.height = size
        p.max_depth = depth
        if tile:
            p.tile_width, p.tile_height = tile
        ds = ctx.upload(s)
        want = render(ctx, ds, p, spp, flags | lf.FRAME_PER_BATCH, batch)
        got = render(ctx, ds, p, spp, flags, batch)
        ctx.set_engine_drain(1)        # neither the one-launch form nor an early drain
        steps = render(ctx, ds, p, spp, flags, batch)
        ds.close()
    for a, b, c in zip(want, got, steps):
        assert a.tobytes() == b.tobytes()
        assert a.tobytes() == c.tobytes()
