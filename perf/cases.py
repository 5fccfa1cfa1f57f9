"""Workloads whose speed is measured, through the public entry points of lavaframe_gb300.

A case is a dict of plain values; `listed()` has the fixed ones, `draw(rng)` gives more of the
same ranges, `prepare` makes what a program has in hand before the call, `run` is one pass,
`work` the bytes and operations a pass cannot do without, and `exact` the results in 64 bits
where they can be had from plain torch or numpy.

Scenes are the procedural ones of the library (the Cornell box, the triangle soup, the
displaced icospheres under an HDR sky, the furnished room). A program builds and uploads its
scene once and then works on it, so built scenes are kept between states here as well; rays,
queries, training samples, network parameters and the seeds of the renders are made from the
seed.
"""
import collections
import ctypes
import math

import numpy as np
import torch

import lavaframe_gb300 as lf


def listed():
    return [
        # picking and probe rays of an editor: a thousand rays from host memory, latency only
        {"name": "pick_1k", "kind": "closest", "scene": "room", "size": 500, "rays": 1000, "host": True, "tmax": 1.0e6},
        # occlusion baking: rays of limited length against a furnished room, from host memory
        {"name": "bake_occlusion_300k", "kind": "any", "scene": "room", "size": 4000, "rays": 300007, "host": True, "tmax": 1.5},
        # the intersection microbench (random rays, random triangles), rays and hits on the GPU
        {"name": "soup_closest_4m", "kind": "closest", "scene": "soup", "size": 131072, "rays": 1 << 22, "host": False,
         "tmax": 1.0e6},
        # one refinement step of an interactive view: a sample per pixel, then the display pass
        {"name": "preview_1spp", "kind": "preview", "scene": "cornell", "size": 1, "width": 333, "height": 187, "depth": 4,
         "tonemap": 2},
        # the Cornell box as it is rendered in the benchmark: 256 x 256, 64 samples, depth 4
        {"name": "cornell_64spp", "kind": "frame", "scene": "cornell", "size": 1, "width": 256, "height": 256, "spp": 64,
         "depth": 4, "tile": 0, "fp64": False},
        # the production frame of the benchmark: a million triangles, HDR sky, full HD, 16 samples
        {"name": "spheres_1080p", "kind": "frame", "scene": "spheres", "size": 13, "width": 1920, "height": 1080, "spp": 16,
         "depth": 8, "tile": 0, "fp64": False},
        # a real-time loop that may not allocate: a few samples into the caller's device buffer
        {"name": "noalloc_4spp", "kind": "noalloc", "scene": "cornell", "size": 4, "width": 320, "height": 200, "spp": 4,
         "depth": 4},
        # guided rendering with a trained network held fixed: deep paths in the occluded room
        {"name": "guided_room", "kind": "guided", "scene": "room", "size": 4000, "width": 640, "height": 360, "spp": 8,
         "depth": 10},
        # the guide's mixtures and densities for a batch of queries
        {"name": "guide_eval_100k", "kind": "guide_eval", "queries": 100000},
        # the guide's gradients for the batch size that guided rendering trains with
        {"name": "guide_gradients_16k", "kind": "guide_gradients", "samples": 16384},
        # the display pass of a full HD frame, read back as bytes and floats
        {"name": "display_1080p", "kind": "display", "width": 1920, "height": 1080, "tonemap": 4},
        # a render service: jobs of different scenes, sizes and sample counts in one batch
        {"name": "serve_8_jobs", "kind": "serve", "jobs": 8, "edge": 256, "spp": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["closest", "closest", "any", "frame", "frame", "preview", "noalloc", "guided", "guide_eval",
                       "guide_gradients", "display", "serve"])
    scene = rng.choice(["cornell", "soup", "spheres", "room"])
    size = {"cornell": _log(rng, 1, 64), "soup": _log(rng, 1000, 131072), "spheres": rng.randint(2, 13),
            "room": _log(rng, 50, 8000)}[scene]
    if kind in ("closest", "any"):
        host = rng.random() < 0.5
        return {"kind": kind, "scene": scene, "size": size, "rays": _log(rng, 100, 1 << (20 if host else 22)), "host": host,
                "tmax": 1.0e6 if kind == "closest" else rng.choice([1.5, 10.0, 1.0e6])}
    if kind == "frame":
        width, height = _log(rng, 48, 1280), _log(rng, 32, 720)
        most = max(1, 16_000_000 // (width * height))
        return {"kind": kind, "scene": scene, "size": size, "width": width, "height": height,
                "spp": _log(rng, 1, min(64, most)), "depth": rng.randint(2, 8), "tile": rng.choice([0, 0, 64, 100]),
                "fp64": rng.random() < 0.3}
    if kind == "preview":
        return {"kind": kind, "scene": scene, "size": size, "width": _log(rng, 64, 960), "height": _log(rng, 48, 540),
                "depth": rng.randint(2, 6), "tonemap": rng.randint(0, 6)}
    if kind == "noalloc":
        return {"kind": kind, "scene": scene, "size": size, "width": _log(rng, 32, 400), "height": _log(rng, 32, 300),
                "spp": _log(rng, 1, 16), "depth": rng.randint(2, 6)}
    if kind == "guided":
        return {"kind": kind, "scene": "room", "size": _log(rng, 50, 8000), "width": _log(rng, 96, 640),
                "height": _log(rng, 64, 360), "spp": rng.randint(1, 8), "depth": rng.randint(3, 10)}
    if kind == "guide_eval":
        return {"kind": kind, "queries": _log(rng, 100, 300000)}
    if kind == "guide_gradients":
        return {"kind": kind, "samples": _log(rng, 100, 65536)}
    if kind == "display":
        return {"kind": kind, "width": _log(rng, 64, 1920), "height": _log(rng, 48, 1080), "tonemap": rng.randint(0, 6)}
    return {"kind": "serve", "jobs": rng.randint(2, 12), "edge": _log(rng, 48, 320), "spp": _log(rng, 1, 16)}


# ------------------------------------------------------------------ scenes and handles
class _Scene:
    """A built host scene and its device copy, released with the last state that uses it."""

    def __init__(self, ctx, host):
        self.ctx, self.host = ctx, host
        self.dev = ctx.upload(host)
        v = host.view()
        nodes = np.ctypeslib.as_array(v.nodes, shape=(v.num_nodes * 9,)).reshape(-1, 9)
        root = nodes[v.top_level_index]
        self.lo, self.hi, self.triangles = root[0:3].copy(), root[3:6].copy(), int(v.num_tris)

    def __del__(self):
        self.dev.close()


class _State:
    """Handles of one case's state; closed in reverse order when the state goes."""

    def __init__(self, case):
        self.case, self.handles = case, []

    def own(self, h):
        self.handles.append(h)
        return h

    def __del__(self):
        while self.handles:
            self.handles.pop().close()


_CONTEXT = None
_SCENES = collections.OrderedDict()
_SCENES_KEPT = 4


def _context():
    """The program's context; one for all states, as a user's program has it."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = lf.Context(0)
    return _CONTEXT


def _generate(kind, size):
    h = lf.HostScene()
    if kind == "cornell":
        h.gen_cornell(256, 256, size)
    elif kind == "soup":
        h.gen_soup(size, 10, 1)
    elif kind == "spheres":
        h.gen_icospheres(size, 6, 3, 1024, 512)
    else:
        h.gen_room(size, 4)
    return h.build()


def _scene(kind, size):
    key = (kind, size)
    if key not in _SCENES:
        _SCENES[key] = _Scene(_context(), _generate(kind, size))
        while len(_SCENES) > _SCENES_KEPT:
            _SCENES.popitem(last=False)
    _SCENES.move_to_end(key)
    return _SCENES[key]


def _params(scene, case, seed):
    p = scene.host.render_params()
    p.width, p.height, p.max_depth = case["width"], case["height"], case["depth"]
    p.seed = seed & 0x7FFFFFFF
    return p


def _rays(scene, n, tmax, seed):
    """Origins uniform in the scene's box, directions uniform on the sphere."""
    r = np.random.default_rng(seed)
    out = np.empty((n, 8), np.float32)
    out[:, 0:3] = scene.lo + (scene.hi - scene.lo) * r.random((n, 3), np.float32)
    out[:, 3] = 0.0
    d = r.standard_normal((n, 3), np.float32)
    out[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    out[:, 7] = tmax
    return out


def _unit(r, n):
    d = r.standard_normal((n, 3), np.float32)
    return d / np.linalg.norm(d, axis=1, keepdims=True)


_BOX = (np.array([-1.0, 0.0, -2.0], np.float32), np.array([3.0, 2.0, 2.0], np.float32))


def _guide_params(seed):
    """Weights and grid tables of a trained network's magnitude, all FP16 values."""
    r = np.random.default_rng(seed)
    w = np.concatenate([r.uniform(-1, 1, n).astype(np.float32) * s for n, s in
                        ((3 * 4096, 0.22), (48 * 64, 0.25))])
    w[3 * 4096 + 40 * 64:] = 0.0
    g = r.uniform(-0.5, 0.5, 8 * 16384 * 4).astype(np.float32)
    return w.astype(np.float16).astype(np.float32), g.astype(np.float16).astype(np.float32)


def _guide_records(n, seed):
    """Shading points on a few planes of the box, outgoing directions, normals, sampled
    directions and sample weights (luminance over pdf)."""
    r = np.random.default_rng(seed + 1)
    lo, hi = _BOX
    out = np.zeros((n, 16), np.float32)
    out[:, 0:3] = lo + (hi - lo) * r.random((n, 3), np.float32)
    out[: n // 2, 1] = lo[1]
    out[:, 3:6] = _unit(r, n)
    out[:, 6:9] = _unit(r, n)
    out[:, 9:12] = _unit(r, n)
    out[:, 12] = np.exp(r.standard_normal(n, np.float32))
    return out


# ------------------------------------------------------------------ states
def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    s = _State(case)
    s.ctx = ctx
    if kind in ("closest", "any"):
        s.scene = _scene(case["scene"], case["size"])
        rays = _rays(s.scene, case["rays"], case["tmax"], seed)
        if case["host"]:
            s.rays = rays
        else:
            s.rays = torch.from_numpy(rays).cuda()
            s.out = torch.empty((case["rays"], 4) if kind == "closest" else (case["rays"],),
                                dtype=torch.int32 if kind == "closest" else torch.uint8, device="cuda")
            torch.cuda.synchronize()
    elif kind in ("frame", "preview", "guided"):
        s.scene = _scene(case["scene"], case["size"])
        p = _params(s.scene, case, seed)
        if case.get("tile"):
            p.tile_width = p.tile_height = case["tile"]
        if kind == "guided":
            g = s.own(lf.Guide(ctx, s.scene.lo, s.scene.hi, seed=1))
            g.set_params(*_guide_params(7))
        s.frame = s.own(lf.Frame(ctx, s.scene.dev, p, lf.FRAME_FP64_ACCUM if case.get("fp64") else 0))
        if kind == "guided":
            s.frame.set_batch(case["spp"])
            s.frame.set_guide(g, 0.5, 0)
        elif kind == "preview":
            s.post = lf.PostParams.defaults(case["tonemap"])
    elif kind == "noalloc":
        s.scene = _scene(case["scene"], case["size"])
        s.params = _params(s.scene, case, seed)
        s.accum = torch.zeros((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
    elif kind in ("guide_eval", "guide_gradients"):
        s.guide = s.own(lf.Guide(ctx, *_BOX, seed=1))
        s.guide.set_params(*_guide_params(seed))
        s.records = _guide_records(case["queries" if kind == "guide_eval" else "samples"], seed)
    elif kind == "display":
        s.scene = _scene("cornell", 1)
        p = _params(s.scene, dict(case, depth=4), seed)
        s.frame = s.own(lf.Frame(ctx, s.scene.dev, p))
        s.frame.render(0, 4)
        s.frame.sync()
        s.post = lf.PostParams.defaults(case["tonemap"])
    else:
        r = np.random.default_rng(seed)
        pool = [_scene("cornell", 16), _scene("room", 400), _scene("spheres", 2)]
        s.ctx = s.own(lf.Context(0))   # a server owns the engine of its context
        s.server = s.own(lf.Server(s.ctx))
        ids = [s.server.add_scene(sc.host) for sc in pool]
        s.scenes, s.jobs = pool, []
        for j in range(case["jobs"]):
            which = j % len(pool)
            e = case["edge"] >> (j & 1)
            p = _params(pool[which], {"width": e + 8 * (j % 3), "height": max(16, e - 5 * (j % 4)), "depth": 4 + j % 4},
                        int(r.integers(1 << 30)))
            s.jobs.append((ids[which], p, max(1, case["spp"] >> (j % 3))))
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind in ("closest", "any"):
        if not case["host"]:
            call = lf.lib().lf_trace_closest_device if kind == "closest" else lf.lib().lf_trace_any_device
            s.ctx._c(call(s.ctx.h, s.scene.dev.h, s.rays.data_ptr(), case["rays"], s.out.data_ptr(), 0))
            return {"t": s.out.view(torch.float32)[:, 0], "ids": s.out[:, 1:]} if kind == "closest" else s.out
        if kind == "any":
            return s.ctx.trace_any(s.scene.dev, s.rays)
        hits = s.ctx.trace_closest(s.scene.dev, s.rays)
        return {"t": hits["t"], "ids": [hits["instance"], hits["prim"], hits["light"]]}
    if kind in ("frame", "guided"):
        s.frame.reset()
        s.frame.render(0, case["spp"])
        out = {"sum": s.frame.accum()}
        if case.get("fp64"):
            out["sum64"] = s.frame.accum64()
        return out
    if kind == "preview":
        s.frame.reset()
        s.frame.render(0, 1)
        return list(s.frame.postprocess(1, s.post))
    if kind == "noalloc":
        s.accum.zero_()
        torch.cuda.current_stream().synchronize()
        s.ctx._c(lf.lib().lf_render_noalloc(s.scene.dev.h, ctypes.byref(s.params), 0, case["spp"], s.accum.data_ptr()))
        return s.accum
    if kind == "guide_eval":
        return list(s.guide.eval(s.records))
    if kind == "guide_gradients":
        return list(s.guide.gradients(s.records))
    if kind == "display":
        return list(s.frame.postprocess(4, s.post))
    jobs = [s.server.submit(sid, p, spp) for sid, p, spp in s.jobs]
    out = []
    for j in jobs:
        s.server.wait(j)
        out.append(s.server.read(j))
        s.server.release(j)
    return out


# ------------------------------------------------------------------ work
# Floating-point operations of one ray against n triangles: a four-wide tree of log4(n) levels
# (four slab tests of 15 operations each) and a handful of triangle tests of 45.
def _ray_flops(triangles):
    return 60.0 * max(1.0, math.log(max(2, triangles), 4)) + 4 * 45.0


_TRIANGLES = {"cornell": lambda n: 34 * n * n, "soup": lambda n: 10 * n, "spheres": lambda n: 81920 * n,
              "room": lambda n: 12 * n + 40}
_MLP_FLOPS = 2.0 * (3 * 64 * 64 + 48 * 64)


def work(case):
    kind = case["kind"]
    tri = _TRIANGLES[case["scene"]](case["size"]) if "scene" in case else 0
    if kind in ("closest", "any"):
        return {"bytes": case["rays"] * (48 if kind == "closest" else 33), "flops": case["rays"] * _ray_flops(tri)}
    if kind in ("frame", "preview", "noalloc", "guided"):
        pixels, spp = case["width"] * case["height"], case.get("spp", 1)
        out = 16 if kind == "noalloc" else 15 if kind == "preview" else 12 + (24 if case.get("fp64") else 0)
        # an extension ray and a next-event ray per vertex, 600 operations of shading
        per_vertex = 2 * _ray_flops(tri) + 600 + (_MLP_FLOPS if kind == "guided" else 0)
        return {"bytes": pixels * out, "flops": pixels * spp * max(1, case["depth"] - 1) * per_vertex}
    if kind == "guide_eval":
        return {"bytes": case["queries"] * (9 * 4 + 4 * 41), "flops": case["queries"] * _MLP_FLOPS}
    if kind == "guide_gradients":
        return {"bytes": case["samples"] * 13 * 4 + 6 * (15360 + 8 * 16384 * 4), "flops": 3 * case["samples"] * _MLP_FLOPS}
    if kind == "display":
        return {"bytes": case["width"] * case["height"] * (16 + 15), "flops": case["width"] * case["height"] * 150}
    paths = sum(((case["edge"] >> (j & 1)) + 8 * (j % 3)) * max(16, (case["edge"] >> (j & 1)) - 5 * (j % 4)) *
                max(1, case["spp"] >> (j % 3)) for j in range(case["jobs"]))
    return {"bytes": 12.0 * paths / max(1, case["spp"]), "flops": paths * 4 * (2 * _ray_flops(20000) + 600)}


# ------------------------------------------------------------------ results in 64 bits
def _exact_closest(case, seed):
    """Every ray against every triangle (all instances of these scenes have identity transforms)."""
    scene = _scene(case["scene"], case["size"])
    a = scene.host.arrays()
    v = torch.from_numpy(a["vertices"][:, 0:3].astype(np.float64)).cuda()
    i = torch.from_numpy(a["vert_indices"].astype(np.int64)).cuda()
    v0, e0, e1 = v[i[:, 0]], v[i[:, 1]] - v[i[:, 0]], v[i[:, 2]] - v[i[:, 0]]
    rays = torch.from_numpy(_rays(scene, case["rays"], case["tmax"], seed)).cuda().double()
    best = torch.empty(case["rays"], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 24) // len(i))
    for k in range(0, case["rays"], step):
        o, d, far = rays[k:k + step, None, 0:3], rays[k:k + step, None, 4:7], rays[k:k + step, 7]
        p = torch.linalg.cross(d, e1[None], dim=-1)
        det = (e0[None] * p).sum(-1)
        t0 = o - v0[None]
        q = torch.linalg.cross(t0, e0[None].expand_as(t0), dim=-1)
        u, w, t = (t0 * p).sum(-1) / det, (d * q).sum(-1) / det, (e1[None] * q).sum(-1) / det
        ok = (u >= 0) & (w >= 0) & (t >= 0) & (u + w <= 1)
        t = torch.where(ok, t, torch.full_like(t, math.inf)).amin(1)
        best[k:k + step] = torch.minimum(t, far)
    return {"t": best, "ids": None if not case["host"] else [None, None, None]}


def _exact_network(w, g, rec):
    """Outputs (n, 40) of the guide's network in 64 bits, differentiable in w and g."""
    lo, hi = (torch.from_numpy(b).cuda().double() for b in _BOX)
    p01 = ((rec[:, 0:3] - lo) / (hi - lo)).clamp(0, 1)
    growth = math.exp((math.log(512.0) - math.log(16.0)) / 7)
    tables, feats = g.reshape(8, 16384, 4), []
    for level in range(8):
        res = math.floor(16.0 * growth ** level)
        pos = p01 * res
        i0 = pos.floor().long().clamp(max=res - 1)
        fr = pos - i0
        acc = 0
        for c in range(8):
            at = [i0[:, k] + ((c >> k) & 1) for k in range(3)]
            wt = 1
            for k in range(3):
                wt = wt * (fr[:, k] if (c >> k) & 1 else 1 - fr[:, k])
            if (res + 1) ** 3 <= 16384:
                idx = at[0] + at[1] * (res + 1) + at[2] * (res + 1) ** 2
            else:
                idx = (at[0] ^ (at[1] * 2654435761) ^ (at[2] * 805459861)) & 16383
            acc = acc + wt[:, None] * tables[level][idx]
        feats.append(acc)
    bins = (torch.arange(8, device="cuda", dtype=torch.float64) + 0.5) / 8
    for k in (3, 6):
        d = rec[:, k:k + 3]
        for a in (torch.arccos(d[:, 2].clamp(-1, 1)) / math.pi, (torch.atan2(d[:, 1], d[:, 0]) + math.pi) / (2 * math.pi)):
            feats.append(torch.exp(-0.5 * ((a[:, None] - bins) * 8) ** 2))
    h = torch.cat(feats, 1)
    for layer in range(3):
        h = torch.relu(h @ w[4096 * layer:4096 * (layer + 1)].reshape(64, 64).T)
    return (h @ w[3 * 4096:].reshape(48, 64).T)[:, :40].reshape(-1, 8, 5)


def _density(mu, kappa, share, d):
    cos = (mu * d[:, None, :]).sum(-1)
    f = kappa / (2 * math.pi * (1 - torch.exp(-2 * kappa))) * torch.exp(kappa * (cos - 1))
    return (share * f).sum(1)


def _exact_guide(case, seed):
    w, g = (torch.from_numpy(a).cuda().double() for a in _guide_params(seed))
    n = case["queries"] if case["kind"] == "guide_eval" else case["samples"]
    rec = torch.from_numpy(_guide_records(n, seed)).cuda().double()
    if case["kind"] == "guide_eval":
        mixes, pdfs = [], []
        for part in rec.split(1 << 16):
            o = _exact_network(w, g, part)
            mu = o[..., 0:3] / o[..., 0:3].norm(dim=-1, keepdim=True)
            kappa, share = torch.exp(o[..., 3].clamp(-3, 7)), torch.softmax(o[..., 4], 1)
            mixes.append(torch.cat([mu, kappa[..., None], share.cumsum(1)[..., None]], -1).reshape(-1, 40))
            pdfs.append(_density(mu, kappa, share, part[:, 9:12]))
        return [torch.cat(mixes), torch.cat(pdfs)]
    w.requires_grad_(True)
    g.requires_grad_(True)
    total = 0.0
    for part in rec.split(1 << 14):
        o = _exact_network(w, g, part)
        raw = o[..., 0:3]
        mu = raw / torch.sqrt((raw * raw).sum(-1, keepdim=True) + 1e-6)
        q = _density(mu, torch.exp(o[..., 3].clamp(-3, 7)), torch.softmax(o[..., 4], 1), part[:, 9:12])
        loss = (-part[:, 12] * torch.log(q + 1e-12)).sum() / n
        loss.backward()
        total += float(loss.detach())
    return [total, w.grad, g.grad]


def _exact_tonemap(mode, c):
    gamma = 1 / 2.2
    if mode == 1:
        return (c / (1 + (c @ np.array([0.3, 0.6, 0.1]))[..., None] / 2)) ** gamma
    if mode == 2:
        return np.clip(c * (2.51 * c + 0.03) / (c * (2.43 * c + 0.59) + 0.14), 0, 1) ** gamma
    if mode == 3:
        return np.clip(c / (c + 1), 0, 1) ** gamma
    if mode == 4:
        v = c * (c * (1.2295 * c + 0.3135) + 1.1935 * 0.4655) / (c * (1.1935 * c + 0.4655) + 0.073)
        return np.clip(0.8 * (v ** 1.7) ** (1 / 0.8), 0, 1) ** gamma
    if mode == 5:
        v = np.maximum(0, c - 0.004)
        return v * (6.2 * v + 0.5) / (v * (6.2 * v + 1.7) + 0.06)
    if mode == 6:
        v = (c * (0.15 * c + 0.05) + 0.004) / (c * (0.15 * c + 0.5) + 0.06) - 0.02 / 0.3
        return np.maximum(v, 0) ** gamma * 1.75
    return c


def exact(case, seed):
    kind = case["kind"]
    if kind == "closest" and case["scene"] in ("soup", "room"):
        if case["rays"] * _TRIANGLES[case["scene"]](case["size"]) > 2e10:
            return None
        return _exact_closest(case, seed)
    if kind in ("guide_eval", "guide_gradients"):
        return _exact_guide(case, seed)
    if kind == "display":
        # the mean radiance at the pixel centres is the render's own; tone map and gamma in 64 bits
        s = prepare(case, seed)
        return [None, _exact_tonemap(case["tonemap"], s.frame.accum().astype(np.float64) / 4)]
    return None
