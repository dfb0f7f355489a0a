"""What a user of the framework has it do, as timed cases.

Ray casts (the Intersectable surface), renders (the Renderer / Tracer surface,
one scene or a batch) and the radiance cache (queries and online training), each
through the public Python entry points over the C ABI.  Scenes and sizes are
those of the repository's own generators, tests and benchmark configurations:
the triangle soup and its ray sets, the Cornell box, the production scene
(terrain and GGX / Lambert spheres under a sun and an environment) and the
multi-scene batch.

listed() are the cases that are always timed, draw() one more from the same
ranges; prepare() makes what a user's program holds before the call, run() is
the call, work() what it cannot do without, exact() its result in 64 bits where
plain torch can say it.
"""
import math

import numpy as np
import torch

from banshee_b200 import abi, capi, scenes

_CTX = None


def _ctx():
    """One context per process, as every user's program keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = capi.Context(0)
    return _CTX


def listed():
    return [
        # Banshee's own tracer over GpuAccelerator: World::Intersect, one ray per call, host memory
        dict(name="cast_one_ray_host", kind="cast", tris=1 << 20, rays=1, coherent=False, any=False, host=True,
             width=0, watertight=False),
        # a small batch of shadow rays (a light-map texel row, a game's line-of-sight queries)
        dict(name="cast_4k_shadow", kind="cast", tris=100_000, rays=4096, coherent=False, any=True, host=False,
             width=0, watertight=False),
        # camera rays of a 1 Mpixel view into the 1M-triangle soup
        dict(name="cast_1m_camera", kind="cast", tris=1 << 20, rays=1 << 20, coherent=True, any=False, host=False,
             width=0, watertight=False),
        # the incoherent closest-hit set of the ray-cast benchmark at full size
        dict(name="cast_16m_incoherent", kind="cast", tris=1 << 20, rays=1 << 24, coherent=False, any=False,
             host=False, width=0, watertight=False),
        # shadow rays in a ragged number on the compressed 8-wide nodes
        dict(name="cast_3m_shadow_wide8", kind="cast", tris=300_007, rays=3_000_017, coherent=False, any=True,
             host=False, width=8, watertight=False),
        # one progressive sample of a small Cornell view: the smallest render, latency counts
        dict(name="render_cornell_preview", kind="render", scene="cornell", nterrain=0, nspheres=0, seg=0, w=64,
             h=64, spp=1, tracer="gi", depth=5, sampler="random", host=False),
        # the Cornell benchmark at full size
        dict(name="render_cornell_64spp", kind="render", scene="cornell", nterrain=0, nspheres=0, seg=0, w=256,
             h=256, spp=64, tracer="gi", depth=5, sampler="random", host=False),
        # a ragged production view in host memory, Sobol camera samples, 2 spp of a progressive render
        dict(name="render_host_sobol", kind="render", scene="production", nterrain=256, nspheres=24, seg=40, w=500,
             h=333, spp=2, tracer="gi", depth=8, sampler="sobol", host=True),
        # the 6.09M-triangle production frame, 8 samples per pixel in one call
        dict(name="render_1080p_6m", kind="render", scene="production", nterrain=1024, nspheres=200, seg=100, w=1920,
             h=1080, spp=8, tracer="gi", depth=8, sampler="random", host=False),
        # several scenes of uneven size and resolution through one set of queues
        dict(name="batch_8_scenes", kind="batch", scenes=8, tri_lo=1e4, tri_hi=2e5, spp=4, depth=8),
        # cache predictions for the ended paths of a frame
        dict(name="cache_query_200k", kind="query", rows=200_003, log2t=19),
        # four frames' online training, four Adam steps each; then predictions at held-out points and a checkpoint
        dict(name="cache_train_16x16k", kind="train", rows=16384, steps=16, log2t=19),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "cast", "cast", "render", "render", "render", "batch", "query", "train"])
    if kind == "cast":
        host = rng.random() < 0.25
        occlusion = rng.random() < 0.5
        tris = _log_int(rng, 20_000, 1 << 20)   # sparser soups are nearly empty: every ray misses
        rays = _log_int(rng, 256 if occlusion else 8, 65_536 if host else 1 << 22)
        return dict(kind="cast", tris=tris, rays=rays, coherent=rng.random() < 0.5, any=occlusion, host=host,
                    width=rng.choice([0, 0, 4, 8]), watertight=rng.random() < 0.2)
    if kind == "render":
        w, h = _log_int(rng, 32, 1024), _log_int(rng, 32, 1024)
        spp = max(1, min(_log_int(rng, 1, 64), 6_000_000 // (w * h)))
        cornell = rng.random() < 0.35
        return dict(kind="render", scene="cornell" if cornell else "production",
                    nterrain=0 if cornell else _log_int(rng, 32, 512), nspheres=0 if cornell else rng.randint(2, 40),
                    seg=0 if cornell else rng.randint(12, 64), w=w, h=h, spp=spp,
                    tracer=rng.choice(["gi", "gi", "gi", "di", "ao"]), depth=rng.randint(2, 8),
                    sampler=rng.choice(["random", "random", "sobol", "cmj"]), host=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="batch", scenes=rng.randint(2, 10), tri_lo=1e4, tri_hi=_log_int(rng, 30_000, 300_000),
                    spp=rng.randint(1, 4), depth=rng.randint(3, 8))
    if kind == "query":
        return dict(kind="query", rows=_log_int(rng, 100, 1_000_000), log2t=rng.randint(14, 19))
    return dict(kind="train", rows=_log_int(rng, 200, 65_536), steps=rng.randint(1, 16), log2t=rng.randint(14, 19))


# ---------------------------------------------------------------- ray casts
def _soup(case, seed):
    return scenes.soup(case["tris"], seed=seed)


def _rays(case, seed):
    """Rays as an (n, 8) tensor: o, tmin, d, tmax.  coherent: a jittered pinhole
    view of the unit cube, row by row; otherwise origins in the cube, directions
    uniform on the sphere.  Shadow rays end within a unit (incoherent) or inside
    the cube (coherent); closest-hit rays end behind the scene."""
    n = case["rays"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.zeros((n, 8), device="cuda")
    u = torch.rand((n, 4), generator=g, device="cuda")
    if case["coherent"]:
        side = max(1, math.isqrt(n - 1) + 1 if n > 1 else 1)
        i = torch.arange(n, device="cuda")
        half = math.tan(math.radians(45.0) / 2)
        x = ((i % side + u[:, 0]) / side * 2 - 1) * half
        y = (1 - (i // side + u[:, 1]) / side * 2) * half
        d = torch.stack([x, y, -torch.ones_like(x)], 1)
        r[:, 0:3] = torch.tensor([0.5, 0.5, 2.5], device="cuda")
        lo, hi = 1.5, 2.5
    else:
        r[:, 0:3] = u[:, 0:3]
        d = torch.randn((n, 3), generator=g, device="cuda")
        lo, hi = 0.0, 1.0
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    r[:, 7] = lo + (hi - lo) * u[:, 3] if case["any"] else 8.0
    return r


def _prepare_cast(case, seed):
    gs = capi.GpuScene(_ctx(), _soup(case, seed), node_width=case["width"], builder=3 if case["tris"] >= 50_000 else 0,
                       intersect=1 if case["watertight"] else 0)
    rays, n = _rays(case, seed), case["rays"]
    st = dict(case=case, gs=gs, n=n)
    if case["host"]:
        st["rays"] = rays.cpu().numpy().reshape(-1).view(abi.RAY_DTYPE)
        return st
    st["rays"] = rays
    if case["any"]:
        st["res"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
        st["out"] = {"occluded": st["res"]}
    else:
        st["res"] = torch.zeros((n, 4), device="cuda")
        st["out"] = {"t": st["res"][:, 0], "prim": st["res"].view(torch.int32)[:, 1], "u": st["res"][:, 2],
                     "v": st["res"][:, 3]}
    return st


def _run_cast(st):
    case, gs = st["case"], st["gs"]
    if case["host"]:
        if case["any"]:
            return {"occluded": gs.intersect_any_host(st["rays"])}
        h = gs.intersect_closest_host(st["rays"])
        return {"t": h["t"], "prim": h["primid"], "u": h["u"], "v": h["v"]}
    fn = gs.intersect_any if case["any"] else gs.intersect_closest
    fn(st["rays"].data_ptr(), st["res"].data_ptr(), st["n"])
    return st["out"]


def _exact_cast(case, seed):
    """Every ray against every triangle in 64 bits (Moller-Trumbore)."""
    if case["any"] or case["tris"] * case["rays"] > 2e10:
        return None
    m = _soup(case, seed).meshes[0]
    tv = torch.from_numpy(m.vertices.reshape(-1, 3, 3)).cuda().double()
    p, e1, e2 = tv[:, 0], tv[:, 1] - tv[:, 0], tv[:, 2] - tv[:, 0]
    rays = _rays(case, seed).double()
    n = rays.shape[0]
    t_out = rays[:, 7].clone()
    uv_out = torch.zeros((2, n), dtype=torch.float64, device="cuda")
    step = max(1, int(2e7) // p.shape[0])
    for a in range(0, n, step):
        r = rays[a:a + step]
        o, d = r[:, None, 0:3], r[:, None, 4:7]
        s1 = torch.linalg.cross(d.expand(-1, p.shape[0], -1), e2[None].expand(r.shape[0], -1, -1))
        inv = 1.0 / (s1 * e1).sum(-1)
        dd = o - p[None]
        b1 = (dd * s1).sum(-1) * inv
        s2 = torch.linalg.cross(dd, e1[None].expand(r.shape[0], -1, -1))
        b2 = (d * s2).sum(-1) * inv
        t = (e2[None] * s2).sum(-1) * inv
        ok = (b1 >= 0) & (b1 <= 1) & (b2 >= 0) & (b1 + b2 <= 1) & (t > r[:, None, 3]) & (t <= r[:, None, 7])
        best, k = torch.where(ok, t, torch.inf).min(1)
        hit = torch.isfinite(best)
        i = torch.arange(r.shape[0], device="cuda")
        t_out[a:a + step] = torch.where(hit, best, r[:, 7])
        uv_out[0, a:a + step] = torch.where(hit, b1[i, k], 0.0)
        uv_out[1, a:a + step] = torch.where(hit, b2[i, k], 0.0)
    return {"t": t_out, "prim": None, "u": uv_out[0], "v": uv_out[1]}


# ---------------------------------------------------------------- renders
_TRACER = {"gi": abi.BG_TRACER_GI, "di": abi.BG_TRACER_DI, "ao": abi.BG_TRACER_AO}
_SAMPLER = {"random": abi.BG_SAMPLER_RANDOM, "sobol": abi.BG_SAMPLER_SOBOL, "cmj": abi.BG_SAMPLER_CMJ}


def _prepare_render(case, seed):
    if case["scene"] == "cornell":
        sc, builder = scenes.cornell(case["w"], case["h"]), 0
    else:
        sc = scenes.production(case["w"], case["h"], nterrain=case["nterrain"], nspheres=case["nspheres"],
                               sphere_seg=case["seg"], seed=seed)
        builder = 3 if sc.ntriangles >= 50_000 else 0
    gs = capi.GpuScene(_ctx(), sc, builder=builder)
    args = dict(seed=seed, tracer=_TRACER[case["tracer"]], maxdepth=case["depth"], sampler=_SAMPLER[case["sampler"]],
                grid=4 if case["sampler"] == "cmj" else 0, ao_radius=2.0 if case["tracer"] == "ao" else 0.0)
    st = dict(case=case, gs=gs, args=args)
    if not case["host"]:
        st["acc"] = torch.zeros((case["h"], case["w"], 4), device="cuda")
    return st


def _run_render(st):
    c = st["case"]
    if c["host"]:
        return st["gs"].render_host(c["w"], c["h"], c["spp"], **st["args"])
    st["acc"].zero_()
    st["gs"].render(st["acc"].data_ptr(), c["w"], c["h"], c["spp"], stats=False, **st["args"])
    return st["acc"]


def _prepare_batch(case, seed):
    """Scenes made as scenes.batch makes them, with the three resolutions in turn."""
    rng = np.random.default_rng(seed)
    items = []
    for k in range(case["scenes"]):
        tris = math.exp(rng.uniform(math.log(case["tri_lo"]), math.log(case["tri_hi"])))
        w, h = ((256, 256), (512, 512), (1024, 768))[k % 3]
        spheres = int(rng.integers(4, 24))
        seg = max(8, math.isqrt(int(0.2 * tris / spheres)))
        terrain = max(8, math.isqrt(int(max(tris - 2 * spheres * seg * seg, 2e3) / 2)) + 1)
        items.append(scenes.production(w, h, nterrain=terrain, nspheres=spheres, sphere_seg=seg,
                                       seed=int(rng.integers(1 << 30))))
    gss = [capi.GpuScene(_ctx(), sc, builder=3) for sc in items]
    batch = capi.Batch(_ctx(), gss)
    accs = [torch.zeros((sc.height, sc.width, 4), device="cuda") for sc in items]
    jobs = [dict(scene=k, width=sc.width, height=sc.height, spp=case["spp"], seed=seed + k, camera=sc.camera_desc(),
                 accum_dev=accs[k].data_ptr()) for k, sc in enumerate(items)]
    return dict(case=case, batch=batch, accs=accs, jobs=jobs)


def _run_batch(st):
    torch._foreach_zero_(st["accs"])
    st["batch"].render(st["jobs"], maxdepth=st["case"]["depth"])
    return st["accs"]


# ---------------------------------------------------------- radiance cache
_RES_LO, _RES_HI, _LEVELS = 16, 2048, 16


def _features(n, g):
    """Query records of path vertices: points of a rolling surface in the unit
    cube, unit outgoing directions and normals, roughness, albedo."""
    f = torch.zeros((n, 16), device="cuda")
    u = torch.rand((n, 7), generator=g, device="cuda")
    f[:, 0], f[:, 2] = u[:, 0], u[:, 1]
    f[:, 1] = 0.5 + 0.2 * torch.sin(9 * u[:, 0]) * torch.cos(7 * u[:, 1]) + 0.05 * u[:, 2]
    for k in (3, 6):
        d = torch.randn((n, 3), generator=g, device="cuda")
        f[:, k:k + 3] = d / d.norm(dim=1, keepdim=True)
    f[:, 9:13] = u[:, 3:7]
    return f


def _params(case, seed):
    """Weights of a network in use: grid features of a tenth to a half, fan-in scaled layers."""
    rng = np.random.default_rng(seed)
    grid = (rng.random(_LEVELS * (1 << case["log2t"]) * 2, dtype=np.float32) - 0.5)
    shapes = [(64, 128)] + [(64, 64)] * 4 + [(16, 64)]
    mlp = np.concatenate([(rng.normal(size=s) * math.sqrt(2.0 / s[1])).astype(np.float32).reshape(-1) for s in shapes])
    return mlp, grid


def _prepare_cache(case, seed):
    gs = capi.GpuScene(_ctx(), scenes.cornell(64, 64))
    cache = capi.RadianceCache(gs, log2_table_size=case["log2t"], base_resolution=_RES_LO, max_resolution=_RES_HI,
                               bbox=((0, 0, 0), (1, 1, 1)), seed=seed)
    mlp, grid = _params(case, seed)
    cache.set_params(mlp, grid)
    g = torch.Generator(device="cuda").manual_seed(seed)
    st = dict(case=case, gs=gs, cache=cache)
    if case["kind"] == "query":
        st["feat"] = _features(case["rows"], g)
        st["out"] = torch.zeros((case["rows"], 4), device="cuda")
        return st
    st["feat"] = [_features(case["rows"], g) for _ in range(case["steps"])]
    st["target"] = []
    for f in st["feat"]:
        t = torch.zeros((case["rows"], 4), device="cuda")
        t[:, 0] = 0.5 + 0.4 * torch.sin(6 * f[:, 0]) * torch.cos(4 * f[:, 1])
        t[:, 1] = 0.3 + 0.2 * f[:, 2] + 0.1 * f[:, 5]
        t[:, 2] = 0.2 + 0.2 * f[:, 10]
        st["target"].append(t)
    st["held"] = _features(4096, g)
    st["out"] = torch.zeros((4096, 4), device="cuda")
    inf = cache.info()
    st["mlp"], st["grid"] = (torch.zeros(inf[k], pin_memory=True) for k in ("mlp_params", "grid_params"))
    return st


def _run_query(st):
    st["cache"].query(st["feat"].data_ptr(), st["out"].data_ptr(), st["case"]["rows"])
    return st["out"]


def _run_train(st):
    """Adam steps on rows of their own: the loss of the last one, predictions of the
    updated network, and its weights and grid as a checkpoint reads them."""
    cache, n = st["cache"], st["case"]["rows"]
    for k, (f, t) in enumerate(zip(st["feat"], st["target"])):
        loss = cache.train(f.data_ptr(), t.data_ptr(), n, want_loss=k + 1 == len(st["feat"]))
    cache.query(st["held"].data_ptr(), st["out"].data_ptr(), 4096)
    capi.check(capi.lib().bg_cache_params(cache.h, st["mlp"].data_ptr(), st["grid"].data_ptr(), None, None))
    return {"loss": np.float32(loss), "held_out": st["out"], "mlp": st["mlp"], "grid": st["grid"]}


def _exact_query(case, seed):
    """Hash-grid and one-blob encoding and the six layers in 64 bits, from the 32-bit parameters."""
    mlp, grid = (torch.from_numpy(a).cuda().double() for a in _params(case, seed))
    f = _features(case["rows"], torch.Generator(device="cuda").manual_seed(seed)).double()
    T = 1 << case["log2t"]
    grid = grid.view(_LEVELS, T, 2)
    u = ((f[:, 0:3] + 1e-3) / 1.002).clamp(0, 1)
    cols = []
    b = math.exp((math.log(_RES_HI) - math.log(_RES_LO)) / (_LEVELS - 1))
    for lvl in range(_LEVELS):
        res = math.floor(_RES_LO * b ** lvl)
        x = u * res
        c = x.floor().clamp(max=res - 1)
        w, c = x - c, c.long()
        feat = torch.zeros((f.shape[0], 2), dtype=torch.float64, device="cuda")
        for k in range(8):
            bit = torch.tensor([k & 1, k >> 1 & 1, k >> 2 & 1], device="cuda")
            i = c + bit
            if (res + 1) ** 3 <= T:
                idx = i[:, 0] + (res + 1) * (i[:, 1] + (res + 1) * i[:, 2])
            else:
                idx = (i[:, 0] ^ i[:, 1] * 2654435761 ^ i[:, 2] * 805459861) & (T - 1)
            feat += torch.where(bit == 1, w, 1 - w).prod(1, keepdim=True) * grid[lvl, idx]
        cols.append(feat)
    centres = (torch.arange(16, device="cuda").double() + 0.5) / 16
    for k in (3, 6):
        d = f[:, k:k + 3]
        for v in (torch.acos(d[:, 2].clamp(-1, 1)) / math.pi, torch.atan2(d[:, 1], d[:, 0]) / (2 * math.pi) + 0.5):
            cols.append(torch.exp(-128.0 * (v[:, None] - centres) ** 2))
    cols += [f[:, 9:13], torch.ones_like(f[:, :1])]
    x = torch.cat(cols, 1)
    x = torch.cat([x, torch.zeros((x.shape[0], 128 - x.shape[1]), dtype=torch.float64, device="cuda")], 1)
    off = 0
    for k, (o, i) in enumerate([(64, 128)] + [(64, 64)] * 4 + [(16, 64)]):
        x = x @ mlp[off:off + o * i].view(o, i).T
        x = x.relu() if k < 5 else x
        off += o * i
    return torch.cat([x[:, :3], torch.zeros_like(x[:, :1])], 1)


# ---------------------------------------------------------------- dispatch
def prepare(case, seed):
    make = {"cast": _prepare_cast, "render": _prepare_render, "batch": _prepare_batch, "query": _prepare_cache,
            "train": _prepare_cache}
    return make[case["kind"]](case, seed)


def run(state):
    go = {"cast": _run_cast, "render": _run_render, "batch": _run_batch, "query": _run_query, "train": _run_train}
    return go[state["case"]["kind"]](state)


def exact(case, seed):
    """None for renders (a path's decisions follow from single 32-bit values: an
    image in 64 bits is another image) and for training (Adam's first steps
    divide each gradient by its own size)."""
    if case["kind"] == "cast":
        return _exact_cast(case, seed)
    if case["kind"] == "query":
        return _exact_query(case, seed)
    return None


def _ray_flops(tris):
    """Finding a ray's triangle by halving the scene: one box test (18 operations)
    per halving, and one triangle test."""
    return 18 * max(1.0, math.log2(tris)) + 50


def work(case):
    k = case["kind"]
    if k == "cast":
        n = case["rays"]
        # a ray touches at most a few triangles; a large set touches the whole scene once
        scene = 36 * min(case["tris"], 8 * n)
        return {"bytes": n * (32 + (1 if case["any"] else 16)) + scene, "flops": n * _ray_flops(case["tris"])}
    if k == "render":
        tris = 36 if case["scene"] == "cornell" else 2 * case["nterrain"] ** 2 + 2 * case["nspheres"] * case["seg"] ** 2
        samples = case["w"] * case["h"] * case["spp"]
        vertices = min(case["depth"], 2) if case["tracer"] == "gi" else 1
        rays = samples * vertices * (2 if case["tracer"] == "ao" else 3)
        return {"bytes": case["w"] * case["h"] * 32 + 36 * min(tris, 8 * rays), "flops": rays * _ray_flops(tris)}
    if k == "batch":
        pixels, tris = case["scenes"] * 370_000, math.sqrt(case["tri_lo"] * case["tri_hi"])
        rays = pixels * case["spp"] * 6
        return {"bytes": pixels * 32 + 36 * case["scenes"] * tris, "flops": rays * _ray_flops(tris)}
    per_row = 2 * (64 * 128 + 4 * 64 * 64 + 16 * 64)
    rows, table = case["rows"], 1 << case["log2t"]
    touched = _LEVELS * min(table, 8 * rows)
    if k == "query":
        return {"bytes": rows * 80 + touched * 8 + 51_200, "flops": rows * per_row}
    # each step reads and writes the value and the two moments of the entries its rows touch
    return {"bytes": case["steps"] * (rows * 80 + touched * 8 * 6) + _LEVELS * table * 8,
            "flops": case["steps"] * rows * per_row * 3}
