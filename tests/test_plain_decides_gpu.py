"""Every other walk against the plain one, where rounding decides.

The plain walk is had by itself in two ways: a scene committed with no room for its
packed nodes casts on it at every size, and a batch that also holds a scene 4e15 units
across renders on it, with node arrays that are copies of the scenes' own.
"""
import numpy as np
import pytest

from banshee_b200 import abi, scenes
from banshee_b200.scene import Mesh, Scene, camera, environment_light, lambert

pytestmark = pytest.mark.gpu

LARGE = 150_000              # rays of a cast that no group of lanes walks


@pytest.fixture(scope="module")
def ctx():
    from banshee_b200 import capi
    return capi.Context(0)


def _plain_twin(ctx, sc, full_kw):
    """(scene, the same scene without packed nodes): they are allocated last in a commit."""
    from banshee_b200 import capi
    full = capi.GpuScene(ctx, sc, commit=False, **full_kw)
    before = capi.alloc_stats()["bytes"]
    full.commit()
    need = capi.alloc_stats()["bytes"] - before
    tight = capi.GpuScene(ctx, sc, commit=False, **full_kw)
    capi.alloc_limit(need - 1)
    try:
        tight.commit()
    finally:
        capi.alloc_limit(None)
    return full, tight


def _small_triangles(n, seed, edge=1e-3):
    """Isolated right-angled triangles, two in three in an axis plane, one in six a sliver."""
    rng = np.random.default_rng(seed)
    p = rng.random((n, 3))
    ax = rng.integers(0, 3, n)
    eye = np.eye(3)
    a, b = eye[ax] * edge, eye[(ax + 1) % 3] * edge
    k = n // 3
    q, _ = np.linalg.qr(rng.normal(size=(k, 3, 3)))
    a[:k], b[:k] = q[:, 0] * edge, q[:, 1] * edge
    s = slice(k // 2, k // 2 + n // 6)
    b[s] = a[s] + 0.01 * b[s]
    return np.stack([p, p + a, p + b], 1).astype(np.float32)


def _mesh(tri):
    k = len(tri)
    idx = np.arange(3 * k, dtype=np.int32).reshape(k, 3)
    return Mesh(tri.reshape(-1, 3), np.array([[0, 0, 1]], np.float32), idx, np.zeros_like(idx), np.zeros(k, np.int32))


def _scene(tri, moved):
    sc = Scene(name="small")
    sc.materials = [lambert((0.5, 0.5, 0.5))]
    sc.meshes = [_mesh(tri)]
    if moved:
        sc.meshes[0].set_transform(scenes._translate((3.0, -2.0, 0.5)) @ scenes._rot_y(33.0) @ scenes._scale(1.7))
    return sc


def _edge_rays(tri, n, seed):
    """Rays at the edges of the triangles, by up to a thousandth of an edge inside or out, from 10 to 100,000
    edges away, most of them grazing; a quarter ends at the triangle by a few roundings more or less."""
    rng = np.random.default_rng(seed)
    t = tri[rng.integers(0, len(tri), n)].astype(np.float64)
    t = np.take_along_axis(t, rng.permuted(np.tile(np.arange(3), (n, 1)), axis=1)[:, :, None], 1)
    w = rng.random((n, 1))
    out = np.where(rng.random((n, 1)) < 0.5, -1, 1) * 10.0 ** rng.uniform(-7, -3, (n, 1))
    p = (t[:, 0] * w + t[:, 1] * (1 - w)) * (1 - out) + t[:, 2] * out
    nrm = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    d = rng.normal(size=(n, 3))
    d -= (d * nrm).sum(1, keepdims=True) * nrm
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d += nrm * 10.0 ** rng.uniform(-4, 0.5, (n, 1)) * rng.choice([-1, 1], (n, 1))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    dist = np.linalg.norm(t[:, 1] - t[:, 0], axis=1, keepdims=True) * 10.0 ** rng.uniform(1, 5, (n, 1))
    r = np.zeros(n, abi.RAY_DTYPE)
    r["o"], r["d"], r["tmin"] = p - d * dist, d, 0.0
    o, d = r["o"].astype(np.float64), r["d"].astype(np.float64)
    along = ((p - o) * d).sum(1) / (d * d).sum(1)
    r["tmax"] = np.where(rng.random(n) < 0.25, along * (1 + rng.integers(-8, 9, n) * 2.0 ** -24), 1e30)
    near = rng.random(n) < 0.1
    r["tmin"] = np.where(near, along * (1 + rng.integers(-8, 9, n) * 2.0 ** -24), 0.0)
    return r


def _cast(gs, dev, lo, hi):
    import torch
    h = torch.full((hi - lo, 4), -5.0, device="cuda")
    o = torch.full((hi - lo,), 9, dtype=torch.uint8, device="cuda")
    piece = dev[lo:hi].contiguous()
    gs.intersect_closest(piece.data_ptr(), h.data_ptr(), hi - lo)
    gs.intersect_any(piece.data_ptr(), o.data_ptr(), hi - lo)
    torch.cuda.synchronize()
    return h.cpu().numpy().view(np.uint32), o.cpu().numpy()


def _same(full, tight, rays, piece, most=0.98):
    import torch
    n = len(rays)
    dev = torch.from_numpy(rays.view(np.uint8).reshape(n, 32)).cuda()
    want, wocc = _cast(tight, dev, 0, n)
    assert 0.02 < (want[:, 1].view(np.int32) >= 0).mean() <= most
    for size in (n, piece) if piece else (n,):
        for lo in range(0, n if size == n else 40 * size, size):
            got, occ = _cast(full, dev, lo, min(n, lo + size))
            assert (got == want[lo:lo + size]).all(), (size, np.nonzero((got != want[lo:lo + size]).any(1))[0][:5] + lo)
            assert (occ == wocc[lo:lo + size]).all(), (size, np.nonzero(occ != wocc[lo:lo + size])[0][:5] + lo)


@pytest.mark.parametrize("moved", [False, True], ids=["identity", "transformed"])
@pytest.mark.parametrize("intersect", [0, 1], ids=["moller", "watertight"])
def test_rays_at_the_edges_of_small_triangles(ctx, intersect, moved):
    tri = _small_triangles(3000, 31)
    sc = _scene(tri, moved)
    full, tight = _plain_twin(ctx, sc, dict(intersect=intersect))
    world = sc.meshes[0].world_vertices().reshape(-1, 3, 3)
    for seed in range(6):
        _same(full, tight, _edge_rays(world, 1 << 20, 40 + seed), 2000)


@pytest.mark.parametrize("intersect", [0, 1], ids=["moller", "watertight"])
@pytest.mark.parametrize("name", ["grid", "ties"])
def test_ties_and_shared_edges(ctx, name, intersect):
    from tests.test_walks_gpu import _rays, _scene as walks_scene
    sc, builder = walks_scene(name)
    full, tight = _plain_twin(ctx, sc, dict(builder=builder, intersect=intersect))
    _same(full, tight, _rays(LARGE, 51), 3001)


# Slivers in planes of constant x and rays from the other side of the scene whose tmin lies just
# in front of the hit and, by up to nine roundings, behind the slab distance of the plane.
SLIVERS = [
    "fb94f0p-1 dd87b6p-4 -9cf9ecp-1 fb94f0p-1 2360ecp-3 -9060ccp-1 fb94f0p-1 2376a6p-3 -906ed2p-1 "
    "-f200fep-1 -000000p+0 -000000p+0 b2dd54p-1 f6707cp-2 751a1ep-4 27fd20p+1",
    "d39a08p-1 bb2a48p-1 -728526p-2 d39a08p-1 a5bd86p-1 -9a8036p-2 d39a08p-1 a64d76p-1 -9ae512p-2 "
    "-f2fbc6p-1 43ff84p-1 -8731cap-1 629446p+2 287832p-1 14b0c0p+0 5cedd4p-2",
    "cd85fap-1 -c7174ep-1 030fc4p-3 cd85fap-1 -bd6860p-1 a214c6p-4 cd85fap-1 -bc2ec2p-1 a706d0p-4 "
    "-f36c04p-1 -4e5f32p-4 9cd4a8p-1 b80b0ap+1 -71de28p+0 -485ceap+0 17853ep-1",
    "d4d596p-1 -a75988p-2 51c7e8p-1 d4d596p-1 -b96158p-2 47e0b0p-1 d4d596p-1 -bb7012p-2 4713bcp-1 "
    "-d84cf0p-1 -f51334p-3 278420p-1 a27692p+1 -51d8e2p-2 d5fd10p-4 1fe026p-1",
    "fcacfcp-1 ee4a32p-3 -0b3bd6p-1 fcacfcp-1 9afe82p-3 -055c7cp-1 fcacfcp-1 9aa30ep-3 -05858ap-1 "
    "-eb129ap-1 8d62f0p-3 -b4486cp-2 659628p+2 2a7a9ap-4 -0711dap-2 65dd8cp-2",
    "fef668p-1 -cc4044p-1 -4bb844p-1 fef668p-1 -c60b48p-1 -4e7296p-1 fef668p-1 -c6052ap-1 -4e318cp-1 "
    "-d581cep-1 -9ccf4ep-1 -2947a0p-1 d2d794p+1 -48fb84p-3 -135feep-3 0cd3f0p-1",
]


def test_hits_just_behind_tmin(ctx):
    """Rays of one octant walk the fused nodes: every sliver alone in its leaf, scene bounds [-1, 1]^3."""
    v = np.array([[float.fromhex(("-" if x[0] == "-" else "") + "0x1." + x.lstrip("-")) for x in c.split()] for c in SLIVERS],
                 np.float32)
    fill = (_small_triangles(1200, 33, 1e-4) * np.float32([0.01, 1, 1]) + np.float32([-0.999, 0, 0]))
    fill[0, 0], fill[1, 0] = (-1, -1, -1), (1, 1, 1)
    sc = _scene(np.concatenate([v[:, :9].reshape(-1, 3, 3), fill.astype(np.float32)]), False)
    full, tight = _plain_twin(ctx, sc, dict(max_leaf=1))
    r = np.zeros(len(v), abi.RAY_DTYPE)
    r["o"], r["d"], r["tmin"], r["tmax"] = v[:, 9:12], v[:, 12:15], v[:, 15], 1e30
    _same(full, tight, np.repeat(r, LARGE // len(v) // 32 * 32), 0, most=1.0)


@pytest.mark.parametrize("intersect", [0, 1], ids=["moller", "watertight"])
@pytest.mark.parametrize("name", ["grid", "soup", "small triangles"])
def test_rays_along_an_axis_plane(ctx, name, intersect):
    """One or two direction components are 0 or -0; a third of the origins lie on planes of the scene."""
    from tests.test_walks_gpu import _scene as walks_scene
    tri = _small_triangles(3000, 31, 0.02)
    sc, builder = (_scene(tri, False), 0) if name == "small triangles" else walks_scene(name)
    full, tight = _plain_twin(ctx, sc, dict(builder=builder, intersect=intersect))
    rng = np.random.default_rng(71)
    n = 1 << 19
    corners = sc.meshes[0].world_vertices().reshape(-1, 3)
    r = np.zeros(n, abi.RAY_DTYPE)
    r["o"], r["d"] = rng.random((n, 3)), rng.normal(size=(n, 3))
    d = r["d"]
    for k in range(2):
        zero = np.arange(n) if k == 0 else np.arange(0, n, 3)
        d[zero, rng.integers(0, 3, len(zero))] = rng.choice(np.float32([0, -0.0]), len(zero))
    d[(d == 0).all(1)] = (0, 1, 0)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    i = np.arange(0, n, 2)
    hit = corners[rng.integers(0, len(corners), len(i))] + 1e-3 * rng.normal(size=(len(i), 3))
    on = np.arange(len(i)) % 3 == 0
    hit[on] = corners[rng.integers(0, len(corners), on.sum())]
    r["o"][i] = hit - d[i] * rng.random((len(i), 1))
    flat = d[i] == 0
    r["o"][i] = np.where(flat, hit, r["o"][i])
    r["tmax"] = np.where(np.arange(n) % 4 == 3, rng.random(n), 8.0)
    r["tmin"] = np.where(np.arange(n) % 16 == 5, -0.25, 0.0)
    _same(full, tight, r, 2500)


def _huge():
    """One triangle 4e15 units away: a batch with it renders on the plain walk."""
    sc = scenes.production(8, 8, nterrain=4, nspheres=0, sphere_seg=4, seed=1)
    v = sc.meshes[0].vertices.reshape(-1, 3)
    v[sc.meshes[0].vidx.reshape(-1, 3)[0]] = np.float32(4e15)
    return sc


def _far_grid(height, n=48):
    """A grid of small quads seen from `height` quads above: camera rays at its vertices and edges."""
    from tests.test_walks_gpu import _grid
    sc = _grid(n)
    sc.lights = [environment_light((1.0, 0.9, 0.8))]
    h = height / n
    sc.camera = camera((0.5, 0.5, 0.25 + h), (0.5, 0.5, 0.0), (0, 1, 0), 1e-4, 1e6, float(np.degrees(2 * np.arctan(0.6 / h))), 1.0)
    return sc


RENDERS = {"cornell": lambda: scenes.cornell(64, 64),
           "production": lambda: scenes.production(64, 64, nterrain=40, nspheres=6, sphere_seg=12, seed=3),
           "grid from 30 quads": lambda: _far_grid(30), "grid from 30,000 quads": lambda: _far_grid(30_000)}


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("name", list(RENDERS))
def test_renders_on_every_walk(ctx, name, width):
    """48 x 48 paths (groups of lanes), 640 x 384 (fused, boxes-first or 8-wide packed walk)."""
    import torch
    from banshee_b200 import capi
    gs = capi.GpuScene(ctx, RENDERS[name](), node_width=width)
    plain = capi.Batch(ctx, [gs, capi.GpuScene(ctx, _huge(), node_width=width)])
    for w, h, spp in ((48, 48, 1), (640, 384, 2)):
        for tracer in (abi.BG_TRACER_GI, abi.BG_TRACER_AO):
            kw = dict(tracer=tracer, ao_radius=0.5)
            want, got = torch.zeros((h, w, 4), device="cuda"), torch.zeros((h, w, 4), device="cuda")
            plain.render([dict(scene=0, width=w, height=h, spp=spp, seed=4, accum_dev=want.data_ptr())], maxdepth=4, **kw)
            gs.render(got.data_ptr(), w, h, spp, seed=4, maxdepth=4, stats=False, **kw)
            torch.cuda.synchronize()
            assert want[..., :3].max() > 0
            assert (got.view(torch.int32) == want.view(torch.int32)).all(), (w, tracer)


@pytest.mark.parametrize("name", ["cornell", "production"])
def test_renders_without_room_for_the_packed_nodes(ctx, name):
    """The fused and the boxes-first walk need none: the same image, in about the same time."""
    import torch
    full, tight = _plain_twin(ctx, RENDERS[name](), {})
    acc = [torch.zeros((512, 640, 4), device="cuda") for _ in range(2)]
    times = [[], []]
    for k in range(12):
        for i, gs in enumerate((full, tight)):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            gs.render(acc[i].data_ptr(), 640, 512, 8, seed=k, maxdepth=5, stats=False)
            b.record()
            torch.cuda.synchronize()
            times[i].append(a.elapsed_time(b))
    assert (acc[0].view(torch.int32) == acc[1].view(torch.int32)).all()
    fast, slow = (min(t) for t in times)
    assert slow < 1.03 * fast, (fast, slow)
