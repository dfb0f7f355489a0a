"""Every walk of the traversal gives the plain walk's bits.

A cast of a few rays goes to groups of 32 or 8 lanes per ray, a larger one to one
lane per ray on packed nodes or, below 1,000 triangles, to the plain walk; the
host entry points read a few rays in place.  The same rays cast in pieces of
every size around those limits must give the same ids, t, u, v and occlusion
bits as one large cast, ties between coincident triangles included.  Scenes of a few nodes
have a walk of their own in large launches: the same bits again.
"""
import numpy as np
import pytest

from banshee_b200 import abi, scenes
from banshee_b200.scene import Mesh, Scene, lambert

pytestmark = pytest.mark.gpu

WARPS = 148 * 5 * 4          # warps of the group walk's grid on a B200
SIZES = (1, 3, 31, 32, 33, 257, WARPS - 1, WARPS, WARPS + 1, 4 * WARPS + 5, 32 * WARPS, 32 * WARPS + 1)


@pytest.fixture(scope="module")
def ctx():
    from banshee_b200 import capi
    return capi.Context(0)


def _ties(n=570):
    """A soup every third triangle of which is there three times, in other meshes' leaves too."""
    sc = scenes.soup(n, seed=5)
    m = sc.meshes[0]
    v = m.vertices.reshape(-1, 3, 3)
    grown = v.mean(1, keepdims=True) + 12 * (v - v.mean(1, keepdims=True))   # large enough to be hit
    tri = np.concatenate([grown, grown[::3], grown[::3]])
    k = tri.shape[0]
    idx = np.arange(3 * k, dtype=np.int32).reshape(k, 3)
    nrm = np.tile(np.array([[0, 0, 1]], np.float32), (k, 1))
    sc.meshes = [Mesh(tri.reshape(-1, 3), nrm, idx, np.repeat(np.arange(k, dtype=np.int32)[:, None], 3, 1),
                      np.zeros(k, np.int32))]
    return sc


def _grid(n=48):
    """A flat grid of quads: rays through its vertices and edges hit several triangles at one t."""
    g = np.linspace(0, 1, n + 1, dtype=np.float32)
    x, y = np.meshgrid(g, g, indexing="ij")
    v = np.stack([x, y, 0.25 * np.ones_like(x)], -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    a = (i * (n + 1) + j).reshape(-1)
    f = np.concatenate([np.stack([a, a + n + 1, a + n + 2], 1), np.stack([a, a + n + 2, a + 1], 1)]).astype(np.int32)
    sc = Scene(name="grid")
    sc.materials = [lambert((0.5, 0.5, 0.5))]
    sc.meshes = [Mesh(v, np.array([[0, 0, 1]], np.float32), f, np.zeros_like(f), np.zeros(len(f), np.int32))]
    return sc


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    r = scenes.soup_rays(n, "incoherent", seed=seed)
    r["tmax"] = 8.0
    k = n // 8
    r["d"][:k] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, k)] * rng.choice([-1, 1], (k, 1))   # axis-parallel
    o = r["o"][k:2 * k]                                                   # at the grid's vertices and edge points
    o[:] = np.stack([rng.integers(0, 97, k) / 96, rng.integers(0, 97, k) / 96, np.where(rng.random(k) < 0.5, 0.0, 1.0)], 1)
    r["d"][k:2 * k] = np.where(o[:, 2:] > 0.5, -1, 1) * np.array([0, 0, 1], np.float32)
    r["d"][2 * k:3 * k] = (np.array([0.5, 0.5, 0.25]) - r["o"][2 * k:3 * k])      # towards one grid vertex
    r["tmax"][3 * k:4 * k] = rng.random(k)
    bad = r[4 * k:4 * k + 40]
    bad["d"][::4] = 0
    bad["o"][1::4] = np.nan
    bad["d"][2::4, 0] = np.inf
    bad["tmax"][3::4] = np.nan
    bad["o"][5] = (np.nan, 0.5, 0.5)
    return r[rng.permutation(n)]


def _scene(name):
    if name == "ties":
        return _ties(), 0
    if name == "grid":
        return _grid(), 0
    if name == "cornell":
        return scenes.cornell(8, 8), 0
    return scenes.soup(20_000, seed=6), 3


@pytest.mark.parametrize("intersect", [0, 1], ids=["moller", "watertight"])
@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("name", ["ties", "grid", "cornell", "soup"])
def test_pieces_give_the_bits_of_one_cast(ctx, name, width, intersect):
    import torch
    from banshee_b200 import capi
    sc, builder = _scene(name)
    gs = capi.GpuScene(ctx, sc, builder=builder, intersect=intersect)
    gs.set_node_width(width)
    rays = _rays(32 * WARPS + 20_000, 11)
    n = len(rays)
    dev = torch.from_numpy(rays.view(np.uint8).reshape(n, 32)).cuda()

    def cast(lo, hi):
        h = torch.full((hi - lo, 4), -5.0, device="cuda")
        o = torch.full((hi - lo,), 9, dtype=torch.uint8, device="cuda")
        piece = dev[lo:hi].contiguous()
        gs.intersect_closest(piece.data_ptr(), h.data_ptr(), hi - lo)
        gs.intersect_any(piece.data_ptr(), o.data_ptr(), hi - lo)
        torch.cuda.synchronize()
        return h.cpu().numpy().view(np.uint32), o.cpu().numpy()

    whole, occ = cast(0, n)
    prim = whole[:, 1].view(np.int32)
    assert 0.05 < (prim >= 0).mean() < 1.0
    fin = np.isfinite(rays["tmax"])
    assert (occ[fin] == (prim[fin] >= 0)).all()
    for k, size in enumerate(SIZES):
        lo = (k * 977) % (n - size + 1)
        h, o = cast(lo, lo + size)
        assert (h == whole[lo:lo + size]).all(), size
        assert (o == occ[lo:lo + size]).all(), size
    for size in (1, 1024, 1025):                                        # in place, staged
        h = gs.intersect_closest_host(rays[:size])
        assert (h.view(np.uint32).reshape(-1, 4) == whole[:size]).all(), size
        assert (gs.intersect_any_host(rays[:size]) == occ[:size]).all(), size
    assert gs.error_flags() == 0


@pytest.mark.parametrize("name", ["ties", "soup"])
def test_closest_hits_match_the_oracle(ctx, oracle_built, name):
    """t to the last bit; the id wherever no other triangle has the same t."""
    from banshee_b200 import capi
    sc, builder = _scene(name)
    gs = capi.GpuScene(ctx, sc, builder=builder)
    rays = scenes.soup_rays(4096, "incoherent", seed=12)
    want = oracle_built.Oracle(sc).intersect_closest(rays)
    for got in (gs.intersect_closest_host(rays), np.concatenate([gs.intersect_closest_host(rays[i:i + 700]) for i in range(0, 4096, 700)])):
        assert (got["t"].view(np.uint32) == want["t"].view(np.uint32)).all()
        if name == "soup":
            assert (got["primid"] == want["primid"]).all()


def test_coordinates_beyond_the_packed_range_keep_the_plain_walk(ctx, oracle_built):
    """One triangle 4e15 units away puts the scene outside the packed arithmetic's range."""
    from banshee_b200 import capi
    sc = scenes.soup(5000, seed=9)
    m = sc.meshes[0]
    v = m.vertices.reshape(-1, 3, 3)
    v[:] = v.mean(1, keepdims=True) + 6 * (v - v.mean(1, keepdims=True))
    v[0] = np.float32(4e15)
    gs = capi.GpuScene(ctx, sc)
    rays = scenes.soup_rays(2048, "incoherent", seed=13)
    rays["tmax"] = 8.0
    want = oracle_built.Oracle(sc).intersect_closest(rays)
    got = gs.intersect_closest_host(rays)
    assert (want["primid"] >= 0).mean() > 0.05
    assert (got["primid"] == want["primid"]).all()
    assert (got["t"].view(np.uint32) == want["t"].view(np.uint32)).all()


@pytest.mark.parametrize("intersect", [0, 1], ids=["moller", "watertight"])
@pytest.mark.parametrize("ntris", [1, 3, 6, 10])
def test_scenes_of_few_nodes_give_the_bits_of_the_groups(ctx, oracle_built, ntris, intersect):
    """One to four nodes, every third triangle there three times: one large cast against
    casts small enough for groups of lanes, and t against the oracle."""
    import torch
    from banshee_b200 import capi
    sc = _ties(ntris)
    gs = capi.GpuScene(ctx, sc, intersect=intersect)
    n = 32 * WARPS + 20_000
    rays = _rays(n, 17)
    dev = torch.from_numpy(rays.view(np.uint8).reshape(n, 32)).cuda()

    def cast(lo, hi):
        h = torch.full((hi - lo, 4), -5.0, device="cuda")
        o = torch.full((hi - lo,), 9, dtype=torch.uint8, device="cuda")
        piece = dev[lo:hi].contiguous()
        gs.intersect_closest(piece.data_ptr(), h.data_ptr(), hi - lo)
        gs.intersect_any(piece.data_ptr(), o.data_ptr(), hi - lo)
        torch.cuda.synchronize()
        return h.cpu().numpy().view(np.uint32), o.cpu().numpy()

    whole, occ = cast(0, n)
    for lo in range(0, n, 32 * WARPS):
        h, o = cast(lo, min(n, lo + 32 * WARPS))
        assert (h == whole[lo:lo + 32 * WARPS]).all()
        assert (o == occ[lo:lo + 32 * WARPS]).all()
    if intersect == 0:
        plain = scenes.soup_rays(n, "incoherent", seed=18)
        got = gs.intersect_closest_host(plain)
        want = oracle_built.Oracle(sc).intersect_closest(plain)
        assert (got["t"].view(np.uint32) == want["t"].view(np.uint32)).all()
    assert gs.error_flags() == 0


@pytest.mark.parametrize("spp", [1, 3])
def test_cornell_renders_the_same_in_a_batch(ctx, spp):
    """A pass of more paths than groups of lanes take: one scene of nine nodes against
    the same scene as a batch, whose rays walk the tree from a root of their own."""
    import torch
    from banshee_b200 import capi
    w, h = 320, 304
    gs = capi.GpuScene(ctx, scenes.cornell(w, h))
    assert gs.info()["nnodes"] <= 16
    want = gs.render_host(w, h, spp, seed=3, maxdepth=5)
    batch = capi.Batch(ctx, [gs])
    acc = torch.zeros((h, w, 4), device="cuda")
    batch.render([dict(scene=0, width=w, height=h, spp=spp, seed=3, accum_dev=acc.data_ptr())], maxdepth=5)
    torch.cuda.synchronize()
    assert (acc.cpu().numpy().view(np.uint32) == want.view(np.uint32)).all()


def test_commit_without_room_for_the_packed_nodes(ctx):
    """The packed nodes are allocated last: a budget one byte short of a commit's needs
    leaves the scene to the plain walk, with the same hits."""
    from banshee_b200 import capi
    sc = scenes.soup(20_000, seed=14)
    rays = scenes.soup_rays(32 * WARPS + 5_000, "incoherent", seed=15)
    full = capi.GpuScene(ctx, sc, commit=False)
    before = capi.alloc_stats()["bytes"]
    full.commit()
    need = capi.alloc_stats()["bytes"] - before
    tight = capi.GpuScene(ctx, sc, commit=False)
    capi.alloc_limit(need - 1)
    try:
        tight.commit()
    finally:
        capi.alloc_limit(None)
    want = full.intersect_closest_host(rays)
    got = tight.intersect_closest_host(rays)
    assert (want["primid"] >= 0).mean() > 0.05
    assert (got.view(np.uint32) == want.view(np.uint32)).all()
    assert (tight.intersect_any_host(rays) == full.intersect_any_host(rays)).all()


@pytest.mark.parametrize("n", [1, 33, 4000])
def test_rays_along_a_wall_give_the_bits_of_the_plain_walk(ctx, n):
    """Rays from the walls of a Cornell box that leave its box by a millionth of their way:
    the first three hit a wall's edge in boxes that the plain walk culls."""
    import torch
    from banshee_b200 import capi
    gs = capi.GpuScene(ctx, scenes.cornell(64, 64))
    h = float.fromhex
    rays = scenes.soup_rays(32 * WARPS + 4096, "incoherent", seed=21)
    rng = np.random.default_rng(22)
    k = len(rays)
    o, d = rng.random((k, 3)).astype(np.float32), rng.normal(size=(k, 3)).astype(np.float32)
    axis = rng.integers(0, 3, k)
    o[np.arange(k), axis] = rng.integers(0, 2, k)
    d[np.arange(k), axis] = np.ldexp(rng.normal(size=k), -rng.integers(16, 28, k))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    fixed = [("0x1.a7aa62p-4", "0x1p+0", "0x1.327fd8p-5", "-0x1.ffff98p-1", "0x1.c56ca6p-21", "0x1.45e482p-9"),
             ("0x1.76e478p-2", "0x1p+0", "0x1.f532fep-4", "0x1.e4f704p-3", "0x1.4dc444p-22", "-0x1.f17020p-1"),
             ("0x1p+0", "0x1.fcb3d2p-1", "0x1.e313e4p-2", "0x1.57aa4cp-20", "0x1.338888p-1", "0x1.99598cp-1")]
    for i, f in enumerate(fixed):
        o[i], d[i] = [h(x) for x in f[:3]], [h(x) for x in f[3:]]
    rays["o"], rays["d"], rays["tmin"], rays["tmax"] = o, d, 0.01, 1e6
    dev = torch.from_numpy(rays.view(np.uint8).reshape(k, 32)).cuda()

    def cast(m):
        out, occ = torch.zeros((m, 4), device="cuda"), torch.zeros((m,), dtype=torch.uint8, device="cuda")
        gs.intersect_closest(dev.data_ptr(), out.data_ptr(), m)
        gs.intersect_any(dev.data_ptr(), occ.data_ptr(), m)
        torch.cuda.synchronize()
        return out.cpu().numpy().view(np.uint32), occ.cpu().numpy()

    whole, occ = cast(k)                        # more rays than groups take: the plain walk
    got, gocc = cast(n)                         # groups of lanes
    assert (got == whole[:n]).all() and (gocc == occ[:n]).all()
    assert (whole[:min(n, 3), 1].view(np.int32) == -1).all()
