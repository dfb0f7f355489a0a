"""The walk a launch is given suits its rays and its scene."""
import pytest

from banshee_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from banshee_b200 import capi
    return capi.Context(0)


def _rays(n, kind, occlusion):
    import torch
    r = scenes.soup_rays(n, kind, seed=61, any_hit=occlusion, tmax_range=(1.5, 2.5) if kind == "coherent" else (0.0, 1.0))
    return torch.from_numpy(r.view("u1").reshape(n, 32)).cuda()


def _us(run):
    """Least time of a call among four."""
    import torch
    times = []
    for k in range(12):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(4):
            run()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 250)
    return min(times)


@pytest.mark.parametrize("kind", ["coherent", "incoherent"])
@pytest.mark.parametrize("tris", [36, 1000, 20_000])
def test_fewer_rays_take_no_longer(ctx, tris, kind):
    """A cast of any size takes at most 1.4 times as long as one of more rays."""
    import torch
    from banshee_b200 import capi
    gs = capi.GpuScene(ctx, scenes.cornell(8, 8) if tris == 36 else scenes.soup(tris, seed=3))
    for occlusion in (False, True):
        times = []
        for side in (64, 128, 180, 256, 306, 362, 420):
            n = side * side
            rays = _rays(n, kind, occlusion)
            out = torch.zeros((n, 16), dtype=torch.uint8, device="cuda")
            cast = gs.intersect_any if occlusion else gs.intersect_closest
            times.append(_us(lambda: cast(rays.data_ptr(), out.data_ptr(), n)))
        for i, t in enumerate(times):
            assert t <= 1.4 * min(times[i:]), (occlusion, [round(x, 1) for x in times])


def test_rays_of_a_middle_column_take_no_longer(ctx):
    """A camera of odd width has rays whose x component is exactly 0."""
    import torch
    from banshee_b200 import capi
    gs = capi.GpuScene(ctx, scenes.soup(100_000, seed=3), builder=3)
    for side in (91, 363):
        times = []
        for w in (side, side + 1):
            n = w * w
            rays = scenes.soup_rays(n, "coherent", seed=61)
            assert (rays["d"][:, 0] == 0).any() == (w == side)
            dev = torch.from_numpy(rays.view("u1").reshape(n, 32)).cuda()
            out = torch.zeros((n, 16), dtype=torch.uint8, device="cuda")
            times.append(_us(lambda: gs.intersect_closest(dev.data_ptr(), out.data_ptr(), n)))
        assert times[0] <= 1.25 * times[1], times
