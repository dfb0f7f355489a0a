"""The default pass size follows the memory there is; the image does not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

@pytest.fixture(scope="module")
def ctx():
    from banshee_b200 import capi
    return capi.Context(0)


@pytest.mark.parametrize("area", [True, False], ids=["area", "environment"])
@pytest.mark.parametrize("spp", [1, 3, 7])
def test_image_is_the_same_in_passes_of_every_size(ctx, area, spp):
    """1920 x 1088 with 1, 3 and 7 samples (below 2^21 paths, one pass, two passes of
    2^23), then with an allocation budget of which passes of 2^22 are an eighth, then
    with one that just holds 2^21: the images are equal bit for bit."""
    from banshee_b200 import capi, scenes
    w, h = 1920, 1088
    sc = scenes.cornell(w, h) if area else scenes.production(w, h, nterrain=24, nspheres=4, sphere_seg=8, seed=2)

    def image(limit):
        gs = capi.GpuScene(ctx, sc)
        before = capi.alloc_stats()["bytes"]
        capi.alloc_limit(limit)
        try:
            img = gs.render_host(w, h, spp, seed=5, maxdepth=3)
        finally:
            capi.alloc_limit(None)
        return img, capi.alloc_stats()["bytes"] - before

    want, most = image(None)
    assert np.isfinite(want).all() and want.max() > 0
    path = most / min(w * h * spp, 1 << 23) + 1          # bytes, staging included
    for limit in (int(8.5 * path * 2 ** 22), int(path * 2 ** 21) + w * h * 64):
        got, used = image(limit)
        assert used <= limit and used <= most
        assert used < most or spp == 1
        assert (got.view(np.uint32) == want.view(np.uint32)).all()
        most = used if spp == 7 else most
