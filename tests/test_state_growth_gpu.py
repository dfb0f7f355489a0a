"""What a scene keeps between renders survives a larger render."""
import numpy as np
import pytest

from banshee_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from banshee_b200 import capi
    return capi.Context(0)


def _accum(w, h):
    import torch
    return torch.zeros((h, w, 4), device="cuda")


@pytest.mark.parametrize("between", ["nothing", "a larger render", "a render without room"])
def test_pending_training_rows_are_trained(ctx, between):
    """A cached frame's rows are trained at the start of the cache's next frame, whatever
    plain renders come between."""
    import torch
    from banshee_b200 import capi
    gs = capi.GpuScene(ctx, scenes.cornell(64, 64))
    cache = capi.RadianceCache(gs, log2_table_size=14, train_paths=1024, train_batch=2048, train_steps=4)
    frame, big = _accum(64, 64), _accum(1920, 1088)
    cache.render(frame.data_ptr(), 64, 64, 1, seed=1, maxdepth=5)
    torch.cuda.synchronize()
    before = cache.params()
    if between == "a larger render":
        gs.render(big.data_ptr(), 1920, 1088, 2, seed=2, maxdepth=2, stats=False)
    elif between == "a render without room":
        capi.alloc_limit(1 << 20)
        try:
            with pytest.raises(capi.BansheeError):
                gs.render(big.data_ptr(), 1920, 1088, 2, seed=2, maxdepth=2, stats=False)
        finally:
            capi.alloc_limit(None)
    cache.render(frame.data_ptr(), 64, 64, 1, seed=3, maxdepth=5)
    torch.cuda.synchronize()
    after = cache.params()
    assert (before[0] != after[0]).mean() > 0.5                      # the network has been trained
    assert 0 < (before[1] != after[1]).sum()
    assert np.isfinite(after[0]).all() and np.isfinite(after[1]).all()


def test_an_unchanged_render_allocates_nothing(ctx):
    """The pass size that a budget allowed stays when the budget has gone: a caller may hold
    the state's memory in a graph, and the call has not changed.  A larger call may grow it."""
    import torch
    from banshee_b200 import capi
    w, h = 1920, 1088
    used = []
    for limit in (None, 0):
        gs = capi.GpuScene(ctx, scenes.cornell(64, 64))
        acc = _accum(w, h)
        before = capi.alloc_stats()["bytes"]
        capi.alloc_limit(limit if limit is None else int(1.2 * used[0] * (1 << 21) / (w * h * 3)))
        try:
            gs.render(acc.data_ptr(), w, h, 3, seed=1, maxdepth=2, stats=False)
        finally:
            capi.alloc_limit(None)
        torch.cuda.synchronize()
        used.append(capi.alloc_stats()["bytes"] - before)
    assert used[1] < 0.7 * used[0]                                # passes of 2^21 instead of one of all
    had = capi.alloc_stats()["bytes"]
    gs.render(acc.data_ptr(), w, h, 3, seed=1, maxdepth=2, stats=False)
    torch.cuda.synchronize()
    assert capi.alloc_stats()["bytes"] < had + (1 << 20)          # (the second staging of the segment tables)
    gs.render(acc.data_ptr(), w, h, 4, seed=1, maxdepth=2, stats=False)
    torch.cuda.synchronize()
    assert capi.alloc_stats()["bytes"] > had + used[1]


@pytest.mark.parametrize("size", [33, 64, 150])
def test_a_small_render_after_a_large_one(ctx, size):
    """The same kernels and the same image as in a scene that has rendered nothing larger."""
    import torch
    from banshee_b200 import capi
    got = []
    for large in (False, True):
        gs = capi.GpuScene(ctx, scenes.cornell(64, 64))
        if large:
            gs.render(_accum(640, 480).data_ptr(), 640, 480, 4, seed=1, maxdepth=5, stats=False)
        acc = _accum(size, size)
        stats = gs.render(acc.data_ptr(), size, size, 1, seed=2, maxdepth=5)
        gs.render(acc.data_ptr(), size, size, 1, seed=3, maxdepth=5, stats=False)
        torch.cuda.synchronize()
        got.append((stats["kernel_launches"], acc.cpu().numpy()))
    assert got[0][0] == got[1][0]
    assert got[0][1].max() > 0 and (got[0][1].view(np.uint32) == got[1][1].view(np.uint32)).all()


def test_deeper_renders_after_a_shallow_one(ctx):
    """The counters of a pass grow with its bounces: a new scene's first small render allocates
    less than a megabyte."""
    import torch
    from banshee_b200 import capi
    images = []
    for depths in ((3, 31, 32, 33, 200, 5), (200, 3, 31, 32, 33, 5)):
        gs = capi.GpuScene(ctx, scenes.cornell(64, 64))
        acc = _accum(8, 8)
        before = capi.alloc_stats()["bytes"]
        for k, depth in enumerate(depths):
            gs.render(acc.data_ptr(), 8, 8, 16, seed=depth, maxdepth=depth, stats=False)
            torch.cuda.synchronize()
            if k == 0 and depth == 3:
                assert capi.alloc_stats()["bytes"] - before < 1024 * 1300 + (1 << 20)   # (beside the state of 1,024 paths)
        images.append(acc.cpu().numpy())
    assert np.allclose(images[0], images[1], rtol=1e-5, atol=0)      # the same frames, summed in another order
    assert images[0].max() > 0 and gs.error_flags() == 0


def test_nodes_that_cannot_be_packed_hold_no_memory(ctx):
    """A triangle beyond the packed range leaves the scene to the plain walk; its packed nodes go."""
    import torch
    from banshee_b200 import capi
    held = []
    capi.GpuScene(ctx, scenes.soup(1 << 20, seed=5), builder=3, node_width=4).close()   # the build's scratch stays
    for far in (False, True):
        sc = scenes.soup(1 << 20, seed=5)
        if far:
            sc.meshes[0].vertices.reshape(-1, 3, 3)[0] = np.float32(4e15)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        gs = capi.GpuScene(ctx, sc, builder=3, node_width=4)
        torch.cuda.synchronize()
        held.append(free - torch.cuda.mem_get_info()[0])
        packed = gs.info()["nnodes"] * 64
        gs.close()
    assert held[1] < held[0] - 0.8 * packed, (held, packed)
