"""The wavefront launch sequence (htcuda.cu launch_wave): overlapping launches, counters in two sets,
the scene image and the coherence sort give the one-pass kernel's bits at the sizes where their
paths change: canvases around one window, the least sorted queue (131072 paths) and the least sorted
canvas (2^19 pixels), object counts around the least sorted one (100) and a chunk, an odd and
an even number of sorts per call; and under stream capture, where a replay must find the counters and
histograms as a call does."""
import numpy as np
import pytest
import torch

from hypertrace_b200 import _lib
from hypertrace_b200 import batch as B
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S

pytestmark = pytest.mark.gpu


def _scene(geometry, n, hops):
    rng = np.random.default_rng(n)
    if geometry == "eu":
        return S.euclidean_scene(n - 1, hops, n, camera=B.random_hom3(rng))
    horo = (2 * n) // 3
    return S.hyperbolic_scene(n - horo, horo, 6.0, hops, 500 + n, camera=S.random_moebius(rng, 0.5))


@pytest.mark.parametrize("tile", [1, 33, 100, 512])
def test_batch_tiles_cover_hop_0_tiles(built, tile):
    """Views whose hop 0 takes 8 x 4 pixel tiles (ragged edges) and views too small for them, batch
    tiles of any size."""
    ctx = P.Context(0)
    views = []
    for i, (geometry, n, W, H) in enumerate([("hy", 20, 131, 67), ("eu", 9, 64, 32), ("hy", 110, 63, 200), ("eu", 5, 257, 33),
                                             ("hy", 40, 72, 31)]):
        views.append(B.View(_scene(geometry, n, 4), W, H, 16, 40 + i))
        views[-1].allocate(ctx)
    renderer = B.BatchRenderer(ctx)
    renderer.set_views(views, [2] * len(views), tile_pixels=tile)
    renderer.render()
    renderer.check()
    for v in views:
        canvas = P.Canvas(ctx, (v.width, v.height), v.global_seed)
        P.Render(ctx, v.scene.recipe, v.scene.hops).render_wavefront(v.buffer, canvas, 1)
        P.Render(ctx, v.scene.recipe, v.scene.hops).render(v.buffer, canvas)
        assert np.array_equal(_bits(canvas)[0], _bits(v.canvas)[0]) and np.array_equal(_bits(canvas)[1], _bits(v.canvas)[1])


@pytest.mark.parametrize("W,H", [(1024, 767), (1024, 768), (1280, 1023), (1280, 1024)])
@pytest.mark.parametrize("n", [15, 16])
def test_euclidean_routes_agree(built, W, H, n):
    """Around the canvas sizes and object counts where Euclidean calls become wavefronts."""
    ctx = P.Context(0)
    scene = _scene("eu", n, 3)
    render = P.Render(ctx, scene.recipe, scene.hops)
    buffer = P.EntityBuffer(ctx, scene)
    canvases = [P.Canvas(ctx, (W, H), 5) for _ in range(3)]
    for _ in range(2):
        render.render(buffer, canvases[0])
    render.render_passes(buffer, canvases[1], 2)
    render.render_wavefront(buffer, canvases[2], 2)
    for c in canvases[1:]:
        assert np.array_equal(_bits(canvases[0])[0], _bits(c)[0]) and np.array_equal(_bits(canvases[0])[1], _bits(c)[1])


@pytest.mark.parametrize("W,H,n", [(512, 287, 120), (512, 288, 120), (512, 288, 5), (512, 288, 6), (1024, 767, 5), (1024, 768, 5)])
def test_hyperbolic_routes_agree(built, W, H, n):
    """Around the canvas sizes and object counts where hyperbolic calls become wavefronts."""
    ctx = P.Context(0)
    scene = _scene("hy", n, 4)
    render = P.Render(ctx, scene.recipe, scene.hops)
    buffer = P.EntityBuffer(ctx, scene)
    canvases = [P.Canvas(ctx, (W, H), 6) for _ in range(3)]
    for _ in range(2):
        render.render(buffer, canvases[0])
    render.render_passes(buffer, canvases[1], 2)
    render.render_wavefront(buffer, canvases[2], 2)
    for c in canvases[1:]:
        assert np.array_equal(_bits(canvases[0])[0], _bits(c)[0]) and np.array_equal(_bits(canvases[0])[1], _bits(c)[1])


@pytest.mark.parametrize("kinds", [[("hy", 30, 2, 3), ("eu", 9, 7, 1)], [("eu", 6, 1, 4), ("hy", 5, 5, 1), ("eu", 20, 3, 2)],
                                   [("eu", 9, 4, 2)], [("hy", 120, 4, 2), ("hy", 3, 1, 1)]])
@pytest.mark.parametrize("capture", [False, True])
def test_batch_geometries_side_by_side(built, kinds, capture):
    """Batches whose geometries differ in hops and passes, or that have one only, called directly and
    as a captured graph that is replayed: (geometry, objects, hops, passes) of each view."""
    ctx = P.Context(0)
    views = []
    for i, (geometry, n, hops, _) in enumerate(kinds):
        views.append(B.View(_scene(geometry, n, hops), 300 + 17 * i, 120, 16, 70 + i))
        views[-1].allocate(ctx)
    renderer = B.BatchRenderer(ctx)
    renderer.set_views(views, [k[3] for k in kinds])
    calls = 3
    if capture:
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            renderer.render()
        for _ in range(calls):
            graph.replay()
    else:
        for _ in range(calls):
            renderer.render()
    torch.cuda.synchronize()
    renderer.check()
    for v, k in zip(views, kinds):
        canvas = P.Canvas(ctx, (v.width, v.height), v.global_seed)
        P.Render(ctx, v.scene.recipe, v.scene.hops).render_wavefront(v.buffer, canvas, calls * k[3])
        assert np.array_equal(_bits(canvas)[0], _bits(v.canvas)[0]) and np.array_equal(_bits(canvas)[1], _bits(v.canvas)[1])


def _bits(canvas):
    return canvas.image.cpu().numpy().view(np.uint32), canvas.seeds.cpu().numpy()


def _capture(render, buffer, canvas, passes, stats=None):
    """`passes` one-pass calls, captured and replayed: on a capturing stream a call has no workspace
    and runs the one-pass kernel, whatever the canvas."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            render.render(buffer, canvas, stats=stats, sync=False)
        for _ in range(passes):
            graph.replay()
        stream.synchronize()


def _plain(ctx, sc, W, H, passes):
    render, buffer, canvas = P.Render(ctx, sc.recipe, sc.hops), P.EntityBuffer(ctx, sc), P.Canvas(ctx, (W, H), 5)
    stats = torch.zeros(8, dtype=torch.int64, device=ctx.device)
    _capture(render, buffer, canvas, passes, stats)
    return _bits(canvas), stats.cpu().tolist()


@pytest.mark.parametrize("geometry,n,W,H,hops,passes", [
    ("hy", 5, 33, 7, 3, 3), ("hy", 31, 64, 32, 4, 2), ("hy", 64, 257, 129, 5, 2), ("hy", 99, 1024, 512, 3, 2),
    ("hy", 100, 1024, 512, 3, 3), ("hy", 130, 1031, 521, 4, 3), ("hy", 201, 1500, 701, 8, 1), ("hy", 140, 1021, 509, 6, 2),
    ("eu", 9, 33, 7, 3, 3), ("eu", 33, 1031, 521, 5, 2)])
def test_wavefronts_equal_one_pass_kernel(built, geometry, n, W, H, hops, passes):
    ctx = P.Context(0)
    sc = _scene(geometry, n, hops)
    want, want_stats = _plain(ctx, sc, W, H, passes)
    for flags in (0, _lib.HTC_FLAG_NO_SORT):
        render, buffer = P.Render(ctx, sc.recipe, sc.hops, flags), P.EntityBuffer(ctx, sc)
        for _ in range(2):   # the second call reuses the program's buffers
            canvas = P.Canvas(ctx, (W, H), 5)
            stats = torch.zeros(8, dtype=torch.int64, device=ctx.device)
            render.render_wavefront(buffer, canvas, passes, stats=stats)
            got = _bits(canvas)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
            assert stats.cpu().tolist() == want_stats


@pytest.mark.parametrize("hops,passes", [(4, 1), (3, 2)])   # 3 and 4 sorts per call
def test_captured_wavefronts_replay(built, hops, passes):
    ctx = P.Context(0)
    sc = _scene("hy", 130, hops)
    W, H = 1031, 521
    want, _ = _plain(ctx, sc, W, H, 4 * passes)
    render, buffer, canvas = P.Render(ctx, sc.recipe, sc.hops), P.EntityBuffer(ctx, sc), P.Canvas(ctx, (W, H), 5)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        render.render_wavefront(buffer, canvas, passes)   # reserves the program's buffers
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            render.render_wavefront(buffer, canvas, passes, sync=False)
        for _ in range(3):
            graph.replay()
        stream.synchronize()
    got = _bits(canvas)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("geometry,n,W,H,hops", [("hy", 40, 512, 288, 4), ("hy", 40, 511, 289, 4), ("hy", 130, 1031, 521, 4),
                                                ("hy", 40, 512, 288, 17), ("eu", 16, 1024, 1024, 3), ("eu", 15, 1024, 1024, 3)])
def test_one_pass_calls_on_two_streams(built, geometry, n, W, H, hops):
    """One program, one-pass and small multi-pass calls on two streams at once: each call works in
    memory of its own, and both canvases come out as on one stream (sizes around the least that
    render as wavefronts)."""
    ctx = P.Context(0)
    sc = _scene(geometry, n, hops)
    render, buffer = P.Render(ctx, sc.recipe, sc.hops), P.EntityBuffer(ctx, sc)
    canvases = [P.Canvas(ctx, (W, H), s) for s in (5, 6, 5, 6)]
    for c in canvases[2:]:
        for _ in range(4):
            render.render(buffer, c)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    small = W * H < 1 << 19 and n < 100
    for k in range(2):
        for c, stream in zip(canvases[:2], streams):
            with torch.cuda.stream(stream):
                render.render(buffer, c, sync=False)
                if small:
                    render.render_passes(buffer, c, 1, sync=False)
                else:
                    render.render(buffer, c, sync=False)
    torch.cuda.synchronize()
    for a, b in zip(canvases[:2], canvases[2:]):
        assert np.array_equal(_bits(a)[0], _bits(b)[0]) and np.array_equal(_bits(a)[1], _bits(b)[1])


@pytest.mark.parametrize("geometry,n,W,H,hops", [("hy", 130, 1031, 521, 4), ("hy", 20, 400, 300, 3), ("hy", 20, 512, 289, 3),
                                                ("eu", 20, 1200, 900, 5)])
def test_one_pass_calls_equal_one_pass_kernel(built, geometry, n, W, H, hops):
    ctx = P.Context(0)
    sc = _scene(geometry, n, hops)
    want, want_stats = _plain(ctx, sc, W, H, 3)
    render, buffer, canvas = P.Render(ctx, sc.recipe, sc.hops), P.EntityBuffer(ctx, sc), P.Canvas(ctx, (W, H), 5)
    stats = torch.zeros(8, dtype=torch.int64, device=ctx.device)
    render.render(buffer, canvas, stats=stats)
    render.render_passes(buffer, canvas, 2, stats=stats)
    got = _bits(canvas)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert stats.cpu().tolist() == want_stats


@pytest.mark.parametrize("geometry,n,W,H", [("eu", 9, 2, 262144), ("eu", 9, 3, 262141), ("eu", 3, 1, 524291), ("eu", 15, 4, 300001),
                                            ("hy", 5, 2, 262145)])
def test_canvases_of_more_rows_than_the_one_pass_kernel_takes(built, geometry, n, W, H):
    ctx = P.Context(0)
    scene = _scene(geometry, n, 3)
    render = P.Render(ctx, scene.recipe, scene.hops)
    buffer = P.EntityBuffer(ctx, scene)
    canvases = [P.Canvas(ctx, (W, H), 6) for _ in range(2)]
    render.render_passes(buffer, canvases[0], 2)
    render.render_wavefront(buffer, canvases[1], 2)
    assert np.array_equal(_bits(canvases[0])[0], _bits(canvases[1])[0]) and np.array_equal(_bits(canvases[0])[1], _bits(canvases[1])[1])
