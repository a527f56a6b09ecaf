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


def _bits(canvas):
    return canvas.image.cpu().numpy().view(np.uint32), canvas.seeds.cpu().numpy()


def _plain(ctx, sc, W, H, passes):
    render, buffer, canvas = P.Render(ctx, sc.recipe, sc.hops), P.EntityBuffer(ctx, sc), P.Canvas(ctx, (W, H), 5)
    stats = torch.zeros(8, dtype=torch.int64, device=ctx.device)
    for _ in range(passes):
        render.render(buffer, canvas, stats=stats)
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
