"""One program used from several streams and threads: what its calls share may not reach their results."""
import threading

import numpy as np
import pytest
import torch

from hypertrace_b200 import batch as B
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S

pytestmark = pytest.mark.gpu


def _scene(geometry, n, hops, seed):
    rng = np.random.default_rng(seed)
    if geometry == "eu":
        return S.euclidean_scene(n - 1, hops, seed, camera=B.random_hom3(rng))
    horo = n // 2
    return S.hyperbolic_scene(n - horo, horo, 3.0, hops, seed, camera=S.random_moebius(rng, 0.5))


def _same(a, b):
    return torch.equal(a.image.view(torch.int32), b.image.view(torch.int32)) and torch.equal(a.seeds, b.seeds)


# canvases of the one-pass kernel and of the pooled wavefronts
@pytest.mark.parametrize("geometry,W,H", [("hy", 200, 150), ("hy", 512, 288), ("eu", 200, 150), ("eu", 1024, 768)])
@pytest.mark.parametrize("threads", [False, True])
def test_double_support_scenes_on_two_streams(built, geometry, W, H, threads):
    """Two scenes of a double_support program on two streams, the second one larger (its narrowed bytes
    need a larger buffer) and enqueued while passes over the first are still to run: each canvas is
    that of its own scene."""
    ctx = P.Context(0, P.Config(double_support=True))
    buffers = [P.EntityBuffer(ctx, _scene(geometry, n, 4, 30 + n)) for n in (17, 30)]
    recipe = _scene(geometry, 17, 4, 47).recipe
    want = [P.Canvas(ctx, (W, H), 5) for _ in buffers]
    alone = P.Render(ctx, recipe, 4)
    for buffer, canvas in zip(buffers, want):
        for _ in range(3):
            alone.render_passes(buffer, canvas, 8)
    render, got = P.Render(ctx, recipe, 4), [P.Canvas(ctx, (W, H), 5) for _ in buffers]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in buffers]

    def calls(i):
        with torch.cuda.stream(streams[i]):
            render.render_passes(buffers[i], got[i], 8, sync=False)

    for _ in range(3):
        if threads:
            workers = [threading.Thread(target=calls, args=(i,)) for i in range(2)]
            for w in workers:
                w.start()
            for w in workers:
                w.join()
        else:
            calls(0)
            calls(1)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert _same(a, b)
