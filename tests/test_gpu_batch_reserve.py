"""htc_batch_set_views does not wait for the launches enqueued before it: not for view sets within an
htc_batch_reserve, and not for scenes that are larger than any before."""
import numpy as np
import pytest
import torch

from hypertrace_b200 import batch as B
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S

pytestmark = pytest.mark.gpu

W, H = 160, 96


def _views(ctx, objects, hops):
    views = []
    for i, n in enumerate(objects):
        rng = np.random.default_rng(n + i)
        scene = (S.euclidean_scene(n - 1, hops, n, camera=B.random_hom3(rng)) if i % 3 == 2 else
                 S.hyperbolic_scene(n - n // 2, n // 2, 4.0, hops, n, camera=S.random_moebius(rng, 0.5)))
        views.append(B.View(scene, W, H, 16, 50 + i))
        views[-1].allocate(ctx)
    return views


def _check(ctx, views):
    for v in views:
        canvas = P.Canvas(ctx, (v.width, v.height), v.global_seed)
        P.Render(ctx, v.scene.recipe, v.scene.hops).render(v.buffer, canvas)
        assert torch.equal(canvas.image.view(torch.int32), v.canvas.image.view(torch.int32))
        assert torch.equal(canvas.seeds, v.canvas.seeds)


@pytest.mark.parametrize("max_views,sets,reserved", [
    (8, [([20], 3), ([20, 9, 12], 5), ([290, 40, 33, 5, 7, 250, 8, 1200], 8), ([60], 2)], True),
    (1024, [([5, 6, 7], 8), ([300] * 8, 8)], True),
    (8, [([20, 30], 8), ([400, 300], 8), ([30, 1500], 8), ([20, 30], 8)], False)])
def test_set_views_does_not_wait(built, max_views, sets, reserved):
    ctx = P.Context(0)
    sets = [_views(ctx, objects, hops) for objects, hops in sets]
    warm = B.BatchRenderer(ctx, 8)   # the kernels are loaded
    warm.set_views(_views(ctx, [20, 110, 9], 3), [1] * 3)
    warm.render()
    renderer = B.BatchRenderer(ctx, max_views)
    if reserved:
        renderer.reserve(W * H * max(len(s) for s in sets), 8)
    else:
        renderer.set_views(sets[0], [1] * len(sets[0]))
        renderer.render()
    torch.cuda.synchronize()
    stream = torch.cuda.current_stream()
    torch.cuda._sleep(1 << 30)   # half a second of work for the launches below to stand behind
    for views in sets if reserved else sets[1:]:
        renderer.set_views(views, [1] * len(views))
        assert not stream.query()
        renderer.render()
        if views is sets[1]:   # its pinned staging slots are two: the third set waits for the first
            torch.cuda.synchronize()
            torch.cuda._sleep(1 << 30)
    torch.cuda.synchronize()
    renderer.check()
    for views in sets:
        _check(ctx, views)
