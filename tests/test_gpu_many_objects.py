"""Hyperbolic scenes of object counts beyond the workloads': the staging's order by distance up to 1024
objects and by index beyond (ranks by ballot), the largest scenes that shared memory stages, and the few
objects that are staged in index order too. Every form of the render agrees with the others bit for bit and
with the CPU oracle."""
import numpy as np
import pytest
import torch

from hypertrace_b200 import _lib
from hypertrace_b200 import batch as B
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S
from oracle import oracle

from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu

W, H, HOPS, PASSES = 97, 61, 5, 2


def _bits(canvas):
    return canvas.image.cpu().numpy().view(np.uint32), canvas.seeds.cpu().numpy()


@pytest.mark.parametrize("planes,horospheres", [(3, 3), (4, 3), (201, 399), (500, 524), (511, 514), (333, 1167), (1501, 0), (0, 1300),
                                                (1399, 1400)])
@pytest.mark.parametrize("address_width", [32, 64])
def test_every_form_agrees(built, planes, horospheres, address_width):
    ctx = P.Context(0, P.Config(address_width=address_width))
    rng = np.random.default_rng(planes)
    scene = S.hyperbolic_scene(planes, horospheres, 6.0, HOPS, 70 + horospheres, camera=S.random_moebius(rng, 0.5))
    buffer = P.EntityBuffer(ctx, scene)
    render = P.Render(ctx, scene.recipe, HOPS)
    canvases = [P.Canvas(ctx, (W, H), 5) for _ in range(4)]
    for _ in range(PASSES):
        render.render(buffer, canvases[0])
    render.render_wavefront(buffer, canvases[1], PASSES)
    _lib.call("htc_render_passes_noalloc", scene.recipe, HOPS, address_width, 0, W, H, buffer.ptr(), buffer.size,
              canvases[2].image.data_ptr(), canvases[2].seeds.data_ptr(), PASSES, None, None, ctx.stream())
    view = B.View(scene, W, H, 16, 5)
    view.allocate(P.Context(0))
    batch = B.BatchRenderer(P.Context(0), 2)
    batch.set_views([view], [PASSES])
    batch.render()
    batch.check()
    canvases[3] = view.canvas
    torch.cuda.synchronize()
    for canvas in canvases[1:]:
        for a, b in zip(_bits(canvases[0]), _bits(canvas)):
            assert np.array_equal(a, b)
    seeds = S.pixel_seeds(5, W * H)
    ref = oracle.render(S.serialize(scene, 32), scene.recipe, HOPS, W, H, np.arange(W * H), seeds, passes=PASSES, threads=8)
    _compare(canvases[0].image.cpu().numpy().reshape(-1, 4), canvases[0].seeds.cpu().numpy().view(np.uint32), ref,
             f"{planes} planes, {horospheres} horospheres")
