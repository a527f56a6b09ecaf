"""The device's pool of workspaces: a program made for a frame or two maps none, later calls take theirs
from it with the same results, and the last program gives it back."""
import gc

import numpy as np
import pytest
import torch

from hypertrace_b200 import batch as B
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S

pytestmark = pytest.mark.gpu

HOPS = 4


def _scene(geometry, n):
    rng = np.random.default_rng(n)
    if geometry == "eu":
        return S.euclidean_scene(n - 1, HOPS, n, camera=B.random_hom3(rng))
    return S.hyperbolic_scene(n - n // 2, n // 2, 4.0, HOPS, n, camera=S.random_moebius(rng, 0.5))


def _same(a, b):
    return torch.equal(a.image.view(torch.int32), b.image.view(torch.int32)) and torch.equal(a.seeds, b.seeds)


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


# the least canvases that render as wavefronts, by geometry and number of objects
@pytest.mark.parametrize("geometry,n,W,H", [("hy", 40, 512, 288), ("hy", 6, 512, 289), ("hy", 5, 1024, 768), ("eu", 16, 1024, 768)])
def test_workspace_comes_with_the_fifth_pass(built, geometry, n, W, H):
    gc.collect()   # no program of an earlier test
    ctx = P.Context(0)
    scene = _scene(geometry, n)
    buffer = P.EntityBuffer(ctx, scene)
    want, got = P.Canvas(ctx, (W, H), 7), P.Canvas(ctx, (W, H), 7)
    reference = P.Render(ctx, scene.recipe, HOPS)
    for _ in range(5):   # loads the kernels; its queues and the pool go with it
        reference.render(buffer, P.Canvas(ctx, (W, H), 1))
    reference.render_wavefront(buffer, want, 5)
    reference.render_wavefront(buffer, want, 1)
    reference.render_wavefront(buffer, want, 1)
    del reference
    torch.cuda.synchronize()
    empty = _free()
    render = P.Render(ctx, scene.recipe, HOPS)
    for _ in range(4):
        render.render(buffer, got)
    assert empty - _free() < 8 << 20   # the program itself, no workspace of 136 bytes a pixel (19 MB and more)
    render.render(buffer, got)
    assert empty - _free() >= 136 * W * H
    render.render(buffer, got)
    render.render_passes(buffer, got, 1)
    assert _same(got, want)
    del render
    assert empty - _free() < 8 << 20


def test_a_long_call_takes_its_workspace_at_once(built):
    gc.collect()
    ctx = P.Context(0)
    scene = _scene("hy", 40)
    W, H = 512, 288
    buffer, want, got = P.EntityBuffer(ctx, scene), P.Canvas(ctx, (W, H), 7), P.Canvas(ctx, (W, H), 7)
    reference = P.Render(ctx, scene.recipe, HOPS)
    reference.render_wavefront(buffer, want, 9)
    del reference
    render = P.Render(ctx, scene.recipe, HOPS)
    empty = _free()
    render.render_passes(buffer, got, 9)
    assert empty - _free() >= 136 * W * H
    assert _same(got, want)
