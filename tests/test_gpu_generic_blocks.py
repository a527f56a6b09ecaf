"""Block shapes and scan forms of the generic scene programs (ht_generic.cuh render_generic): the
hearth scene type compiled generically must give the hand-written kernel's bits on canvases
that tiles fit, overhang or cannot cover, and for object counts below, at and above the sizes
at which the scan stages distance bounds (32 to 256 elements)."""
import numpy as np
import pytest
import torch

from hypertrace_b200 import _lib
from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S
from hypertrace_b200 import types as T

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hearth(built):
    return {}


def _render(render, data, W, H, passes, seed):
    ctx = render.context
    scene = P.EntityBuffer(ctx, data)
    canvas = P.Canvas(ctx, (W, H), seed)
    stats = torch.zeros(8, dtype=torch.int64, device=ctx.device)
    render.render_passes(scene, canvas, passes, stats=stats)
    return canvas.image.cpu().numpy(), canvas.seeds.cpu().numpy(), stats.cpu().tolist()


@pytest.mark.parametrize("W,H", [(1, 1), (1, 37), (33, 7), (640, 16), (129, 65), (320, 240), (1003, 301)])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 257])
def test_generic_hearth_equals_handwritten(hearth, W, H, n):
    if n == 257 and W * H > 40000:
        pytest.skip("one canvas size covers the unstaged scan")
    ctx = P.Context(0)
    horo = (2 * n) // 3
    scene = S.hyperbolic_scene(n - horo, horo, 3.0, 5, 700 + n, camera=S.random_moebius(np.random.default_rng(n), 0.5))
    data = scene.to_bytes()
    hand = _render(P.Render(ctx, scene.recipe, scene.hops), data, W, H, 3, n)
    if "render" not in hearth:
        hearth["render"] = P.Render.build(ctx, T.hearth_type(), scene.hops)
    got = _render(hearth["render"], data, W, H, 3, n)
    assert np.array_equal(got[0].view(np.uint32), hand[0].view(np.uint32))
    assert np.array_equal(got[1], hand[1])
    for k in (0, 1, 3):   # samples, hops, hits
        assert got[2][k] == hand[2][k]


@pytest.mark.parametrize("W,H", [(1, 37), (33, 7), (640, 16), (129, 65)])
@pytest.mark.parametrize("recipe", [_lib.HTC_RECIPE_HY_TILED, _lib.HTC_RECIPE_EU_GRADIENT])
def test_example_passes_equal_single_passes(built, recipe, W, H):
    ctx = P.Context(0)
    if recipe == _lib.HTC_RECIPE_HY_TILED:
        data = T.serialize(T.hy_tiled_type(), T.hy_tiled_random_value(5, 40, 3.0))
    else:
        data = T.serialize(T.eu_gradient_type(), T.eu_gradient_random_value(5, 6))
    render = P.Render(ctx, recipe, 4)
    a = _render(render, data, W, H, 4, 9)
    scene, canvas = P.EntityBuffer(ctx, data), P.Canvas(ctx, (W, H), 9)
    for _ in range(4):
        render.render(scene, canvas)
    assert np.array_equal(a[0].view(np.uint32), canvas.image.cpu().numpy().view(np.uint32))
    assert np.array_equal(a[1], canvas.seeds.cpu().numpy())
    assert a[2][0] == 4 * W * H


@pytest.mark.parametrize("W,H", [(64, 64), (333, 77)])
def test_vector_below_a_mapped_object(built, W, H):
    """A vector that is not the scene's top-level object has no staged bounds and takes no test of a
    whole warp: under an identity map it finds what the same vector at the top finds. One hop: the
    map moves a ray by its last bits, so only pixels within some 1e-6 of an object's edge may differ."""
    ctx = P.Context(0)
    scene = S.hyperbolic_scene(14, 26, 3.0, 1, 77, camera=S.random_moebius(np.random.default_rng(7), 0.5))
    flat = T.hearth_type()
    vector = T.ObjectVec("Hy", T.MappedObject("Hy", T.Covered("Hy", T.ShapeChoice("Hy", ("Plane", T.PlaneHy()), ("Horosphere", T.Horosphere())),
                                                              T.hearth_material()), T.Moebius()))
    nested = T.SceneImpl("Hy", T.MappedView("Hy", T.PointView("Hy"), T.Moebius()), T.MappedObject("Hy", vector, T.Moebius()), T.ConstBg())
    value = T.hearth_value(scene)
    below = dict(value, object={"map": np.array([[1, 0], [0, 1]], dtype=np.complex128), "inner": value["object"]})
    a = _render(P.Render.build(ctx, flat, 1), T.serialize(flat, value), W, H, 2, 3)
    b = _render(P.Render.build(ctx, nested, 1), T.serialize(nested, below), W, H, 2, 3)
    assert b[2][0] == a[2][0] == 2 * W * H
    same = (a[0].view(np.uint32).reshape(-1, 4) == b[0].view(np.uint32).reshape(-1, 4)).all(axis=1)
    assert same.mean() >= 0.999 and (a[1] == b[1]).mean() >= 0.999
