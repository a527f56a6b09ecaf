"""Stream capture beside other calls: what a captured call needs is there after any earlier call on a canvas
as large, whatever that call's scene, and later calls leave a captured graph's memory alone."""
import numpy as np
import pytest
import torch

from hypertrace_b200 import processing as P
from hypertrace_b200 import scene as S

pytestmark = pytest.mark.gpu

W, H, HOPS = 1031, 521, 3   # above the least sorted canvas (2^19 pixels)


def _scene(n):
    rng = np.random.default_rng(n)
    horo = n // 2
    return S.hyperbolic_scene(n - horo, horo, 5.0, HOPS, 60 + n, camera=S.random_moebius(rng, 0.5))


def _same(a, b):
    return torch.equal(a.image.view(torch.int32), b.image.view(torch.int32)) and torch.equal(a.seeds, b.seeds)


def _want(ctx, buffer, recipe, passes):
    canvas = P.Canvas(ctx, (W, H), 5)
    P.Render(ctx, recipe, HOPS).render_passes(buffer, canvas, passes)
    return canvas


@pytest.mark.parametrize("first,captured", [(40, 150), (150, 40), (40, 99), (120, 700)])
def test_capture_after_a_call_with_another_scene(built, first, captured):
    ctx = P.Context(0)
    scenes = [_scene(first), _scene(captured)]
    buffers = [P.EntityBuffer(ctx, s) for s in scenes]
    want = [_want(ctx, b, scenes[0].recipe, 4) for b in buffers]
    render, canvases = P.Render(ctx, scenes[0].recipe, HOPS), [P.Canvas(ctx, (W, H), 5) for _ in buffers]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        render.render_passes(buffers[0], canvases[0], 2)
        with torch.cuda.graph(graph, stream=stream):
            render.render_passes(buffers[1], canvases[1], 2, sync=False)
        graph.replay()
        render.render_passes(buffers[0], canvases[0], 2)   # with the first scene again
        graph.replay()
        stream.synchronize()
    for a, b in zip(canvases, want):
        assert _same(a, b)
    torch.cuda.synchronize()


@pytest.mark.parametrize("first", [30, 120])   # a captured call in queue order, one that sorts
def test_graph_survives_a_call_with_a_larger_scene(built, first):
    ctx = P.Context(0)
    scenes = [_scene(first), _scene(150), _scene(900)]
    buffers = [P.EntityBuffer(ctx, s) for s in scenes]
    want = [_want(ctx, b, scenes[0].recipe, 2) for b in buffers]
    render, canvases = P.Render(ctx, scenes[0].recipe, HOPS), [P.Canvas(ctx, (W, H), 5) for _ in buffers]
    spare = P.Canvas(ctx, (W, H), 5)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        render.render_passes(buffers[0], spare, 1)
        with torch.cuda.graph(graph, stream=stream):
            render.render_passes(buffers[0], canvases[0], 1, sync=False)
        for k in (1, 2):
            render.render_passes(buffers[k], canvases[k], 2)
            graph.replay()
        stream.synchronize()
    for a, b in zip(canvases, want):
        assert _same(a, b)


@pytest.mark.parametrize("earlier", [None, 9])
def test_captured_call_without_queues(built, earlier):
    """A captured multi-pass call of a size that uses the program's queues, on a program that has none: new,
    or whose earlier call on that canvas ran the one-pass kernel for its few objects."""
    ctx = P.Context(0)
    size = (1024, 640)
    scenes = [S.euclidean_scene(n - 1, HOPS, n) for n in (20, earlier or 20)]
    buffers = [P.EntityBuffer(ctx, s) for s in scenes]
    want, got = P.Canvas(ctx, size, 5), P.Canvas(ctx, size, 5)
    P.Render(ctx, scenes[0].recipe, HOPS).render_passes(buffers[0], want, 4)
    render = P.Render(ctx, scenes[0].recipe, HOPS)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        if earlier:
            render.render_passes(buffers[1], P.Canvas(ctx, size, 5), 1)
        with torch.cuda.graph(graph, stream=stream):
            render.render_passes(buffers[0], got, 2, sync=False)
        graph.replay()
        graph.replay()
        stream.synchronize()
    assert _same(got, want)


@pytest.mark.parametrize("size", [(200, 150), (512, 288), (1031, 521)])
@pytest.mark.parametrize("earlier_call", [False, True])
def test_one_pass_call_on_another_stream_while_one_captures(built, size, earlier_call):
    """The capture forbids calls that might disturb it, on every stream and thread (the global mode, torch's
    default): a one-pass call on a stream of its own is none, whatever workspace it takes."""
    ctx = P.Context(0)
    scene = _scene(40)
    buffer = P.EntityBuffer(ctx, scene)
    want = P.Canvas(ctx, size, 5)
    captured, beside = P.Canvas(ctx, size, 5), P.Canvas(ctx, size, 5)
    reference = P.Render(ctx, scene.recipe, HOPS)
    for _ in range(2):
        reference.render(buffer, want)
    del reference   # the device has no program, and no pool, but this one's
    render = P.Render(ctx, scene.recipe, HOPS)
    if earlier_call:
        render.render(buffer, P.Canvas(ctx, size, 5))
    streams, graph = [torch.cuda.Stream(), torch.cuda.Stream()], torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=streams[0]):
        render.render(buffer, captured, sync=False)
        with torch.cuda.stream(streams[1]):
            render.render(buffer, beside, sync=False)
            render.render(buffer, beside, sync=False)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for canvas in (captured, beside):
        assert _same(canvas, want)
