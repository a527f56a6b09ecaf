"""The Euclidean scan's bounds never change the winner: tests/cull_check/eu_check.c restates them
on the CPU and runs, on every hop of sampled paths, both the full scan of the reference and the
culled scan of the kernel (adversarial mode: approximated values pushed 2^-21 relative the way that
culls more). Scenes: the workloads' (axis-aligned, spheres and a ground plane); rotated spheres
and slanted planes around the camera, at the origin, far from it (250: beyond it planes are not
culled; 10^4: beyond it nothing is), and maps whose quaternions are not of unit length."""
import os
import subprocess

import numpy as np
import pytest

from hypertrace_b200 import batch as B
from hypertrace_b200 import scene as S

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cull_check", "eu_check.c")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cull") / "eu_check")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fno-fast-math", "-o", exe, SRC, "-lm", "-lpthread"], check=True)
    return exe


def _run(exe, tmp_path, scene, pixels, seed, adversarial):
    path = tmp_path / "scene.bin"
    path.write_bytes(scene.to_bytes())
    out = subprocess.run([exe, str(path), "640", "480", str(scene.hops), str(pixels), str(seed), str(int(adversarial))],
                         check=True, capture_output=True, text=True).stdout.split()
    return int(out[1]), float(out[3]), int(out[5])


@pytest.mark.parametrize("adversarial", [False, True])
@pytest.mark.parametrize("spheres,hops", [(8, 4), (24, 8), (70, 6)])
def test_workload_scenes(checker, tmp_path, spheres, hops, adversarial):
    scene = S.euclidean_scene(spheres, hops, 40 + spheres, camera=B.random_hom3(np.random.default_rng(spheres)))
    n, exact, wrong = _run(checker, tmp_path, scene, 20000, spheres, adversarial)
    assert n > 25000 and wrong == 0
    assert exact < 3


@pytest.mark.parametrize("far,scale", [(0, 1.0), (30, 1.0), (240, 1.0), (300, 1.0), (3000, 1.0), (12000, 1.0),
                                       (0, 1.0 + 4e-6), (0, 1.01)])
def test_rotated_objects_and_slanted_planes(checker, tmp_path, far, scale):
    rng = np.random.default_rng(far + 1)
    scene = S.euclidean_scene(40, 8, 5)
    offset = far * np.array([1.0, 0.5, -0.3]) / 1.8
    quat = lambda: (lambda q: scale * q / np.linalg.norm(q))(rng.normal(size=4))
    for o in scene.objects:
        o.map = S.Hom3(o.map.shift + offset, quat() if o.shape == S.SHAPE_SPHERE else o.map.rot)
    for _ in range(4):
        scene.objects.append(S.SceneObject(S.Hom3(offset + rng.uniform(-6, 6, 3), quat()), S.SHAPE_PLANE, S.Mixture.mirror()))
    scene.camera = S.Hom3(offset, scene.camera.rot)
    n, exact, wrong = _run(checker, tmp_path, scene, 10000, 7, True)
    assert n > 20000 and wrong == 0
    if far == 0 and scale < 1.001:
        assert exact < 4
