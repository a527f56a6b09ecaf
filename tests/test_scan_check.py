"""The hyperbolic scan's bounds never change the winner: tests/cull_check/scan_check.c restates them
on the CPU (allowances by each map's conditioning, slots by distance from the camera, estimate
over six planes and six horospheres) and runs, on every hop of sampled paths, both the full scan of
the reference and the culled scan of the kernel; they must pick the same object at the same
distance. Scenes: the headline frame, random ones of every object count of the workloads,
and far-flung maps (translations up to 6.8, the largest entries a record is made for) seen from
cameras deep in the scene, where the reference's own rounding is largest. In adversarial mode
values taken from PTX approximations are pushed 2^-21 relative the way that culls more; the
margins also hold with room to spare at a quarter of their size."""
import os
import subprocess

import numpy as np
import pytest

from hypertrace_b200 import scene as S

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cull_check", "scan_check.c")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("cull") / "scan_check")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fno-fast-math", "-o", exe, SRC, "-lm", "-lpthread"], check=True)
    return exe


def _run(exe, tmp_path, scene, W, H, pixels, seed, adversarial, tighten=1.0):
    path = tmp_path / "scene.bin"
    path.write_bytes(scene.to_bytes())
    out = subprocess.run([exe, str(path), str(W), str(H), str(scene.hops), str(pixels), str(seed & 0xFFFFFFFF),
                          str(int(adversarial)), str(tighten)], check=True, capture_output=True, text=True).stdout.split()
    return int(out[1]), float(out[3]), int(out[5])


@pytest.mark.parametrize("adversarial,tighten", [(False, 1.0), (True, 1.0), (True, 0.25)])
def test_headline_frame(checker, tmp_path, adversarial, tighten):
    wl = S.config2()
    hops, exact, wrong = _run(checker, tmp_path, wl.scene, wl.width, wl.height, 4000, wl.global_seed, adversarial, tighten)
    assert hops > 15000 and wrong == 0
    assert exact < 2.4


@pytest.mark.parametrize("n,far,camera", [(1, 3.0, 0.5), (2, 3.0, 0.5), (18, 3.0, 0.5), (33, 2.0, 1.0), (77, 6.0, 0.5),
                                          (120, 6.8, 3.0), (200, 6.0, 0.5), (290, 6.8, 5.0)])
def test_random_scenes(checker, tmp_path, n, far, camera):
    rng = np.random.default_rng(n)
    horo = int(round(n * rng.uniform(0.2, 0.8)))
    scene = S.hyperbolic_scene(n - horo, horo, far, 8, 300 + n, camera=S.random_moebius(rng, camera))
    hops, exact, wrong = _run(checker, tmp_path, scene, 640, 480, 2500, n, True)
    assert hops >= 2500 and wrong == 0
    assert exact < 6
