"""The warp pre-cull of the hyperbolic scans (ht_bound.cuh warp_survivors) drops a slot only if every lane's own
point test drops it too, in float arithmetic: tests/cull_check/warp_scan_check.c restates both on the
present records and allowances and checks them on warps of 8 x 4 pixels, on later hops in queue order and sorted,
and on tight warps, where the slack of 2^-16 is all that lies between the two tests. With a slack of 2^-20 on
the wrong side the check finds violations there. CPU only."""
import os
import subprocess

import numpy as np
import pytest

from hypertrace_b200 import scene as S

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cull_check", "warp_scan_check.c")


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("warp") / "warp_scan_check")
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fno-fast-math", "-o", exe, SRC, "-lm", "-lpthread"], check=True)
    return exe


def _run(exe, tmp_path, scene, W, H, tiles, seed, slack):
    path = tmp_path / "scene.bin"
    path.write_bytes(scene.to_bytes())
    out = subprocess.run([exe, str(path), str(W), str(H), str(scene.hops), str(tiles), str(seed & 0xFFFFFFFF), str(slack)],
                         check=True, capture_output=True, text=True).stdout.split()
    return {out[i]: int(out[i + 1]) for i in range(0, len(out), 2)}


def _scene(n):
    if n is None:
        wl = S.config2()
        return wl.scene, wl.width, wl.height, wl.global_seed
    rng = np.random.default_rng(n)
    return S.hyperbolic_scene(n - n // 2, n // 2, 6.0, 8, 800 + n, camera=S.random_moebius(rng, 1.0)), 1280, 720, n


@pytest.mark.parametrize("n", [None, 5, 33, 130, 290])
def test_what_a_warp_culls_every_lane_culls(checker, tmp_path, n):
    v = _run(checker, tmp_path, *_scene(n)[:3], 150, _scene(n)[3], 1.0)
    assert v["violations"] == 0 and v["tight_violations"] == 0
    assert v["warps"] > 300 and v["tight_warps"] > 300
    assert v["culled"] > (0.3 if n is None or n > 33 else 0.0) * v["slots"]   # the warp test is doing work


def test_the_check_sees_a_slack_of_the_wrong_sign(checker, tmp_path):
    v = _run(checker, tmp_path, *_scene(None)[:3], 150, _scene(None)[3], -1.0 / 16)
    assert v["tight_violations"] > 0
