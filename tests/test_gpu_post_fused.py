"""The fused post kernel's FP32 power (htcuda.cu gamma_pack) must give the bytes of the separate
stages, whose power is FP64: on random radiance over the whole range of exponents, next to the
values where a byte changes (the exact threshold (k / 255)^(1 / gamma) and its neighbours), at and
around 0, 1, infinities, NaN, negative and denormal values, for the exponents a filter uses
and for those that take the FP64 path throughout."""
import ctypes

import numpy as np
import pytest
import torch

from hypertrace_b200 import _lib
from hypertrace_b200 import processing as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gamma", [1.0 / 2.2, 1.0 / 2.4, 0.1, 1.0, 2.2, 15.9, 16.0, 40.0, 0.0, -1.0])
@pytest.mark.parametrize("passes", [1, 7])
def test_fused_bytes_equal_separate_stages(built, gamma, passes):
    ctx = P.Context(0)
    rng = np.random.default_rng(int(gamma * 100) + 1000)
    values = [np.array([0.0, -0.0, 1.0, np.nextafter(np.float32(1), np.float32(0)), np.inf, -np.inf, np.nan, -1.0, 1e-45, 1e-38,
                        3.4e38], dtype=np.float32),
              rng.uniform(0, 1.2, 100000).astype(np.float32), np.exp2(rng.uniform(-30, 2, 100000)).astype(np.float32)]
    if gamma > 0:
        edge = (np.arange(1, 256) / 255.0) ** (1.0 / gamma) * passes
        for k in range(-40, 41):
            e = edge.astype(np.float32).view(np.int32) + k
            values.append(e.astype(np.int32).view(np.float32))
    x = np.concatenate(values)
    x = np.concatenate([x, np.zeros(-len(x) % 4, np.float32)])
    n = len(x) // 4
    canvas = torch.from_numpy(x).to(ctx.device)
    a, b, image = (torch.empty(4 * n, dtype=t, device=ctx.device) for t in (torch.uint8, torch.uint8, torch.float32))
    g = ctypes.c_float(gamma)
    _lib.call("htc_extract_gamma_pack", n, 1, passes, g, canvas.data_ptr(), a.data_ptr(), ctx.stream())
    _lib.call("htc_extract", n, 1, passes, canvas.data_ptr(), image.data_ptr(), ctx.stream())
    _lib.call("htc_gamma", n, 1, g, image.data_ptr(), image.data_ptr(), ctx.stream())
    _lib.call("htc_pack", n, 1, image.data_ptr(), b.data_ptr(), ctx.stream())
    assert torch.equal(a, b)
