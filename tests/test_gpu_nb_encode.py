"""fp32 negabinary encoder: value counts around a block, a warp's 32 blocks and
a chunk's 256, inputs at any 4-byte offset, any plane count, scales that are no
normal float, equal the oracle's streams."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


@pytest.mark.parametrize("B", [1, 7, 31, 32])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 8191, 8192, 8193, 16384, 300001])
def test_streams_equal_the_oracle(n, offset, B):
    from prodm_gb300 import api
    rng = np.random.default_rng(n + B)
    x = (rng.standard_normal(n) * 2.0 ** rng.integers(-30, 1, n)).astype(np.float32)
    whole = torch.zeros(n + 4, device="cuda")
    whole[offset:offset + n] = torch.from_numpy(x).cuda()
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("negabinary", whole[offset:offset + n], e, B)
    want, wsizes = O.encode("negabinary", x, e, B)[:2]
    assert np.array_equal(sizes, wsizes)
    assert np.array_equal(blob.cpu().numpy(), want)


@pytest.mark.parametrize("scale", [1e-39, 3e-38, 1e37])
def test_scales_without_a_normal_float(scale):
    from prodm_gb300 import api
    x = (np.random.default_rng(1).uniform(-1, 1, 5000) * scale).astype(np.float32)
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("negabinary", torch.from_numpy(x).cuda(), e, 32)
    want, _ = O.encode("negabinary", x, e, 32)[:2]
    assert np.array_equal(blob.cpu().numpy(), want)
