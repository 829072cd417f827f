"""fp64 negabinary encoder and decoder: value counts around a block, the eight
blocks written and read together, a warp's 32 and a chunk's 256; plane counts
on both sides of 32; whole and partial decodes; equal the oracle's streams and
values bit for bit, and scales whose values leave the fixed-point range."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


@pytest.mark.parametrize("B", [1, 4, 31, 32, 33, 59, 60])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 448, 511, 512, 513, 2047, 2048, 2049, 16383, 16384, 16385, 100000])
def test_streams_and_values_equal_the_oracle(n, B):
    from prodm_gb300 import api
    rng = np.random.default_rng(n + B)
    x = rng.standard_normal(n) * 2.0 ** rng.integers(-70, 1, n)
    x[rng.random(n) < 0.1] = 0
    x[0] = -1.5
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("negabinary", torch.from_numpy(x).cuda(), e, B)
    want, wsizes = O.encode("negabinary", x, e, B)[:2]
    assert np.array_equal(sizes, wsizes)
    assert np.array_equal(blob.cpu().numpy(), want)
    at = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])
    for s, k in ((0, B), (0, (B + 1) // 2), (B // 3, B - B // 3)):
        if k == 0:
            continue
        dec = api.ProgressiveDecoder("negabinary", torch.float64)
        part = want[at[s]:at[s + k]]
        got = dec.decode(torch.from_numpy(np.append(part, np.zeros(8, np.uint8))).cuda(), sizes[s:s + k], n, e, s, k, 0, B)
        ref = O.nb_decode(part, sizes[s:s + k], n, e, s, k, np.float64)
        assert np.array_equal(got.cpu().numpy().view(np.uint64), np.asarray(ref).view(np.uint64)), (s, k)


@pytest.mark.parametrize("scale", [5e-324 * 2 ** 20, 1e-300, 1e300])
def test_extreme_scales(scale):
    from prodm_gb300 import api
    x = np.random.default_rng(1).uniform(-1, 1, 3000) * scale
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("negabinary", torch.from_numpy(x).cuda(), e, 60)
    want, _ = O.encode("negabinary", x, e, 60)[:2]
    assert np.array_equal(blob.cpu().numpy(), want)
    dec = api.ProgressiveDecoder("negabinary", torch.float64)
    got = dec.decode(blob, sizes, x.size, e, 0, 60, 0, 60)
    ref = O.nb_decode(want, sizes, x.size, e, 0, 60, np.float64)
    assert np.array_equal(got.cpu().numpy().view(np.uint64), np.asarray(ref).view(np.uint64))
