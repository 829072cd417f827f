"""Per-bit export: the streams of fields around the warps' 32 groups and the
chunks' 256, with elements that all start in one plane, never start, or start
anywhere, and plane counts around the ten loaded at a time, equal the oracle's."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


@pytest.mark.parametrize("dt,B", [(np.float64, 1), (np.float64, 9), (np.float64, 10), (np.float64, 11), (np.float64, 32),
                                  (np.float64, 33), (np.float64, 60), (np.float32, 20), (np.float32, 31), (np.float32, 32)])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 8191, 8192, 8193, 16384 + 37, 270000])
@pytest.mark.parametrize("kind", ["same", "spread", "sparse"])
def test_streams_equal_the_oracle(kind, n, dt, B):
    from prodm_gb300 import api
    rng = np.random.default_rng(n + B)
    x = rng.uniform(0.5, 1, n) * rng.choice([-1.0, 1.0], n)
    if kind == "spread":
        x *= 2.0 ** -rng.integers(0, 64, n)
    elif kind == "sparse":
        x[rng.random(n) < 0.9] = 0
        x[0] = -0.75
    x = x.astype(dt)
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("perbit", torch.from_numpy(x).cuda(), e, B)
    want, wsizes = O.pb_encode(x, e, B)
    assert np.array_equal(sizes, wsizes)
    assert np.array_equal(blob.cpu().numpy(), want)
