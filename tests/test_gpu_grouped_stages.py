"""Grouped writer and decoder around their groups of blocks: block counts about
the 8 and 16 blocks whose words leave together, blocks that all start in one
plane (two words a block there) or start everywhere, plane counts that are no
multiple of the rows written together, on both sides of 32."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


def data(kind, n, bs, rng, dt):
    x = rng.uniform(0.5, 1, n) * rng.choice([-1.0, 1.0], n)
    if kind == "spread":      # blocks start in any plane, some nowhere
        x *= np.repeat(2.0 ** -rng.integers(0, 66, (n + bs - 1) // bs), bs)[:n]
    elif kind == "runs":      # eight blocks of a size, then eight others
        x *= np.where(np.arange(n) // (8 * bs) % 2, 1.0, 2.0 ** -3)
    return x.astype(dt)


@pytest.mark.parametrize("kind", ["same", "spread", "runs"])
@pytest.mark.parametrize("dt,B", [(np.float32, 2), (np.float32, 5), (np.float32, 31), (np.float32, 32), (np.float64, 7),
                                  (np.float64, 32), (np.float64, 33), (np.float64, 59), (np.float64, 60)])
@pytest.mark.parametrize("blocks,extra", [(1, -3), (7, 0), (8, 1), (15, 0), (16, 0), (17, -1), (31, 0), (32, 5), (40, 0),
                                          (255, 0), (256, 1), (530, -7)])
def test_streams_and_values_equal_the_oracle(blocks, extra, dt, B, kind):
    from prodm_gb300 import api
    bs = 32 if dt is np.float32 else 64
    n = blocks * bs + extra
    x = data(kind, n, bs, np.random.default_rng(n + B), dt)
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("grouped", torch.from_numpy(x).cuda(), e, B)
    want, wsizes = O.encode("grouped", x, e, B)[:2]
    assert np.array_equal(sizes, wsizes)
    assert np.array_equal(blob.cpu().numpy(), want)
    at = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])
    dec, ref = api.ProgressiveDecoder("grouped", torch.float32 if dt is np.float32 else torch.float64), O.grouped_state(dt)
    for s, k in ((0, (B + 1) // 3), ((B + 1) // 3, B - (B + 1) // 3)):
        part = want[at[s]:at[s + k]]
        got = dec.decode(torch.from_numpy(np.append(part, np.uint8(0))).cuda(), sizes[s:s + k], n, e, s, k, 0, B)
        exp = ref.decode(part, sizes[s:s + k], n, e, s, k, 0)
        assert np.array_equal(got.cpu().numpy().view(np.uint8), np.asarray(exp).view(np.uint8)), (s, k)
