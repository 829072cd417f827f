"""The per-bit parse where its windows can go wrong: sign rates that jump from
group to group (true starts outside their windows), groups without unseen
elements among the others, constant and zero levels, lengths around the
128-group chunks and the 32-element groups; decoded in pieces against the
oracle's progressive decode."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


def values(kind, n, rng):
    x = rng.standard_normal(n)
    if kind == "bursts":        # runs of groups that turn significant at once
        return x * 2.0 ** -np.repeat(rng.integers(0, 24, n // 32 + 1), 32)[:n]
    if kind == "mixed":         # half of every group is significant from the start
        return np.where(rng.random(n) < 0.5, 1.0 + np.abs(x), x * 1e-6)
    if kind == "smooth":        # zero for most of the level, then noise
        return np.where(np.arange(n) < n // 2, 0.0, x * 1e-9) + (np.arange(n) == n - 1)
    if kind == "equal":
        return np.full(n, -0.75)
    return np.zeros(n)


@pytest.mark.parametrize("kind", ["bursts", "mixed", "smooth", "equal", "zero"])
@pytest.mark.parametrize("n", [31, 33, 4064, 4095, 4096, 4097, 8200, 40960, 65000])
@pytest.mark.parametrize("dt,B", [(np.float64, 60), (np.float32, 32)])
def test_parse_equals_the_oracle(kind, n, dt, B):
    from prodm_gb300 import api
    x = values(kind, n, np.random.default_rng(n)).astype(dt)
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes = O.pb_encode(x, e, B)
    offs = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])
    dev = api.ProgressiveDecoder("perbit", torch.float64 if dt is np.float64 else torch.float32)
    st = O.perbit_state(dt)
    d = torch.from_numpy(blob).cuda()
    for a, b in [(0, 3), (3, 21), (21, B)]:
        got = dev.decode(d[offs[a]:offs[b]], sizes[a:b], n, e, a, b - a, 0, B).cpu().numpy()
        ref = st.decode(blob[offs[a]:offs[b]], sizes[a:b], n, e, a, b - a, 0)
        assert np.array_equal(got.view(np.uint8), ref.view(np.uint8)), (a, b)
