"""Adjoint level for gradients near the largest finite value and for infinities
and NaN: each value is weighted before it is added, so a result is finite where
the sum of the weighted values, node by node, is."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(5,), (66,), (131,), (9, 64), (10, 67), (17, 18, 66), (6, 35, 131), (5, 64, 4)]


def node_by_node(g):
    """The coarse gradient of one level: acc += weight * value over the values at,
    before and behind each coarse node, dim 0 outermost."""
    dt = g.dtype.type
    axes = []
    for n in g.shape:
        c = np.array([min(2 * m, n - 1) for m in range(n // 2 + 1)])
        odd = [(c >= 1) & (c - 1 < 2 * (n - c.size)) & (c % 2 == 0), c // 2 < n - c.size]
        odd[0] &= c // 2 - 1 < n - c.size
        if n % 2 == 0:
            odd[1][-1] = odd[0][-1] = False
        axes.append((c, odd))
    acc = np.zeros([c.size for c, _ in axes], g.dtype)
    offs = (0, -1, 1)
    with np.errstate(all="ignore"):
        for steps in np.ndindex(*([3] * g.ndim)):
            on = np.ones(acc.shape, bool)
            idx, w = [], dt(1)
            for d, k in enumerate(steps):
                c, odd = axes[d]
                here = np.ones(c.size, bool) if k == 0 else odd[k - 1]
                on &= here.reshape([-1 if e == d else 1 for e in range(g.ndim)])
                idx.append(np.clip(c + offs[k], 0, g.shape[d] - 1))
                w = w if k == 0 else w * dt(0.5)
            acc = np.where(on, acc + w * g[np.ix_(*idx)], acc)
    return acc


def coarse_of(g):
    from prodm_gb300 import api
    got = api.recompose_adjoint(torch.from_numpy(g).cuda(), 1).cpu().numpy()
    n = int(np.prod([k // 2 + 1 for k in g.shape]))
    return got[:n].reshape([k // 2 + 1 for k in g.shape])


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_gradients_near_the_largest_value(shape, dt):
    big = float(np.finfo(dt).max)
    x = sum(np.ix_(*[np.arange(n) for n in shape]))
    alternating = np.where(x % 2, dt(0.9 * big), dt(-0.9 * big))
    rng = np.random.default_rng(sum(shape))
    noise = (rng.uniform(0.5, 1.0, shape) * rng.choice([-1, 1], shape)).astype(dt) * dt(big)
    for g in (alternating, noise, np.full(shape, dt(big / 8))):
        got, ref = coarse_of(g), node_by_node(g)
        ok = np.isfinite(ref)
        assert np.isfinite(got[ok]).all()
        # at most 27 values of weight 8 in all, a handful of roundings
        assert np.all(np.abs(got[ok] / 32 - ref[ok] / 32) <= np.finfo(dt).eps * float(np.abs(g).max()))
        assert ok.any()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_infinities_and_nan(shape, dt):
    rng = np.random.default_rng(sum(shape) + 1)
    g = rng.standard_normal(shape).astype(dt)
    flat = g.reshape(-1)
    for k, v in enumerate((np.inf, -np.inf, np.nan, np.finfo(dt).max, -np.finfo(dt).max)):
        flat[rng.integers(0, flat.size, 1 + flat.size // 200)] = v
    got, ref = coarse_of(g), node_by_node(g)
    ok = np.isfinite(ref)
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.array_equal(got[~ok], ref[~ok], equal_nan=True)
    assert np.isfinite(got[ok]).all()
