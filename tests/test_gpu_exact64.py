"""Division and square root on the integer pipes: the QoI values and estimates
equal IEEE arithmetic bit for bit, over significands at and next to the ends of
their range and with long runs of zeros and ones, quotients and roots next to
a halfway point, all exponents, zeros, subnormals, infinities and NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
R, G, MU, TR, S = 287.1, 1.4, 1.716e-5, 273.15, 110.4
SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2e-308, 2.2250738585072014e-308, 1.7976931348623157e308,
                    8.9e307, 9e307, 1.0, -1.0, 4.0, 2.0, 1e-160, 1e160])


def hard(n, rng, lo=1, hi=2047):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = rng.integers(0, 52, n).astype(np.uint64)
    one, ones = np.uint64(1), np.uint64((1 << 52) - 1)
    kind = rng.integers(0, 6, n)
    m = np.where(kind == 1, ones - (m & np.uint64(15)), m)
    m = np.where(kind == 2, m & np.uint64(15), m)
    m = np.where(kind == 3, m & ~((one << k) - one), m)
    m = np.where(kind == 4, m | ((one << k) - one), m)
    m = np.where(kind == 5, m >> k, m)
    e = rng.integers(lo, hi, n).astype(np.uint64)
    return ((e << np.uint64(52)) | m).view(np.float64)


def fields(kind, n, rng):
    near = kind != "wide"
    f = [hard(n, rng, 1000 if near else 1, 1046 if near else 2047) * rng.choice([-1.0, 1.0], n) for _ in range(5)]
    if kind == "squares":      # one component only, its square a unit or two off: roots next to halfway points
        f[0] = np.nextafter(f[0], f[0] * rng.choice([0.0, 2.0], n))
        f[1][:], f[2][:] = 0.0, 0.0
        f[3] = f[3] * (np.abs(f[4]) * R)      # quotients next to short ones
        f[3] = np.where(rng.random(n) < 0.5, np.nextafter(f[3], np.inf), f[3])
    if kind == "special":
        for a in f:
            at = rng.random(n) < 0.5
            a[at] = rng.choice(SPECIAL, int(at.sum()))
    return f


def same(got, want):
    got = got.cpu().numpy()
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got.view(np.uint64)[~nan], want.view(np.uint64)[~nan])


def bx2(x, eb):
    return 2.0 * np.abs(x) * eb + eb * eb


@pytest.mark.parametrize("n", [1, 33, 1 << 18])
@pytest.mark.parametrize("kind", ["near", "wide", "squares", "special"])
def test_values_and_bounds_equal_ieee_arithmetic(kind, n):
    from prodm_gb300 import api
    rng = np.random.default_rng(n)
    vx, vy, vz, p, d = fields(kind, n, rng)
    dev = [torch.from_numpy(a.copy()).cuda() for a in (vx, vy, vz, p, d)]
    with np.errstate(all="ignore"):
        v = np.sqrt(vx * vx + vy * vy + vz * vz)
        t = p / (d * R)
        c = np.sqrt(G * R * t)
        m = v / c
        mt = 1.0 + (G - 1) / 2 * m * m
        mt2 = mt * mt
        pt = p * np.sqrt(mt2 * mt2 * mt2 * mt)
        tr = t / TR
        mu = MU * np.sqrt(tr * tr * tr) * ((TR + S) / (t + S))
        for got, want in zip(api.qoi_ge_values(*dev), (v, t, c, m, pt, mu)):
            same(got, want)
        for ebs, ebp, ebd in (((0.01, 0.0, 3.0), 10.0, 1e-4), ((1e-9, 1e-9, 1e-9), 0.0, 1e-12), ((-0.0, -0.0, -0.0), 1e3, -0.0),
                              ((1e200, 1.0, 1e-300), 1e-310, 1e250), ((np.inf, 0.0, 0.0), 1.0, np.inf)):
            e2 = bx2(vx, ebs[0]) + bx2(vy, ebs[1]) + bx2(vz, ebs[2])
            v2 = vx * vx + vy * vy + vz * vz
            bv = np.where(v2 == 0, np.sqrt(e2), np.where(v2 > e2, e2 / (np.sqrt(v2 - e2) + np.sqrt(v2)), e2 / np.sqrt(v2)))
            num = np.abs(p) * ebd + np.abs(d) * ebp
            bt = 1.0 / R * np.where(ebd < np.abs(d), num / np.where(d > 0, d * (d - ebd), d * (d + ebd)), 0.0)
            got_v, got_t, mx = api.qoi_ge_bounds(dev[:3], ebs, dev[3], dev[4], ebp, ebd)
            same(got_v, bv)
            same(got_t, bt)
            want = [float(np.max(np.where(np.isnan(b), 0.0, b))) for b in (bv, bt)]
            assert [float(x) for x in mx] == want
