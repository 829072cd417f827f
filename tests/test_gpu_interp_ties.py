"""Interpreter on levels whose planes tie (one-block levels of 2-D fields,
sizes in power-of-two ratios under error tables that halve per plane): the
device walks past a tied group as a unit, so its plane counts and sizes must
equal the oracle's heap walk for stops before, inside and behind such groups."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


def tables(rng, nl, B, ratio, squared):
    sizes = np.empty((nl, B), np.uint32)
    errs = np.empty((nl, B + 1))
    for l in range(nl):
        sizes[l] = max(1, int(rng.integers(1, 3)) * ratio ** l) * 4
        top = 2.0 ** float(rng.integers(-2, 3))
        errs[l, 1:] = top * 0.5 ** np.arange(B)
        errs[l, 0] = top * rng.uniform(1.0, 2.0)
    return (sizes, errs * errs) if squared else (sizes, errs)


@pytest.mark.parametrize("kind,est", [("greedy", "max_hb"), ("sign_exclude", "max_hb"), ("sign_exclude", "max_ob"),
                                      ("negabinary", "max_hb"), ("negabinary", "l2_hb")])
@pytest.mark.parametrize("nl,B,ratio,dt", [(1, 32, 2, np.float32), (2, 32, 1, np.float32), (9, 32, 4, np.float32),
                                           (11, 32, 2, np.float32), (7, 60, 8, np.float64), (17, 60, 1, np.float64)])
def test_tied_groups_equal_the_heap_walk(kind, est, nl, B, ratio, dt):
    from prodm_gb300 import api
    rng = np.random.default_rng(nl * 100 + B + ratio)
    tdt = torch.float32 if dt is np.float32 else torch.float64
    for _ in range(6):
        sizes, errs = tables(rng, nl, B, ratio, est == "l2_hb")
        idx = np.zeros(nl, np.uint8)
        for tol in sorted(float(errs[:, 0].sum()) * 10.0 ** rng.uniform(-9, 0.3, 8), reverse=True):
            want = O.interpret(kind, est, sizes, errs, tol, idx, ndims=2, dtype=dt)
            got = api.interpret(kind, est, sizes, errs, tol, idx, ndims=2, dtype=tdt)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (tol, got, want)
            idx = want[0]   # progressive: the next tolerance goes on from here
            if kind == "greedy" and idx.max() == B:
                break   # the reference's greedy walk reads past the tables of a level that is complete at its start
