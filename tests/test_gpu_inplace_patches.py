"""In-place decomposition and recomposition through the patch kernels and by
elements: any grid lengths, 1-D to 3-D, equal the oracle's reordered box and its
recomposition bit for bit; interleaving and its inverse on the same grids."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()

SHAPES = [((n,), 2) for n in (8, 65, 66, 130)] + [((12, n), 2) for n in (62, 63, 64, 65, 66, 67, 129, 130)]
SHAPES += [((8, 10, 62), 1), ((9, 16, 64), 2), ((10, 17, 66), 2), ((17, 18, 130), 3), ((33, 34, 35), 4), ((5, 6, 7), 1)]


@pytest.mark.parametrize("items", ["1", "1000000"])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape,L", SHAPES)
def test_in_place_equals_the_oracle(shape, L, dt, items, monkeypatch):
    from prodm_gb300 import api
    monkeypatch.setenv("PRODM_PATCH_MIN_ITEMS", items)
    x = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dt)
    d = torch.from_numpy(x.copy()).cuda()
    api.decompose(d, L)
    want = O.decompose(x, shape, L)
    assert np.array_equal(d.cpu().numpy().view(np.uint8), np.asarray(want).reshape(shape).view(np.uint8))
    api.recompose(d, L)
    back = O.recompose(np.asarray(want).reshape(shape).copy(), shape, L)
    assert np.array_equal(d.cpu().numpy().view(np.uint8), np.asarray(back).reshape(shape).view(np.uint8))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("fine,coarse", [((40, 36, 31), (21, 19, 16)), ((40, 36, 32), (21, 19, 17)), ((31, 40, 129), (16, 21, 65)),
                                         ((1300, 33), (651, 17)), ((35, 40, 260), (0, 0, 0)), ((37, 41, 64), (37, 21, 33))])
def test_interleaving_by_rows_and_by_elements(fine, coarse, dt):
    from prodm_gb300 import api
    x = np.random.default_rng(sum(fine)).standard_normal(fine).astype(dt)
    want = O.interleave(x, fine, np.asarray(fine, np.uint32), np.asarray(coarse, np.uint32))
    d = torch.from_numpy(x.copy()).cuda()
    buf = api.interleave(d, fine, coarse)
    assert np.array_equal(buf.cpu().numpy().view(np.uint8), np.asarray(want).view(np.uint8))
    back = torch.from_numpy(np.full(fine, 7, dt)).cuda()
    api.reposition(buf, back, fine, coarse)
    ref = np.full(fine, 7, dt)
    corner = tuple(slice(0, c) for c in coarse)
    ref[:] = x
    if all(coarse):
        ref[corner] = 7
    assert np.array_equal(back.cpu().numpy().view(np.uint8), ref.view(np.uint8))
