"""The L2 correction of the orthogonal basis at lengths around its blocks: rows
around the 8-node tiles (odd and even, d' kept on chip, and through memory for
long rows and many of them), strided lines around the 4- and 8-node blocks, on
natural rows (in-place decomposition) and on packed coefficients."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()

SHAPES = [((6, 5, n), 1) for n in (5, 6, 7, 8, 13, 14, 15, 16, 17, 18, 29, 30, 31, 32, 33, 34, 49)]
SHAPES += [((5, 6, n), 1) for n in (1500, 1509, 1510, 1511, 1512, 1513, 1514, 3100, 3117, 3118, 3119)]
SHAPES += [((n, 5, 6), 1) for n in (7, 8, 9, 10, 14, 15, 16, 17, 18, 19, 33, 34)] + [((5, n, 7), 1) for n in (8, 9, 17, 18, 19)]
SHAPES += [((170, 160, 152), 1), ((40, 300), 2), ((5000,), 3), ((34, 35, 36), 3)]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape,L", SHAPES)
def test_correction_equals_the_oracle(shape, L, dt):
    from prodm_gb300 import api
    x = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dt)
    ref = O.decompose(x.astype(np.float64), shape, L, False)
    # per level and dim a value passes through a five-point sum and two contracting
    # recurrences: at most 32 roundings of values of the data's size
    tol = 3 * L * 32 * (np.finfo(dt).eps / 2) * float(np.abs(x).max())
    d = torch.from_numpy(x.copy()).cuda()
    api.decompose(d, L, "orthogonal")
    assert np.max(np.abs(d.cpu().numpy().astype(np.float64) - ref)) <= tol
    m = api.MDRField(shape, torch.float32 if dt is np.float32 else torch.float64, L, 32, "negabinary", "orthogonal")
    m.refactor(torch.from_numpy(x).cuda())
    coef, dims = m.coefficients(), m.level_dims
    want = np.concatenate([O.interleave(ref, shape, dims[l], dims[l - 1] if l else np.zeros(len(shape), np.uint32))
                           for l in range(L + 1)])
    assert np.max(np.abs(coef.cpu().numpy().astype(np.float64) - want)) <= tol
    back = api.recompose_packed(coef, shape, L, basis="orthogonal").cpu().numpy()
    assert np.max(np.abs(back.astype(np.float64) - x)) <= 4 * tol
