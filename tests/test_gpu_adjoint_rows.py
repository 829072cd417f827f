"""Adjoint levels on odd, even and mixed grids, 1-D and 2-D fields: row lengths
around the 32-column groups (lone columns in and behind the last group) and
around the 8-row strips, against the FP64 oracle; the dot-product identity for
the orthogonal basis on the same shapes."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()

SHAPES = [((n,), 1) for n in (4, 5, 63, 64, 65, 66, 67, 129, 130)] + [((9, n), 2) for n in (64, 65, 66, 67, 128, 129, 130, 131)]
SHAPES += [((16, 17, 65), 2), ((17, 18, 66), 2), ((33, 16, 130), 2), ((10, 35, 131), 1), ((5, 64, 4), 1), ((8, 8, 8), 1)]


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape,L", SHAPES)
def test_adjoint_equals_the_oracle(shape, L, dt):
    from prodm_gb300 import api
    g = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dt)
    got = api.recompose_adjoint(torch.from_numpy(g).cuda(), L).cpu().numpy()
    ref = O.recompose_adjoint(g.astype(np.float64), shape, L)
    # a node sums at most 27 values of weight <= 1 in a handful of roundings per level
    tol = 4 * L * np.finfo(dt).eps * float(np.abs(ref).max())
    assert np.max(np.abs(got.astype(np.float64) - ref)) <= tol


@pytest.mark.parametrize("shape,L", SHAPES)
def test_orthogonal_dot_product(shape, L):
    from prodm_gb300 import api
    rng = np.random.default_rng(sum(shape) + 1)
    c = torch.from_numpy(rng.standard_normal(int(np.prod(shape)))).cuda()
    g = torch.from_numpy(rng.standard_normal(shape)).cuda()
    f = api.recompose_packed(c, shape, L, basis="orthogonal")
    h = api.recompose_adjoint(g, L, basis="orthogonal")
    assert abs(float((f * g).sum() - (c * h).sum())) <= 1e-11 * float((f * g).abs().sum() + (c * h).abs().sum())
