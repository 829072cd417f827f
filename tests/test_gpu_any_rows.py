"""Level kernels on grids of any lengths: even dims (whose last two coarse
nodes have no odd node behind them), mixed ones, 1-D and 2-D fields. The
patch and the row kernels give the oracle's coefficients and recompositions
bit for bit, at row lengths around the 32-column groups and strips around the
8 steps; the fused finest level gives the oracle's retrieval on even rows."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()

SHAPES = [((n,), 2) for n in (8, 62, 64, 65, 66, 67, 126, 128, 129, 130, 4097, 10000)]
SHAPES += [((12, n), 2) for n in (61, 62, 63, 64, 65, 66, 126, 130)] + [((31, 9), 2), ((32, 130), 3), ((34, 200), 3)]
SHAPES += [((8, 10, 62), 1), ((9, 16, 64), 1), ((10, 17, 66), 2), ((11, 34, 65), 2), ((16, 33, 128), 2),
           ((17, 18, 130), 2), ((6, 6, 6), 1), ((7, 8, 9), 1), ((20, 36, 33), 3), ((5, 64, 12), 1)]


@pytest.mark.parametrize("mode", ["patch", "rows"])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shape,L", SHAPES)
def test_level_kernels_equal_the_oracle(shape, L, dt, mode, monkeypatch):
    from prodm_gb300 import api
    monkeypatch.setenv("PRODM_PATCH_MIN_ITEMS", "1")
    monkeypatch.setenv("PRODM_DECOMPOSE_PATCH", "1" if mode == "patch" else "0")
    x = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dt)
    m = api.MDRField(shape, torch.float32 if dt is np.float32 else torch.float64, L, 32, "negabinary")
    m.refactor(torch.from_numpy(x).cuda())
    coef = m.coefficients()
    u = O.decompose(x, shape, L)
    dims = m.level_dims
    want = np.concatenate([O.interleave(u, shape, dims[l], dims[l - 1] if l else np.zeros(len(shape), np.uint32))
                           for l in range(L + 1)])
    assert np.array_equal(coef.cpu().numpy().view(np.uint8), want.view(np.uint8))
    back = api.recompose_packed(coef, shape, L).cpu().numpy()
    assert np.array_equal(back.view(np.uint8), O.recompose_packed(want, shape, L).view(np.uint8))
    _, bounds, _ = m.level_info()
    at = np.concatenate([[0], np.cumsum(m.level_elements.astype(np.int64))])
    assert np.array_equal(bounds, [4 * float(np.abs(want[at[l]:at[l + 1]]).max()) for l in range(L + 1)])


@pytest.mark.parametrize("shape,L", [((40, 32, 62), 2), ((33, 34, 64), 2), ((36, 30, 256), 2), ((35, 33, 258), 2),
                                     ((34, 33, 300), 3), ((33, 32, 502), 2), ((1030, 66), 3), ((1026, 258), 4),
                                     ((33, 33, 1002), 2), ((1040, 1025), 4), ((34, 32, 1950), 3),
                                     ((1024, 1216), 3), ((1025, 2049), 3), ((1026, 3600), 2), ((1024, 4870), 2)])
def test_fused_level_on_even_rows_equals_the_oracle(shape, L):
    from prodm_gb300 import api
    B = 32
    x = np.cumsum(np.random.default_rng(sum(shape)).standard_normal(shape), axis=-1).astype(np.float32)
    m = api.MDRField(shape, torch.float32, L, B, "negabinary")
    m.refactor(torch.from_numpy(x).cuda())
    sizes, bounds, _ = m.level_info()
    blob = np.concatenate([m.export_level(l) for l in range(L + 1)])
    for planes in (0, 1, 2, 9, 17, 31, 32):
        idx = np.full(L + 1, planes, np.uint8)
        got = m.retrieve_planes(idx).cpu().numpy()
        ref = O.retrieve(shape, L, B, blob, sizes, bounds.astype(np.float32), idx, "negabinary", True)
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)), planes
    m.status()
