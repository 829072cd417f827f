"""Grouped and per-bit handles encode and decode all levels of a field in one
launch: the streams of every level equal the oracle's encoder on the level's
coefficients, and a retrieval equals the single-level decoders' values
recomposed; level sizes around the kernels' chunks (256 blocks, 128 groups)
and levels smaller than a block among them."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()

SHAPES = [((9, 9, 9), 1), ((8190,), 3), ((16386,), 5), ((92, 91), 4), ((21, 20, 22), 2), ((65, 33, 40), 3), ((5, 6, 7), 0)]


@pytest.mark.parametrize("enc,dt,B", [("grouped", np.float32, 32), ("grouped", np.float64, 60), ("grouped", np.float32, 9),
                                      ("perbit", np.float64, 60), ("perbit", np.float32, 32), ("perbit", np.float64, 20)])
@pytest.mark.parametrize("shape,L", SHAPES)
def test_levels_in_one_launch_equal_single_levels(shape, L, enc, dt, B):
    from prodm_gb300 import api
    tdt = torch.float32 if dt is np.float32 else torch.float64
    rng = np.random.default_rng(sum(shape) + B)
    x = np.cumsum(rng.standard_normal(shape), axis=-1).astype(dt)
    x[rng.random(shape) < 0.3] = 0
    m = api.MDRField(shape, tdt, L, B, enc)
    m.refactor(torch.from_numpy(x).cuda())
    coef = m.coefficients().cpu().numpy()
    sizes, bounds, _ = m.level_info()
    at = np.concatenate([[0], np.cumsum(m.level_elements.astype(np.int64))])
    exps, blobs = [], []
    for l in range(L + 1):
        c = coef[at[l]:at[l + 1]]
        exps.append(math.frexp(float(np.abs(c).max()))[1])
        blob, osz = (O.pb_encode(c, exps[l], B) if enc == "perbit" else O.encode(enc, c, exps[l], B)[:2])
        assert np.array_equal(sizes[l], osz)
        assert np.array_equal(m.export_level(l), blob)
        blobs.append(blob)
    for idx in ([B] * (L + 1), [0] * (L + 1), [1 + (3 * l) % B for l in range(L + 1)], [(B - 2 * l) % (B + 1) for l in range(L + 1)]):
        got = m.retrieve_planes(idx)
        dec = api.ProgressiveDecoder(enc, tdt)
        vals = []
        for l, k in enumerate(idx):
            n, nbytes = int(m.level_elements[l]), int(sizes[l][:k].astype(np.int64).sum())
            blob = torch.from_numpy(blobs[l][:max(nbytes, 1)].copy()).cuda()
            vals.append(dec.decode(blob, sizes[l][:k], n, exps[l], 0, k, l, B))
        want = api.recompose_packed(torch.cat(vals), shape, L)
        assert torch.equal(got.view(torch.uint8), want.view(torch.uint8)), idx
