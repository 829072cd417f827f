"""Kernels that only large inputs take: the grouped codecs on both sides of the
chunk counts where their launches change (fp32 decoder above 8 x 152 chunks of
8,192 values, fp64 first pass and decoder above 152 of 16,384), against the
oracle; batched fields of long rows (fused units of 8, 4, 2 and 1 rows, and rows
too long for a unit), against the single-field path."""
import math

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
O = oracle.oracle()


@pytest.mark.parametrize("dt,B,n", [(np.float32, 32, 1216 * 8192), (np.float32, 19, 1216 * 8192 + 8192 + 45),
                                    (np.float64, 60, 152 * 16384), (np.float64, 37, 152 * 16384 + 77)])
def test_grouped_codec_of_many_chunks(dt, B, n):
    from prodm_gb300 import api
    rng = np.random.default_rng(n)
    bs = 32 if dt is np.float32 else 64
    x = rng.uniform(0.5, 1, n) * rng.choice([-1.0, 1.0], n)
    x = (x * np.repeat(2.0 ** -rng.integers(0, B + 6, n // bs + 1), bs)[:n]).astype(dt)
    e = math.frexp(float(np.abs(x).max()))[1]
    blob, sizes, _ = api.encode("grouped", torch.from_numpy(x).cuda(), e, B)
    want, wsizes = O.encode("grouped", x, e, B)[:2]
    assert np.array_equal(sizes, wsizes)
    assert np.array_equal(blob.cpu().numpy(), want)
    at = np.concatenate([[0], np.cumsum(sizes.astype(np.int64))])
    for parts in ((0, B), (0, B // 3, B)):
        dec = api.ProgressiveDecoder("grouped", torch.float32 if dt is np.float32 else torch.float64)
        ref = O.grouped_state(dt)
        for s, k in zip(parts, np.diff(parts).tolist()):
            part = want[at[s]:at[s + k]]
            got = dec.decode(torch.from_numpy(np.append(part, np.uint8(0))).cuda(), sizes[s:s + k], n, e, s, k, 0, B)
            exp = ref.decode(part, sizes[s:s + k], n, e, s, k, 0)
            assert np.array_equal(got.cpu().numpy().view(np.uint8), np.asarray(exp).view(np.uint8)), (s, k)


@pytest.mark.parametrize("ws", ["1", "0"])
def test_batched_fields_of_long_rows(ws, monkeypatch):
    from prodm_gb300 import api, fields
    monkeypatch.setenv("PRODM_BATCH_WS", ws)
    shapes = [(20, 607), (12, 1216), (20, 1217), (9, 7, 1300), (20, 2049), (15, 2432), (17, 2500), (20, 3600), (6, 4801),
              (6, 5000), (5, 6, 5001), (33, 65)]
    xs = [fields.spectral_grf(s, slope=-2.0, seed=80 + i).contiguous() for i, s in enumerate(shapes)]
    levels = [fields.batch_level(s, api.max_level(s)) for s in shapes]
    batch = api.MDRBatch(xs, levels, 32)
    batch.refactor()
    for digits in (1, 4):
        tols = [float(x.max() - x.min()) * 10.0 ** (-digits - i % 3) for i, x in enumerate(xs)]
        batch.set_tolerances(tols)
        batch.reset()
        outs = batch.retrieve("negabinary", "max_hb")
        torch.cuda.synchronize()
        batch.status()
        for i, (s, x) in enumerate(zip(shapes, xs)):
            one = api.MDRField(s, torch.float32, levels[i], 32, "negabinary", "hierarchical", "max")
            one.refactor(x)
            for l in range(levels[i] + 1):
                assert np.array_equal(batch.export_level(i, l), one.export_level(l)), (s, l)
            assert torch.equal(one.retrieve(tols[i], interpreter="negabinary", estimator="max_hb"), outs[i]), s
