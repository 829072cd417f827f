"""Calls that bring tables made on the host: a stream capture refuses them before
anything is queued (no graph keeps the address of a table that is gone, and no
state of a handle runs ahead of its device), the tables arrive whole at every
size of their transport, and calls queued behind one another without a wait do
not see each other's."""
import numpy as np
import pytest
import torch

import oracle
from stream_capture import Capture

pytestmark = pytest.mark.gpu
O = oracle.oracle()
EUNSUPPORTED = 6


def refused(stream, call):
    from prodm_gb300 import _lib
    with Capture(stream) as c:
        with pytest.raises(_lib.ProdmError) as e:
            call()
    assert e.value.status == EUNSUPPORTED and c.status == 0
    c.close()


def noise(shape, dt, seed):
    return torch.randn(shape, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("dt", [torch.float32, torch.float64])
def test_orthogonal_basis_refuses_capture(dt):
    from prodm_gb300 import api
    shape, L = (17, 20, 33), 2
    side = torch.cuda.Stream()
    x = noise(shape, dt, 1)
    y = x.clone()
    for f in (api.decompose, api.recompose):
        want = y.clone()
        f(want, L, "orthogonal")
        refused(side, lambda: f(y, L, "orthogonal", stream=side))
        f(y, L, "orthogonal")
        assert torch.equal(y, want)
    for f, arg in ((lambda a, **k: api.recompose_packed(a, shape, L, basis="orthogonal", **k), x.reshape(-1)),
                   (lambda a, **k: api.recompose_adjoint(a, L, basis="orthogonal", **k), x)):
        want, out = f(arg), torch.empty_like(x).reshape(-1)
        refused(side, lambda: f(arg, out=out, stream=side))
        assert torch.equal(f(arg), want)


@pytest.mark.parametrize("enc,dt,B", [("grouped", torch.float32, 32), ("grouped", torch.float64, 50),
                                      ("perbit", torch.float64, 40)])
def test_progressive_decode_refuses_capture(enc, dt, B):
    from prodm_gb300 import api
    n, side = 5000, torch.cuda.Stream()
    blob, sizes, _ = api.encode(enc, noise(n, dt, 2), 4, B)
    cut = int(np.asarray(sizes[:9], np.int64).sum())
    d, e = (api.ProgressiveDecoder(enc, dt) for _ in range(2))
    refused(side, lambda: d.decode(blob, sizes, n, 4, 0, 9, 0, B, stream=side))
    assert torch.equal(d.decode(blob, sizes, n, 4, 0, 9, 0, B), e.decode(blob, sizes, n, 4, 0, 9, 0, B))
    rest = blob[cut:].clone()
    refused(side, lambda: d.decode(rest, sizes[9:], n, 4, 9, B - 9, 0, B, stream=side))
    assert torch.equal(d.decode(rest, sizes[9:], n, 4, 9, B - 9, 0, B), e.decode(rest, sizes[9:], n, 4, 9, B - 9, 0, B))


@pytest.mark.parametrize("enc,dt,B", [("grouped", torch.float32, 32), ("grouped", torch.float64, 50),
                                      ("perbit", torch.float64, 40)])
def test_loaded_files_unpack_outside_a_capture(enc, dt, B):
    from prodm_gb300 import api
    shape, L = (17, 20, 33), 2
    side = torch.cuda.Stream()
    x = noise(shape, dt, 3)
    m, r = (api.MDRField(shape, dt, L, B, enc) for _ in range(2))
    m.refactor(x)
    r.load_metadata(m.metadata())
    for l in range(L + 1):
        r.load_level(l, m.export_level(l))
    out, tol = torch.empty_like(x), 1e-2 * float(x.abs().max())
    torch.cuda.synchronize()
    refused(side, lambda: r.retrieve(tol, out=out, stream=side))
    want = m.retrieve(tol)
    assert torch.equal(r.retrieve(tol, out=out), want)
    with Capture(side) as c:   # everything is unpacked now
        r.retrieve(tol, out=out, stream=side)
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        c.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    c.close()


@pytest.mark.parametrize("enc,dt,B", [("negabinary", torch.float32, 32), ("grouped", torch.float64, 50),
                                      ("perbit", torch.float64, 40)])
def test_lossless_export_refuses_capture(enc, dt, B):
    from prodm_gb300 import api
    shape, L = (17, 20, 33), 2
    side = torch.cuda.Stream()
    m = api.MDRField(shape, dt, L, B, enc)
    m.set_lossless(26)
    m.refactor(noise(shape, dt, 4))
    for l in range(L + 1):
        want = m.export_level(l)
        for out in (torch.zeros(len(want), dtype=torch.uint8, device="cuda"),
                    torch.zeros(len(want), dtype=torch.uint8, pin_memory=True)):
            refused(side, lambda: m.export_level_into(l, out, stream=side))
            m.export_level_into(l, out)
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want)


# 3 nc + 7 words: 256 and 259, 2047 and 2050, 7999 and 8002 (the parameters' limits),
# 64000 and 64003 (copied above)
@pytest.mark.parametrize("n", [165, 167, 1359, 1361, 5327, 5329, 42661, 42663])
def test_tables_of_every_size(n):
    from prodm_gb300 import api
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    ref = O.decompose(x.astype(np.float64), (n,), 1, False)
    d = torch.from_numpy(x.copy()).cuda()
    api.decompose(d, 1, "orthogonal")
    # a value passes through a five-point sum and two contracting recurrences: at
    # most 32 roundings of values of the data's size
    tol = 3 * 32 * (np.finfo(np.float32).eps / 2) * float(np.abs(x).max())
    assert np.max(np.abs(d.cpu().numpy().astype(np.float64) - ref)) <= tol


def test_tables_of_calls_behind_one_another():
    from prodm_gb300 import api
    shapes = [(9, 10, n) for n in range(11, 131, 3)]
    xs = [noise(s, torch.float64, i) for i, s in enumerate(shapes)]
    want = []
    for x in xs:
        y = x.clone()
        api.decompose(y, 1, "orthogonal")
        torch.cuda.synchronize()
        want.append(y)
    got = [x.clone() for x in xs]
    a = torch.randn(4096, 4096, device="cuda")
    for _ in range(20):   # the stream is busy while all calls are queued
        a = a @ a / 64.0
    for y in got:
        api.decompose(y, 1, "orthogonal")
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
