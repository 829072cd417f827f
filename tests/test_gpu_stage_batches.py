"""The lossless stage over all levels at once: level files exported to device
memory at odd offsets (streams whose place is not 4-byte aligned go through
scratch), read by a second handle in pieces that split planes, a handle whose
metadata is loaded twice with larger streams the second time, an all-zero
field (streams of no bytes), scratch trimmed between calls."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [("negabinary", torch.float32, 32), ("grouped", torch.float32, 32), ("grouped", torch.float64, 50),
         ("perbit", torch.float64, 40), ("negabinary", torch.float64, 40)]


@pytest.mark.parametrize("latter", [26, 3])
@pytest.mark.parametrize("enc,dt,B", CASES)
def test_files_in_device_memory_round_trip(enc, dt, B, latter):
    from prodm_gb300 import _lib, api
    shape, L = (37, 30, 41), 3
    gen = torch.Generator(device="cuda").manual_seed(B)
    m, r = (api.MDRField(shape, dt, L, B, enc) for _ in range(2))
    m.set_lossless(latter)
    idx = [min(B, 5 + 6 * l) for l in range(L + 1)]
    fields = [torch.zeros(shape, dtype=dt, device="cuda"),
              torch.cumsum(torch.randn(shape, dtype=dt, device="cuda", generator=gen), -1),
              torch.randn(shape, dtype=dt, device="cuda", generator=gen)]
    for k, x in enumerate(fields):   # stored sizes grow from field to field
        m.refactor(x)
        want = m.retrieve_planes(idx)
        host = [m.export_level(l) for l in range(L + 1)]
        if k:
            r.load_metadata(m.metadata())
        else:
            r = api.MDRField(shape, dt, L, B, enc)
            r.load_metadata(m.metadata())
        for off in (0, 1, 4, 7):
            for l in range(L + 1):
                buf = torch.full((len(host[l]) + 16,), 170, dtype=torch.uint8, device="cuda")
                assert m.export_level_into(l, buf[off:]) == len(host[l])
                assert np.array_equal(buf[off:off + len(host[l])].cpu().numpy(), host[l])
                assert bool((buf[off + len(host[l]):] == 170).all())   # nothing behind the file
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        for l in range(L + 1):   # on another stream: there for the current one
            assert np.array_equal(m.export_level_device(l, stream=side).cpu().numpy(), host[l])
        for l in range(L + 1):
            f = torch.from_numpy(host[l]).cuda()
            cut = len(f) // 3 | 1
            for a, b in ((0, cut), (cut, 2 * cut), (2 * cut, len(f))):
                r.load_level(l, f[a:b], offset=a)
            if l == 1:
                r.retrieve_planes([idx[0], idx[1]] + [0] * (L - 1))   # levels expanded at different times
        assert torch.equal(r.retrieve_planes(idx).view(torch.uint8), want.view(torch.uint8))
        _lib.call("prodm_trim_scratch")


def test_decoder_dropped_with_its_work_in_flight():
    from prodm_gb300 import api
    n, B = 1 << 20, 32
    x = torch.randn(n, device="cuda")
    blob, sizes, _ = api.encode("grouped", x, 4, B)
    want = api.ProgressiveDecoder("grouped", torch.float32).decode(blob, sizes, n, 4, 0, B, 0, B).clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(8):   # each decoder's state goes back to the pool while the other stream works
        d = api.ProgressiveDecoder("grouped", torch.float32)
        with torch.cuda.stream(side):
            a = d.decode(blob, sizes, n, 4, 0, B, 0, B)
        side.synchronize()
        b = d.decode(blob, sizes, n, 4, 0, B, 1, B)
        del d
        outs += [a, b]
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
