"""Level files exported to device memory on one stream are there when the call
returns, for a reader on any other stream."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("latter", [-1, 26])
@pytest.mark.parametrize("enc,dt,B", [("negabinary", torch.float32, 32), ("grouped", torch.float64, 50),
                                      ("perbit", torch.float64, 40)])
def test_export_to_device_memory_returns_with_the_bytes(enc, dt, B, latter):
    from prodm_gb300 import _lib, api
    shape, L = (33, 34, 35), 2
    m = api.MDRField(shape, dt, L, B, enc)
    if latter >= 0:
        m.set_lossless(latter)
    m.refactor(torch.randn(shape, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(B)))
    side = torch.cuda.Stream()
    a = torch.ones(2048, 2048, device="cuda")
    for l in range(L + 1):
        want = torch.from_numpy(m.export_level(l)).cuda()
        for odd in (0, 1):
            buf = torch.zeros(len(want) + odd, dtype=torch.uint8, device="cuda")[odd:]
            torch.cuda.synchronize()
            with torch.cuda.stream(side):   # the export waits behind this
                for _ in range(30):
                    a = a @ a / 2048.0
            n = C.c_uint64()
            _lib.call("prodm_mdr_export_level", m.h, l, C.c_void_p(buf.data_ptr()), len(want), 0, C.byref(n),
                      C.c_void_p(side.cuda_stream))
            assert n.value == len(want) and torch.equal(buf, want)
