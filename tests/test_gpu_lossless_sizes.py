"""Level files and metadata of a handle whose lossless stage is on and has no
stored sizes: before the first refactor, and after a refactor that failed in
the stage (its wait is refused while the stream is captured)."""
import numpy as np
import pytest
import torch

from stream_capture import Capture, clear_error

pytestmark = pytest.mark.gpu

EINVAL = 1
SHAPE, L = (17, 20, 33), 2


def refused(m):
    from prodm_gb300 import _lib
    dev = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    for l in range(L + 1):
        for f in (lambda: m.export_level(l), lambda: m.export_level_device(l), lambda: m.export_level_into(l, dev),
                  lambda: m.export_level_range_into(l, 0, dev[:8]), lambda: m.metadata()):
            with pytest.raises(_lib.ProdmError) as e:
                f()
            assert e.value.status == EINVAL and "refactor first" in str(e.value)


@pytest.mark.parametrize("enc,dt,B", [("negabinary", torch.float32, 32), ("grouped", torch.float64, 50),
                                      ("perbit", torch.float64, 40)])
def test_stage_without_sizes(enc, dt, B):
    from prodm_gb300 import _lib, api
    m = api.MDRField(SHAPE, dt, L, B, enc)
    m.set_lossless(26)
    refused(m)
    x = torch.randn(SHAPE, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(B))
    m.refactor(x)
    files, meta = [m.export_level(l) for l in range(L + 1)], m.metadata()
    side = torch.cuda.Stream()
    with Capture(side) as c:
        with pytest.raises(_lib.ProdmError):
            m.refactor(x, stream=side)
    assert c.status != 0
    clear_error()
    refused(m)
    m.refactor(x)
    assert m.metadata() == meta
    for l in range(L + 1):
        assert np.array_equal(m.export_level(l), files[l])
