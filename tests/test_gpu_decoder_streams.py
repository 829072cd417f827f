"""Progressive decoding of one level in parts on several streams, with no wait of
the host between them: the level's state is handed on in the order of the calls."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("enc,dt,B", [("grouped", torch.float32, 32), ("grouped", torch.float64, 50),
                                      ("perbit", torch.float32, 32), ("perbit", torch.float64, 40)])
@pytest.mark.parametrize("n", [100, 70001])
def test_parts_of_a_level_on_several_streams(enc, dt, B, n):
    from prodm_gb300 import api
    x = torch.randn(n, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    blob, sizes, _ = api.encode(enc, (x * torch.exp(3 * x)).clamp(-255, 255), 8, B)   # below 2^8
    cuts = [0, 3, 11, 12, B]
    at = np.concatenate([[0], np.cumsum(np.asarray(sizes, np.int64))])
    parts = [blob[int(at[a]):int(at[b])].clone() for a, b in zip(cuts, cuts[1:])]

    def decode(d, i):
        return d.decode(parts[i], sizes[cuts[i]:cuts[i + 1]], n, 8, cuts[i], cuts[i + 1] - cuts[i], 0, B)

    one = api.ProgressiveDecoder(enc, dt)
    want = [decode(one, i) for i in range(len(parts))]
    streams = [torch.cuda.Stream() for _ in range(3)]
    a = torch.ones(2048, 2048, device="cuda")
    torch.cuda.synchronize()
    for turn in range(3):
        d, got = api.ProgressiveDecoder(enc, dt), []
        for i in range(len(parts)):
            with torch.cuda.stream(streams[(turn + i) % 3]):
                if i % 2 == 0:   # the next part's stream is free while this one's works
                    for _ in range(20):
                        a = a @ a / 2048.0
                got.append(decode(d, i))
        del d   # with the last part's work in flight
        torch.cuda.synchronize()
        assert all(torch.equal(g, w) for g, w in zip(got, want))
