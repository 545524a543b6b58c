"""The short convolution on both sides of the line between one and eight rows a thread, weights on and off 16 bytes, against
64 bits: portions that begin inside a run of eight, kept inputs in front of them, idle rows behind the last."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n,channels", [(1465, 1024), (1464, 1024), (20, 132), (366, 4100), (365, 4100)])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("off_by", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rows_and_weights(n, channels, taps, off_by, dtype):
    from tokenizer_b200.kernels import ops as o
    g = torch.Generator().manual_seed(n + taps)
    live = n - 3
    cuts = [0, min(2, live), live // 3, live // 2 + 1, live]
    x = torch.randn(n, channels + 8, generator=g).to(dtype)
    w, bias = torch.randn(channels, taps, generator=g), torch.randn(channels, generator=g)
    kept = torch.randn(4, taps - 1, channels, generator=g)
    room = torch.empty(channels * taps + 4, device=DEV)
    weight = room[off_by:off_by + channels * taps].view(channels, taps).copy_(w)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    req = [r for r in range(4) for _ in range(cuts[r + 1] - cuts[r])] + [-1] * (n - live)
    out = torch.full((n, channels), 9.0, device=DEV, dtype=dtype)
    o.short_conv(x.to(DEV), 4, channels, weight, bias.to(DEV), kept.reshape(4, -1).to(DEV), 0, ints(req), ints(cuts),
                 ints(range(4)), out, "silu")
    got = out.cpu().double()
    assert bool((got[live:] == 9.0).all())
    for r in range(4):
        rows = torch.cat([kept[r].double(), x[cuts[r]:cuts[r + 1], 4:4 + channels].double()])
        m = cuts[r + 1] - cuts[r]
        terms = [rows[j:j + m] * w[:, j].double() for j in range(taps)]
        want = torch.nn.functional.silu(sum(terms) + bias.double())
        # taps + 1 sums in 32 bits through silu, whose slope stays below 1.1, and its own few roundings; one to 16 bits
        slack = (sum(t.abs() for t in terms) + bias.double().abs()) * 1.1 * (taps + 1) * 2.0 ** -24 + want.abs() * 2.0 ** -20
        if dtype == torch.bfloat16:
            slack = slack + want.abs() * 2.0 ** -8
        assert bool(((got[cuts[r]:cuts[r + 1]] - want).abs() <= slack + 1e-9).all())
