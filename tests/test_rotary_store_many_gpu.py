"""Rotation and cache write of many tokens (several a block) against the same tokens in portions that take a block each:
both pairings, leading lanes alone rotated, temperatures, idle rows, rows without a slot, values that are keys, odd counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [1184, 1187, 2501])
@pytest.mark.parametrize("heads,kv,dim,rot,layout", [(3, 1, 128, 128, "half"), (2, 2, 64, 64, "interleaved"),
                                                     (5, 1, 40, 16, "interleaved"), (1, 1, 8, 8, "half"), (2, 1, 72, 0, "half"), (3, 1, 128, 64, "half"), (2, 1, 40, 8, "half")])
@pytest.mark.parametrize("out", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("keys_too", [False, True])
def test_many_tokens_as_few(n, heads, kv, dim, rot, layout, out, keys_too):
    from tokenizer_b200.kernels import ops as o
    g = torch.Generator(device=DEV).manual_seed(n + dim)
    width = (heads + (1 if keys_too else 2) * kv) * dim
    proj = torch.randn(n, width + 8, device=DEV, generator=g)
    bias = torch.randn(width, device=DEV, generator=g) if heads != 5 else None
    temp = torch.rand(heads, device=DEV, generator=g) + 0.5 if heads != 1 else None
    freq = torch.rand(rot // 2, device=DEV, generator=g, dtype=torch.float64) if rot else None
    pos = torch.randint(0, 100000, (n,), device=DEV, generator=g, dtype=torch.int32)
    slot = torch.randperm(n, device=DEV, generator=g).int()
    slot[::7] = -1
    req = torch.zeros(n, device=DEV, dtype=torch.int32)
    req[5::11] = -1
    results = []
    for step in (n, 400):
        q = torch.full((n, heads * dim), 9.0, device=DEV, dtype=out)
        k, v = (torch.full((n, kv, dim), 9.0, device=DEV, dtype=out) for _ in range(2))
        for i in range(0, n, step):
            part = slice(i, min(n, i + step))
            o.qkv_rotate_store(proj[part], 4, bias, freq, rot, pos[part], slot[part], req[part], q[part], k, v, heads, kv, dim,
                               dim, dim, temp=temp, layout=layout, values_are_keys=keys_too)
        results.append((q.float(), k.float(), v.float()))
    # the two products of a rotated lane may be fused either way round: 2^-23 of their sizes, and a rounding to 16 bits
    top = float(proj.abs().max() + (bias.abs().max() if bias is not None else 0)) * 3
    for got, want in zip(*results):
        assert bool(((got - want).abs() <= top * 2.0 ** -23 + (want.abs() * 2.0 ** -7 if out == torch.bfloat16 else 0)).all())
        assert torch.equal(got == 9.0, want == 9.0)


def test_queries_alone():
    from tokenizer_b200.kernels import ops as o
    n, heads, dim = 1300, 3, 64
    g = torch.Generator(device=DEV).manual_seed(1)
    proj = torch.randn(n, heads * dim, device=DEV, generator=g)
    freq = torch.rand(dim // 2, device=DEV, generator=g, dtype=torch.float64)
    pos, req = torch.arange(n, device=DEV, dtype=torch.int32), torch.zeros(n, device=DEV, dtype=torch.int32)
    got, want = (torch.full((n, heads * dim), 9.0, device=DEV) for _ in range(2))
    o.qkv_rotate_store(proj, 0, None, freq, dim, pos, None, req, got, None, None, heads, 0, dim, dim, dim, layout="half")
    for i in range(0, n, 650):
        s = slice(i, i + 650)
        o.qkv_rotate_store(proj[s], 0, None, freq, dim, pos[s], None, req[s], want[s], None, None, heads, 0, dim, dim, dim,
                           layout="half")
    assert float((got - want).abs().max()) <= float(proj.abs().max()) * 2.0 ** -22
