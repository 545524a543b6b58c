"""The residual add on both sides of where it takes eight elements a thread, its last partial block, and element counts that
are no whole eights, in both types and over several planes: the same bits as additions in index order."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,planes", [(torch.float32, 1), (torch.float32, 3), (torch.bfloat16, 1)])
@pytest.mark.parametrize("rows,width", [(37887, 8), (37888, 8), (37889, 8), (303104 // 64 + 5, 64), (43301, 7), (2048, 896)])
def test_same_bits_as_additions_in_order(rows, width, dtype, planes):
    from tokenizer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randn(rows, width, generator=g, device=DEV)
    delta = torch.randn((planes, rows, width) if planes > 1 else (rows, width), generator=g, device=DEV).to(dtype)
    want = x.clone()
    for plane in (delta if planes > 1 else delta[None]):
        want += plane.float()
    ops.residual_add(x, delta)
    assert torch.equal(x, want)
