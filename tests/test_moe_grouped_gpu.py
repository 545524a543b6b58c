"""Routed experts over sorted rows against the same experts in 64 bits: ragged groups, groups without a row, all tokens in one
group, edges of a tile of 256 rows, inner sizes that are no whole 128s, with and without a shared expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from tokenizer_b200.kernels import ops as o
    return o


@pytest.mark.parametrize("activation", ["silu", "relu_squared"])
@pytest.mark.parametrize("tokens,hidden,experts,top,ff,shared,skew", [
    (1, 64, 1, 1, 64, 0, 0.0), (255, 136, 4, 2, 64, 192, 0.0), (256, 256, 8, 2, 192, 64, 3.0), (257, 512, 3, 3, 128, 0, 0.0),
    (700, 264, 40, 4, 64, 128, 1.0), (1030, 1024, 8, 2, 704, 1408, 8.0)])
def test_against_64_bits(activation, tokens, hidden, experts, top, ff, shared, skew):
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    inner = experts * ff + shared
    h, gate_up = rnd(tokens, hidden).bfloat16(), (rnd(2 * inner, hidden) / hidden ** 0.5).bfloat16()
    down = (rnd(hidden, inner) / ff ** 0.5).bfloat16()
    # skewed: most tokens choose the first experts, the last ones may get none
    scores = rnd(tokens, experts) - skew * torch.arange(experts, device=DEV)
    best, chosen = torch.topk(scores, top, dim=1)
    share = torch.zeros(tokens, experts + int(shared > 0), device=DEV)
    share.scatter_(1, chosen, torch.softmax(best, dim=1))
    if shared:
        share[:, experts] = torch.sigmoid(rnd(tokens))
    assert o.moe_grouped_supported(tokens, experts, top, ff, shared, hidden, activation)
    got = o.moe_grouped(h, share, gate_up, down, experts, top, ff, shared, activation)
    again = o.moe_grouped(h, share, gate_up, down, experts, top, ff, shared, activation)
    assert torch.equal(got, again)
    both = h.double() @ gate_up.double().t()
    gate, up = both[:, :inner], both[:, inner:]
    act = gate * torch.sigmoid(gate) if activation == "silu" else torch.relu(gate) ** 2
    lanes = torch.cat([share[:, :experts].repeat_interleave(ff, 1), share[:, experts:].expand(-1, shared)], dim=1).double()
    act = act * up * lanes
    want = act @ down.double().t()
    # an inner lane and the result are rounded to bfloat16 once (2^-9 each), sums of k products in 32-bit
    bound = 2.0 ** -8 * (act.abs() @ down.double().abs().t()) + 2.0 ** -8 * want.abs() + 1e-4
    assert bool(((got.double() - want).abs() <= bound).all())
    assert float((got.double() - want).norm() / want.norm()) < 4e-3


def test_what_is_refused():
    o = ops()
    assert not o.moe_grouped_supported(300, 129, 2, 64, 0, 64, "silu")
    assert not o.moe_grouped_supported(300, 8, 2, 96, 0, 64, "silu")
    assert not o.moe_grouped_supported(300, 8, 2, 64, 32, 64, "silu")
    assert not o.moe_grouped_supported(300, 8, 2, 64, 0, 64, "clamped_swish")


def test_a_layer_gives_the_same_either_way():
    """A prompt's rows sorted by expert, and the same rows a few at a time, every expert's lanes for every token."""
    from tokenizer_b200.config import PartSpec
    from tokenizer_b200.parts import Runtime, build_part, part_class
    from tokenizer_b200.weights import WeightStore
    o = ops()
    sizes = dict(experts=16, top=2, expert_inner=512, shared_inner=64, hidden_size=512)
    spec = PartSpec("routed_mlp", dict(sizes, activation="silu"), "mlp")
    g = torch.Generator(device=DEV).manual_seed(5)
    weights = {t.name: (torch.randn(tuple(t.shape), generator=g, device=DEV) / t.shape[1] ** 0.5).bfloat16()
               for t in part_class("feed_forward", "routed_mlp").tensors(spec)}
    layer = build_part("feed_forward", spec, WeightStore(weights), Runtime(torch.device(DEV), torch.bfloat16))
    tokens = 6000
    assert o.moe_grouped_pays(tokens, 16, 2, 512, 64, 512) and not o.moe_grouped_pays(500, 16, 2, 512, 64, 512)
    h = torch.randn(tokens, 512, generator=g, device=DEV).bfloat16()
    whole = layer.forward(h).float()
    parts = [layer.forward(h[i:i + 500].contiguous()) for i in range(0, tokens, 500)]
    parts = torch.cat([p.float() if p.dim() == 2 else p.sum(0) for p in parts])
    # three roundings to bfloat16 on one way, two on the other
    assert float((whole - parts).norm() / parts.norm()) < 6e-3
