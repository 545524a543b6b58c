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


@pytest.mark.parametrize("score", ["sigmoid", "softmax", "softmax_of_chosen"])
@pytest.mark.parametrize("experts,groups,keep", [(64, 1, 1), (40, 1, 1), (64, 8, 4)])
@pytest.mark.parametrize("tokens", [5, 600])
def test_a_token_of_nan_takes_no_more_experts(score, experts, groups, keep, tokens):
    """Rows that are all NaN, or whose scores are NaN for one expert, choose `top` experts like any other; the others choose as
    they do without them."""
    o = ops()
    if groups > 1 and score == "softmax_of_chosen":
        pytest.skip("that score knows no groups")
    top, hidden = 3, 128
    g = torch.Generator(device=DEV).manual_seed(experts)
    h, router = torch.randn(tokens, hidden, generator=g, device=DEV), torch.randn(experts, hidden, generator=g, device=DEV)

    def route(h, router):
        share = torch.full((tokens, experts), 9.0, device=DEV)
        o.moe_route(h, router, experts, top, None, share, score=score, groups=groups, keep=keep)
        return share
    clean = route(h, router)
    assert bool(((clean != 0).sum(1) == top).all())
    bad = h.clone()
    bad[1::3] = float("nan")
    share = route(bad, router)
    assert bool(((share != 0).sum(1) <= top).all())
    healthy = [t for t in range(tokens) if t % 3 != 1]
    assert torch.equal(share[healthy], clean[healthy])
    if score != "softmax_of_chosen":                      # which passes a NaN by
        assert bool(share[1::3].isnan().any(1).all())
        worn = router.clone()
        worn[7, 3] = float("nan")
        share = route(h, worn)
        assert bool(((share != 0).sum(1) <= top).all())


def test_tokens_of_nan_leave_the_others_alone():
    """A request of NaN rows in a routed layer's step: every other row's output is what it is without them, bit for bit."""
    from tokenizer_b200.config import PartSpec
    from tokenizer_b200.parts import Runtime, build_part, part_class
    from tokenizer_b200.weights import WeightStore
    o = ops()
    experts, top, ff, hidden, tokens = 64, 1, 512, 512, 2000
    spec = PartSpec("routed_mlp", dict(experts=experts, top=top, expert_inner=ff, hidden_size=hidden, activation="silu",
                                       score="sigmoid"), "mlp")
    g = torch.Generator(device=DEV).manual_seed(6)
    weights = {t.name: (torch.randn(tuple(t.shape), generator=g, device=DEV) / t.shape[1] ** 0.5).bfloat16()
               for t in part_class("feed_forward", "routed_mlp").tensors(spec)}
    layer = build_part("feed_forward", spec, WeightStore(weights), Runtime(torch.device(DEV), torch.bfloat16))
    assert o.moe_grouped_pays(tokens, experts, top, ff, 0, hidden)
    h = torch.randn(tokens, hidden, generator=g, device=DEV).bfloat16()
    want = layer.forward(h)
    bad = h.clone()
    bad[300:1500] = float("nan")
    got = layer.forward(bad)
    healthy = torch.ones(tokens, dtype=torch.bool, device=DEV)
    healthy[300:1500] = False
    assert torch.equal(got[healthy], want[healthy])
    assert bool(got[~healthy].isnan().all())
