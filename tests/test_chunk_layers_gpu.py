"""The recurrences in chunks of 32 tokens as a layer runs them: against their token-by-token forms, eager and in a captured
step that is replayed with other portions under the same key; steps of many requests and many heads a group; keys that
repeat, where the triangle between a chunk's tokens weighs most."""
import pytest
import torch

from test_delta_chunks_gpu import rule

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")

KINDS = {
    "mamba2": dict(hidden_size=256, heads=64, vdim=64, state=128, groups=2, conv=4, norm_groups=2, eps=1e-6),
    "gated_delta_net": dict(hidden_size=256, heads=8, kv_heads=4, dim=128, vdim=64, conv=4, eps=1e-6),
    "channel_delta_net": dict(hidden_size=256, heads=8, kv_heads=4, dim=128, vdim=64, conv=4, eps=1e-6)}


class Layer:
    """A mixer with its cache, whose steps can be captured: metadata stays at its place, rows in one buffer."""

    def __init__(self, kind):
        from tokenizer_b200.cache.device import DeviceCache
        from tokenizer_b200.config import PartSpec
        from tokenizer_b200.config.spec import LayerCall
        from tokenizer_b200.engine.batch import BatchBuilder
        from tokenizer_b200.parts import Runtime, build_part, part_class
        from tokenizer_b200.weights import WeightStore
        spec, g = PartSpec(kind, KINDS[kind], "mix"), torch.Generator(device=DEV).manual_seed(5)
        tensors = {}
        for t in part_class("mixer", kind).tensors(spec):
            shape = tuple(int(n) for n in t.shape)
            value = torch.randn(shape, generator=g, device=DEV) * (shape[1] ** -0.5 if len(shape) > 1 and t.std == 0.02 else t.std)
            tensors[t.name] = (value + (1.0 if t.init == "one_plus_normal" else -3.5 if t.name.endswith("dt_bias") else 0.0)
                               ).to(torch.bfloat16)
        runtime = Runtime(DEV, torch.bfloat16)
        self.part = build_part("mixer", spec, WeightStore(tensors), runtime)
        self.cache = DeviceCache([self.part.cache_need()], 1, 16, 8, runtime)
        self.binding = self.cache.bindings([LayerCall(0)])[0]
        self.builder = BatchBuilder(self.cache, 2, 1 << 24, DEV, [])
        self.builder.reserve_capacity(1 << 16)
        self.requests = [self.cache.open(i) for i in range(4)]
        self.rows = torch.randn(1024, 256, generator=g, device=DEV).to(torch.bfloat16)

    def context(self, lens):
        from tokenizer_b200.engine.batch import StepEntry
        entries = [StepEntry(r, [0] * n, []) for r, n in zip(self.requests, lens)]
        for r, n in zip(self.requests, lens):
            self.cache.reserve(r, n)
        return self.builder.build(entries, pad_requests=4, pad_tokens=768)[0]

    def forward(self, ctx):
        out = self.part.forward(self.rows[:ctx.n_tokens], ctx, self.binding)
        return out.sum(0) if out.dim() == 3 else out


def alike(got, want, rows):
    """Equal but for the order of 32-bit sums in front of one rounding to bfloat16 and a product: a row may meet a few
    neighbouring bfloat16 values, 2^-9 of those lanes each."""
    diff = (got[:rows].float() - want[:rows].float()).norm() / want[:rows].float().norm()
    assert torch.isfinite(want[:rows].float()).all() and float(diff) < 2.0 ** -9


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_layer_eager_and_replayed(kind):
    layer = Layer(kind)
    portions = [[700], [650, 3]] if kind == "mamba2" else [[300, 260, 1], [256, 40, 300]]
    keys = {layer.part.shape_key(lens) for lens in portions}
    assert len(keys) == 1 and "chunks" in keys.pop()
    state = layer.binding.state
    begin = torch.randn(state.shape, generator=torch.Generator(device=DEV).manual_seed(6), device=DEV) * 0.1

    def step(lens, chunked, run=None):
        ctx = layer.context(lens)
        state.copy_(begin)
        layer.part.chunked = chunked
        out = layer.forward(ctx).clone() if run is None else run()
        return out, state.clone()
    captured = layer.context(portions[0])
    layer.part.chunked = True
    layer.forward(captured)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        place = layer.forward(captured)
    for lens in portions + portions[::-1]:
        want, want_state = step(lens, False)
        got, got_state = step(lens, True)
        alike(got, want, sum(lens))
        # chains of up to 700 tokens, a rounding of the largest value each
        bound = max(lens) * 2.0 ** -24 * float(want_state.abs().max())
        assert float((got_state - want_state).abs().max()) <= bound
        again, again_state = step(lens, True, lambda: (graph.replay(), place.clone())[1])
        assert torch.equal(again[:sum(lens)], got[:sum(lens)]) and torch.equal(again_state, got_state)


@pytest.mark.parametrize("by_channel", [False, True])
def test_delta_rule_of_many_requests(by_channel):
    """40 requests, some of them empty: the search for a block's request takes two turns of 32."""
    from tokenizer_b200.kernels import ops
    groups, heads, dim, vdim, taps = 1, 2, 128, 32, 2
    lengths = [(7 * i * i + 3 * i) % 71 for i in range(40)]
    lengths[3] = lengths[33] = 0
    starts = [0]
    for n in lengths:
        starts.append(starts[-1] + n)
    channels, g = 2 * groups * dim + heads * vdim, torch.Generator().manual_seed(8)
    rnd = lambda *s: torch.randn(*s, generator=g)
    proj, width = rnd(starts[-1], channels + 2 * heads), heads * (dim if by_channel else 1)
    decay = rnd(starts[-1], width) if by_channel else proj[:, channels + heads:]
    conv_w, a_log, dt_bias = rnd(channels, taps) * 0.5, rnd(heads) * 0.5, rnd(width) - 2.0
    off = heads * vdim * 128
    state = torch.zeros(len(lengths), off + (taps - 1) * channels, device=DEV)
    out = torch.empty(starts[-1], heads * vdim, device=DEV)
    d_proj = proj.to(DEV)
    ops.delta_chunks(d_proj, 0, channels, decay.to(DEV) if by_channel else d_proj, 0 if by_channel else channels + heads,
                     by_channel, groups, heads, dim, vdim, taps, conv_w.to(DEV), a_log.to(DEV), dt_bias.to(DEV), state, off,
                     torch.tensor(starts, dtype=torch.int32, device=DEV),
                     torch.arange(len(lengths), dtype=torch.int32, device=DEV), out)
    got, got_state = out.cpu().double(), state[:, :off].cpu().double()
    for r, n in enumerate(lengths):
        span, S = slice(starts[r], starts[r + 1]), torch.zeros(heads, dim, vdim, dtype=torch.float64)
        if n:
            want, _ = rule(proj[span].double(), decay[span].double(), (groups, heads, dim, vdim, taps), by_channel,
                           conv_w.double(), a_log.double(), dt_bias.double(),
                           torch.zeros(taps - 1, channels, dtype=torch.float64), S, dim ** -0.5)
            # 32-bit sums of 128 products, a chain of three chunks at most: some tens of 2^-24 of the largest value
            assert float((got[span] - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))
        assert float((got_state[r].view(heads, vdim, 128).transpose(1, 2) - S).abs().max()) < 1e-5 * max(1.0, float(S.abs().max()))


@pytest.mark.parametrize("by_channel", [False, True])
@pytest.mark.parametrize("spread", [0.0, 1e-3, 0.3])
def test_keys_that_repeat(by_channel, spread):
    """700 tokens whose keys are one vector, nearly one or close to one another, beta and decays next to one: every token
    takes out what the one before it put in."""
    from tokenizer_b200.kernels import ops
    groups, heads, dim, vdim, n = 1, 2, 128, 32, 700
    channels, g = 2 * groups * dim + heads * vdim, torch.Generator().manual_seed(9)
    rnd = lambda *s: torch.randn(*s, generator=g)
    proj, width = rnd(n, channels + 2 * heads), heads * (dim if by_channel else 1)
    proj[:, dim:2 * dim] = rnd(1, dim) + spread * rnd(n, dim)
    proj[:, channels:channels + heads] = 9.0                               # beta: 0.9999
    decay = rnd(n, width) if by_channel else proj[:, channels + heads:]
    conv_w, a_log, dt_bias = torch.ones(channels, 1), torch.zeros(heads), torch.full((width,), -9.0)      # decays: about 0.9999
    off = heads * vdim * 128
    state, out, d_proj = torch.zeros(1, off, device=DEV), torch.empty(n, heads * vdim, device=DEV), proj.to(DEV)
    ops.delta_chunks(d_proj, 0, channels, decay.to(DEV) if by_channel else d_proj, 0 if by_channel else channels + heads,
                     by_channel, groups, heads, dim, vdim, 1, conv_w.to(DEV), a_log.to(DEV), dt_bias.to(DEV), state, off,
                     torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV), out)
    S = torch.zeros(heads, dim, vdim, dtype=torch.float64)
    want, _ = rule(proj.double(), decay.double(), (groups, heads, dim, vdim, 1), by_channel, conv_w.double(), a_log.double(),
                   dt_bias.double(), torch.zeros(0, channels, dtype=torch.float64), S, dim ** -0.5)
    # a token's sums of 128 products round by at most 128 * 2^-24 of their largest terms, in practice by the root of that; the
    # rule itself makes no error grow (I - beta k k^T shortens every vector), so errors add up like the root of the tokens
    bound = 2.0 ** -24 * (128 * n) ** 0.5
    assert float((out.cpu().double() - want).abs().max()) < bound * max(1.0, float(want.abs().max()))
    got = state.cpu().double().view(heads, vdim, 128).transpose(1, 2)
    assert float((got - S).abs().max()) < bound * max(1.0, float(S.abs().max()))


def test_state_space_of_many_requests_and_heads():
    """40 requests, some of them empty, and 16 heads that share a group's B and C: two turns of the search for a block's
    request and of the warps over a group's heads."""
    from tokenizer_b200.kernels import ops
    heads, groups, vdim, n_state = 32, 2, 32, 128
    lengths = [(5 * i * i + 11 * i) % 67 for i in range(40)]
    lengths[2] = lengths[35] = 0
    starts = [0]
    for n in lengths:
        starts.append(starts[-1] + n)
    inner, rows, g = heads * vdim, starts[-1], torch.Generator(device=DEV).manual_seed(13)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    xbc, proj = rnd(rows, inner + 2 * groups * n_state), rnd(rows, heads)
    dt_bias, a_log, skip = rnd(heads) - 2.0, rnd(heads) * 0.5, rnd(heads)
    state, y = torch.zeros(40, inner * n_state, device=DEV), torch.empty(rows, inner, device=DEV)
    ops.ssd_chunks(xbc, proj, 0, dt_bias, a_log, skip, heads, groups, vdim, n_state, state,
                   torch.tensor(starts, dtype=torch.int32, device=DEV), torch.arange(40, dtype=torch.int32, device=DEV), y)
    dt = torch.nn.functional.softplus(proj.double() + dt_bias.double())
    keep = torch.exp(-torch.exp(a_log.double()) * dt)
    x = xbc[:, :inner].double().view(rows, heads, vdim)
    b, c = (t.reshape(rows, groups, n_state).double().repeat_interleave(heads // groups, 1)
            for t in torch.split(xbc[:, inner:], groups * n_state, dim=1))
    for r, n in enumerate(lengths):
        S, want = torch.zeros(heads, n_state, vdim, dtype=torch.float64, device=DEV), []
        for t in range(starts[r], starts[r + 1]):
            S = keep[t][:, None, None] * S + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            want.append(torch.einsum("hnv,hn->hv", S, c[t]) + skip.double()[:, None] * x[t])
        # 32-bit sums of 128 products, a chain of three chunks at most: some tens of 2^-24 of the largest value
        if n:
            want = torch.stack(want).reshape(n, -1)
            assert float((y[starts[r]:starts[r + 1]].double() - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))
        m = state[r].double().view(heads, vdim, n_state).transpose(1, 2)
        assert float((m - S).abs().max()) < 1e-5 * max(1.0, float(S.abs().max()))
