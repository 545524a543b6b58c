"""The delta rules in chunks against the same rule token by token in 64 bits: portions of one token to several chunks and
their remainders, continued portions (a matrix and kept inputs that are not zero), idle rows, decays next to one, next to
zero and mixed by channel, heads of fewer than 128 lanes, values of 16 to 128, taps other than four, both widths of a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from tokenizer_b200.kernels import ops as o
    return o


def rule(proj, decay_in, p, by_channel, conv_w, a_log, dt_bias, kept, S, scale):
    """One request in float64: `proj` [n, channels + heads], `decay_in` [n, heads (* dim)]; returns o and moves S."""
    groups, heads, dim, vdim, taps = p
    n, channels = proj.shape[0], 2 * groups * dim + heads * vdim
    x = torch.cat([kept, proj[:, :channels]])
    y = sum(x[j:j + n] * conv_w[:, j] for j in range(taps))
    y = y * torch.sigmoid(y)
    q, k, v = torch.split(y, [groups * dim, groups * dim, heads * vdim], dim=1)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    q = unit(q.reshape(n, groups, dim)).repeat_interleave(heads // groups, 1) * scale
    k = unit(k.reshape(n, groups, dim)).repeat_interleave(heads // groups, 1)
    v, beta = v.reshape(n, heads, vdim), torch.sigmoid(proj[:, channels:channels + heads])
    rate, soft = torch.exp(a_log), torch.nn.functional.softplus(decay_in + dt_bias)
    g = torch.exp(-rate[:, None] * soft.view(n, heads, dim)) if by_channel else \
        torch.exp(-rate * soft)[..., None].expand(n, heads, dim)
    o = torch.empty(n, heads, vdim, dtype=torch.float64)
    for t in range(n):
        S.mul_(g[t][:, :, None])
        u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S.add_(k[t][:, :, None] * u[:, None, :])
        o[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return o.reshape(n, -1), x[x.shape[0] - (taps - 1):]


@pytest.mark.parametrize("by_channel,columns", [(False, 0), (True, 16), (False, 32), (True, 32)])
@pytest.mark.parametrize("groups,heads,dim,vdim,taps,shift", [
    (1, 2, 128, 128, 4, -3.0), (2, 2, 128, 64, 4, 3.0), (1, 3, 72, 48, 2, 0.0), (2, 4, 100, 16, 1, -6.0)])
def test_against_the_rule(by_channel, columns, groups, heads, dim, vdim, taps, shift):
    o = ops()
    assert o.delta_chunks_supported(dim, vdim)
    lengths = [[1, 33, 0, 64, 95, 32], [31, 2, 40, 1, 0, 70]]          # two portions a request, some of them empty
    n_req, channels = len(lengths[0]), 2 * groups * dim + heads * vdim
    g = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g)
    conv_w, a_log = rnd(channels, taps) * 0.5, rnd(heads) * 0.5
    dt_bias = rnd(heads * (dim if by_channel else 1)) * 2.0 + shift       # decays spread around the shift's
    off = heads * vdim * 128
    size = -(-(off + (taps - 1) * channels) // 4) * 4
    state = torch.zeros(n_req, size)
    matrices = rnd(n_req, heads, dim, vdim) * 0.3
    state[:, :off] = torch.nn.functional.pad(matrices.transpose(2, 3), (0, 128 - dim)).reshape(n_req, -1)
    kept = [rnd(taps - 1, channels) for _ in range(n_req)]
    for r in range(n_req):
        state[r, off:off + (taps - 1) * channels] = kept[r].reshape(-1)
    S, kept = [m.double() for m in matrices], [k.double() for k in kept]
    slots = torch.randperm(n_req, generator=g)
    dev = torch.empty(n_req, size, device=DEV)
    dev[slots.to(DEV)] = state.to(DEV)
    for portion in lengths:
        starts = [0]
        for n in portion:
            starts.append(starts[-1] + n)
        rows = starts[-1] + 5                                             # idle rows behind the last request
        proj = rnd(rows, channels + heads + 8 + heads)
        width = heads * (dim if by_channel else 1)
        decay = rnd(rows, width + 4) if by_channel else proj
        at = 0 if by_channel else channels + heads + 8
        out = torch.full((rows, heads * vdim), 9.0, device=DEV)
        d_proj = proj.to(DEV)
        o.delta_chunks(d_proj, 0, channels, decay.to(DEV) if by_channel else d_proj, at, by_channel, groups, heads, dim, vdim,
                       taps, conv_w.to(DEV), a_log.to(DEV), dt_bias.to(DEV), dev, off,
                       torch.tensor(starts, dtype=torch.int32, device=DEV), slots.int().to(DEV), out,
                       columns=columns)
        got, got_state = out.cpu().double(), dev[slots.to(DEV)].cpu().double()
        assert bool((got[starts[-1]:] == 9.0).all())
        for r, n in enumerate(portion):
            span = slice(starts[r], starts[r + 1])
            if n:
                want, kept[r] = rule(proj[span].double(), decay[span, at:at + width].double(), (groups, heads, dim, vdim, taps),
                                     by_channel, conv_w.double(), a_log.double(), dt_bias.double(), kept[r], S[r], dim ** -0.5)
                # 32-bit sums of 128 products, a chain of three chunks at most: some tens of 2^-24 of the largest value
                assert float((got[span] - want).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))
            m = got_state[r, :off].view(heads, vdim, 128)
            assert bool((m[..., dim:] == 0).all())
            assert float((m[..., :dim].transpose(1, 2) - S[r]).abs().max()) < 1e-5 * max(1.0, float(S[r].abs().max()))
            if taps > 1:
                assert torch.equal(got_state[r, off:off + (taps - 1) * channels], kept[r].reshape(-1))


@pytest.mark.parametrize("by_channel,columns", [(False, 16), (False, 32), (True, 16), (True, 32)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [1, 17, 30, 45])
def test_a_token_changes_nothing_before_it(by_channel, columns, value, at):
    """An infinity or NaN in a token's values or key leaves the rows in front of it in the same chunk as they are, bit for bit."""
    o = ops()
    groups, heads, dim, vdim, n = 1, 2, 128, 32, 50
    channels = 2 * dim + heads * vdim
    g = torch.Generator().manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    conv_w, a_log, dt_bias = rnd(channels, 1), rnd(heads), rnd(heads * (dim if by_channel else 1))      # one tap: a token's own
    proj = rnd(n, channels + 2 * heads)
    decay = rnd(n, heads * dim) if by_channel else proj
    first = rnd(1, heads * vdim * 128)
    q_start = torch.tensor([0, n], dtype=torch.int32, device=DEV)

    def run(proj):
        out, state = torch.empty(n, heads * vdim, device=DEV), first.clone()
        o.delta_chunks(proj, 0, channels, decay if by_channel else proj, 0 if by_channel else channels + heads, by_channel,
                       groups, heads, dim, vdim, 1, conv_w, a_log, dt_bias, state, heads * vdim * 128, q_start,
                       torch.zeros(1, dtype=torch.int32, device=DEV), out, columns=columns)
        return out
    want = run(proj)
    assert torch.isfinite(want).all()
    for column in (2 * dim + 3, dim + 5):                     # a value of the first head, a lane of the key
        bad = proj.clone()
        bad[at, column] = value
        got = run(bad)
        assert torch.equal(got[:at], want[:at])
        assert not torch.isfinite(got[at:]).all()
        if column >= 2 * dim:                                 # a value's column meets no other
            others = [c for c in range(heads * vdim) if c != column - 2 * dim]
            assert torch.equal(got[:, others], want[:, others])


@pytest.mark.parametrize("by_channel", [False, True])
@pytest.mark.parametrize("taps", [4, 2])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_inputs_off_16_bytes(by_channel, taps, shift):
    """Copies of four channels or of one bring the same inputs: the same bits wherever the rows begin."""
    o = ops()
    groups, heads, dim, vdim, n = 1, 2, 72, 32, 75
    channels = 2 * dim + heads * vdim
    g = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    conv_w, a_log, dt_bias = rnd(channels, taps), rnd(heads), rnd(heads * (dim if by_channel else 1))
    proj, rates = rnd(n, channels + 2 * heads), rnd(n, heads * dim)
    first = rnd(1, heads * vdim * 128 + (taps - 1) * channels)
    first[:, :heads * vdim * 128].view(-1, 128)[:, dim:] = 0
    q_start = torch.tensor([0, n], dtype=torch.int32, device=DEV)

    def moved(t, by):                                  # the same rows, `by` floats behind an aligned place
        room = torch.empty(t.numel() + 4, device=DEV)
        room[by:by + t.numel()] = t.reshape(-1)
        return room[by:by + t.numel()].view(t.shape)

    def run(by_proj, by_rates):
        p, d = moved(proj, by_proj), moved(rates, by_rates)
        out, state = torch.empty(n, heads * vdim, device=DEV), first.clone()
        o.delta_chunks(p, 0, channels, d if by_channel else p, 0 if by_channel else channels + heads, by_channel, groups,
                       heads, dim, vdim, taps, conv_w, a_log, dt_bias, state, heads * vdim * 128, q_start,
                       torch.zeros(1, dtype=torch.int32, device=DEV), out)
        return out, state
    want = run(0, 0)
    for moves in ((shift, 0), (0, shift), (shift, shift)):
        for got, ref in zip(run(*moves), want):
            assert torch.equal(got, ref)


def in_chunks(q, k, v, beta, g, S):
    """One head by the chunks' own sums in 64 bits (q scaled): S [dim, vdim] moves on; the rows' outputs."""
    out, n = torch.empty(q.shape[0], v.shape[1], dtype=torch.float64), q.shape[0]
    for t0 in range(0, n, 32):
        m = min(32, n - t0)
        qc, kc, vc, bc, gc = (x[t0:t0 + m] for x in (q, k, v, beta, g))
        G = torch.cumprod(gc, 0)
        between = torch.zeros(m, m, q.shape[1], dtype=torch.float64)
        for s in range(m):
            between[s, s] = 1.0
            for t in range(s + 1, m):
                between[t, s] = between[t - 1, s] * gc[t]
        A = bc[:, None] * torch.einsum("tc,sc,tsc->ts", kc, kc, between).tril(-1)
        M = torch.einsum("tc,sc,tsc->ts", qc, kc, between)
        solve = lambda r: torch.linalg.solve_triangular(A + torch.eye(m, dtype=torch.float64), r, upper=False, unitriangular=True)
        W, U0 = solve(bc[:, None] * G * kc), solve(bc[:, None] * vc)
        U = U0 - W @ S
        for t in range(m):
            out[t0 + t] = (G[t] * qc[t]) @ S + sum(M[t, s] * U[s] for s in range(t + 1))
        S = G[-1][:, None] * S + sum((between[m - 1, s] * kc[s])[:, None] * U[s][None, :] for s in range(m))
    return out, S


@pytest.mark.parametrize("by_channel,columns", [(False, 16), (False, 32), (True, 16), (True, 32)])
@pytest.mark.parametrize("where", ["matrix", "large matrix", "values", "large values"])
@pytest.mark.parametrize("n", [20, 70])
def test_numbers_without_pieces(by_channel, columns, where, n):
    """Infinities, and numbers that round to one in 16 bits, in the matrix or in the values: outputs and matrix hold numbers,
    infinities (with their signs) and NaN where the same sums in 64 bits do, and other columns what they hold without them."""
    o = ops()
    groups, heads, dim, vdim, inf = 1, 2, 128, 32, float("inf")
    channels, off = 2 * dim + heads * vdim, heads * vdim * 128
    gen = torch.Generator().manual_seed(19)
    rnd = lambda *s: torch.randn(*s, generator=gen)
    conv_w, a_log = torch.ones(channels, 1), rnd(heads) * 0.3
    dt_bias = rnd(heads * (dim if by_channel else 1)) - 3.0
    proj = rnd(n, channels + 2 * heads)
    decay = rnd(n, heads * dim) if by_channel else proj
    S = rnd(heads, dim, vdim)
    bad_S, bad_proj, touched = S.clone(), proj.clone(), [5, vdim + 30]       # columns of the two heads side by side
    if where == "matrix":
        bad_S[0, 3, 5], bad_S[1, 127, 30] = inf, -inf
    elif where == "large matrix":
        bad_S[0, 3, 5], bad_S[1, 127, 30] = 3.4e38, -3.395e38
    else:                                         # silu keeps a large number and an infinity above zero
        bad_proj[11, 2 * dim + 5] = bad_proj[17, 2 * dim + vdim + 30] = inf if where == "values" else 3.4e38

    def run(S, proj):
        state, out = S.transpose(1, 2).reshape(1, -1).to(DEV), torch.empty(n, heads * vdim, device=DEV)
        p = proj.to(DEV)
        o.delta_chunks(p, 0, channels, decay.to(DEV) if by_channel else p, 0 if by_channel else channels + heads, by_channel,
                       groups, heads, dim, vdim, 1, conv_w.to(DEV), a_log.to(DEV), dt_bias.to(DEV), state, off,
                       torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV), out,
                       columns=columns)
        return out.cpu(), state.cpu().view(heads, vdim, 128).transpose(1, 2)
    clean, clean_S = run(S, proj)
    got, got_S = run(bad_S, bad_proj)
    others = [c for c in range(heads * vdim) if c not in touched]
    assert torch.equal(got[:, others], clean[:, others])
    flat, flat_clean = (x.permute(1, 0, 2).reshape(dim, -1) for x in (got_S, clean_S))
    assert torch.equal(flat[:, others], flat_clean[:, others])
    x = bad_proj[:, :channels].double()
    y = torch.where(x.isinf(), x, x * torch.sigmoid(x))
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(proj[:, channels:channels + heads].double())
    width = heads * (dim if by_channel else 1)
    at = 0 if by_channel else channels + heads
    soft = torch.nn.functional.softplus(decay[:, at:at + width].double() + dt_bias.double())
    rate = torch.exp(a_log.double())
    for h, column in ((0, 5), (1, 30)):
        g = torch.exp(-rate[h] * (soft[:, h * dim:(h + 1) * dim] if by_channel else soft[:, h:h + 1].expand(n, dim)))
        want, want_S = in_chunks(unit(y[:, :dim]) * dim ** -0.5, unit(y[:, dim:2 * dim]),
                                 y[:, 2 * dim + h * vdim:2 * dim + (h + 1) * vdim], beta[:, h], g, bad_S[h].double())
        for mine, ref in ((got[:, h * vdim + column], want[:, column]), (got_S[h][:, column], want_S[:, column])):
            ref = ref.float()
            assert torch.equal(mine.isnan(), ref.isnan()) and torch.equal(mine.isinf(), ref.isinf())
            assert torch.equal(mine[mine.isinf()], ref[ref.isinf()])
            fine = ref.isfinite()
            if bool(fine.any()):
                size = float(ref[fine].abs().max())
                assert float((mine[fine] - ref[fine]).abs().max()) <= 1e-4 * max(1.0, size)
        if where[:5] == "large":
            assert bool(got[:, h * vdim + column].isfinite().all())
