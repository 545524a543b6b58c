"""The state-space recurrence in chunks against the same recurrence token by token in 64 bits: portions of one token to
several chunks and their remainders, continued portions, idle rows, empty requests, decays next to one and next to zero,
states of fewer than 128 lanes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("heads,groups,vdim,n_state,shift,dtype", [
    (4, 2, 64, 128, -3.0, torch.float32), (3, 1, 32, 72, 3.0, torch.float32), (2, 2, 96, 100, 0.0, torch.bfloat16)])
def test_against_the_recurrence(heads, groups, vdim, n_state, shift, dtype):
    from tokenizer_b200.kernels import ops as o
    assert o.ssd_chunks_supported(vdim, n_state)
    lengths = [[1, 33, 0, 64, 95, 32], [31, 2, 40, 1, 0, 70]]
    n_req, inner, share = len(lengths[0]), heads * vdim, heads // groups
    g = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g)
    dt_bias, a_log, skip = rnd(heads) + shift, rnd(heads) * 0.5, rnd(heads)
    S = [rnd(heads, n_state, vdim) * 0.3 for _ in range(n_req)]
    size = -(-(inner * n_state + 12) // 4) * 4
    slots = torch.randperm(n_req, generator=g)
    dev = torch.full((n_req, size), 7.0, device=DEV)
    for r in range(n_req):
        dev[slots[r], :inner * n_state] = S[r].transpose(1, 2).reshape(-1).to(DEV)
    S = [s.double() for s in S]
    for portion in lengths:
        starts = [0]
        for n in portion:
            starts.append(starts[-1] + n)
        rows = starts[-1] + 3
        xbc, proj = rnd(rows, inner + 2 * groups * n_state), rnd(rows, heads + 11).to(dtype)
        y = torch.full((rows, inner), 9.0, device=DEV)
        o.ssd_chunks(xbc.to(DEV), proj.to(DEV), 11, dt_bias.to(DEV), a_log.to(DEV), skip.to(DEV), heads, groups, vdim, n_state,
                     dev, torch.tensor(starts, dtype=torch.int32, device=DEV), slots.int().to(DEV), y)
        got, got_state = y.cpu().double(), dev[slots.to(DEV)].cpu().double()
        assert bool((got[starts[-1]:] == 9.0).all())
        dt = torch.nn.functional.softplus(proj[:, 11:].double() + dt_bias.double())
        keep = torch.exp(-torch.exp(a_log.double()) * dt)
        x = xbc[:, :inner].double().view(rows, heads, vdim)
        b, c = (t.reshape(rows, groups, n_state).double().repeat_interleave(share, 1)
                for t in torch.split(xbc[:, inner:], groups * n_state, dim=1))
        for r, n in enumerate(portion):
            want = torch.empty(n, heads, vdim, dtype=torch.float64)
            for i, t in enumerate(range(starts[r], starts[r + 1])):
                S[r] = keep[t][:, None, None] * S[r] + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
                want[i] = torch.einsum("hnv,hn->hv", S[r], c[t]) + skip.double()[:, None] * x[t]
            # 32-bit sums of 128 products, a chain of three chunks at most: some tens of 2^-24 of the largest value
            if n:
                assert float((got[starts[r]:starts[r + 1]] - want.reshape(n, -1)).abs().max()) < 1e-5 * max(1.0, float(want.abs().max()))
            m = got_state[r, :inner * n_state].view(heads, vdim, n_state).transpose(1, 2)
            assert float((m - S[r]).abs().max()) < 1e-5 * max(1.0, float(S[r].abs().max()))
        assert bool((got_state[:, inner * n_state:] == 7.0).all())


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [1, 15, 17, 30, 45])
def test_a_token_changes_nothing_before_it(value, at):
    """An infinity or NaN in a token's x, B, C or step leaves the rows in front of it in the same chunk as they are, bit for
    bit."""
    from tokenizer_b200.kernels import ops as o
    heads, groups, vdim, n_state, n = 2, 1, 32, 128, 50
    inner = heads * vdim
    g = torch.Generator().manual_seed(12)
    rnd = lambda *s: torch.randn(*s, generator=g).to(DEV)
    dt_bias, a_log, skip, first = rnd(heads), rnd(heads), rnd(heads), rnd(1, inner * n_state)
    xbc, proj = rnd(n, inner + 2 * groups * n_state), rnd(n, heads)

    def run(xbc, proj):
        y, state = torch.empty(n, inner, device=DEV), first.clone()
        o.ssd_chunks(xbc, proj, 0, dt_bias, a_log, skip, heads, groups, vdim, n_state, state,
                     torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV), y)
        return y
    want = run(xbc, proj)
    assert torch.isfinite(want).all()
    for column in (3, inner + 7, inner + n_state + 9, -1):    # x, B, C, the step
        bad, bad_proj = xbc.clone(), proj.clone()
        if column < 0:
            bad_proj[at, 0] = value
        else:
            bad[at, column] = value
        got = run(bad, bad_proj)
        assert torch.equal(got[:at], want[:at])
        assert not torch.isfinite(got[at:]).all()
        if column == 3:                                       # a column of x meets no other
            others = [c for c in range(inner) if c != 3]
            assert torch.equal(got[:, others], want[:, others])


def in_chunks(xbc, dt_in, dt_bias, a_log, skip, heads, groups, vdim, n_state, S):
    """One request by the chunks' own sums in 64 bits: S [heads, n_state, vdim] moves on in place; the rows' outputs."""
    n, inner, share = xbc.shape[0], heads * vdim, heads // groups
    xbc = xbc.double()
    dt = torch.nn.functional.softplus(dt_in.double() + dt_bias.double())
    keep = torch.exp(-torch.exp(a_log.double()) * dt)
    out = torch.empty(n, heads, vdim, dtype=torch.float64)
    for t0 in range(0, n, 32):
        rows = slice(t0, min(n, t0 + 32))
        for h in range(heads):
            g = h // share
            x = xbc[rows, h * vdim:(h + 1) * vdim]
            b = xbc[rows, inner + g * n_state:inner + (g + 1) * n_state]
            c = xbc[rows, inner + (groups + g) * n_state:inner + (groups + g + 1) * n_state]
            a, d, m = keep[rows, h], dt[rows, h], x.shape[0]
            decay = [[float(torch.prod(a[s + 1:t + 1])) for s in range(m)] for t in range(m)]
            for t in range(m):
                v = sum(decay[t][s] * (c[t] @ b[s]) * d[s] * x[s] for s in range(t + 1))
                out[t0 + t, h] = v + skip[h].double() * x[t] + torch.prod(a[:t + 1]) * (c[t] @ S[h])
            S[h] = torch.prod(a) * S[h] + sum(b[s][:, None] * (decay[m - 1][s] * d[s] * x[s])[None, :] for s in range(m))
    return out.reshape(n, inner)


@pytest.mark.parametrize("where", ["matrix", "x", "B", "C", "large matrix", "large x", "large product"])
@pytest.mark.parametrize("n", [20, 70])
def test_numbers_without_pieces(where, n):
    """Infinities, and numbers that round to one in 16 bits, in the matrix or in what comes in: outputs and matrix hold numbers,
    infinities (with their signs) and NaN where the same sums in 64 bits do."""
    from tokenizer_b200.kernels import ops as o
    heads, groups, vdim, n_state = 2, 1, 64, 100
    inner, inf = heads * vdim, float("inf")
    g = torch.Generator().manual_seed(17)
    rnd = lambda *s: torch.randn(*s, generator=g)
    dt_bias, a_log, skip, S = rnd(heads) - 5.0, rnd(heads) * 0.3, rnd(heads), rnd(heads, n_state, vdim)
    xbc, proj = rnd(n, inner + 2 * n_state), rnd(n, heads)
    if where == "matrix":
        S[0, 3, 5], S[1, 99, 63] = inf, -inf
    elif where == "x":
        xbc[6, 5], xbc[18, vdim + 40] = inf, -inf
    elif where == "B":
        xbc[9, inner + 50] = inf
    elif where == "C":
        xbc[9, inner + n_state + 50] = -inf
    elif where == "large matrix":                   # one lane of it alone meets C, at an eighth
        xbc[:, inner + n_state + 3] *= 2.0 ** -4
        S[0, 3, 5], S[1, 3, 63] = 3.4e38, -3.395e38
    elif where == "large x":
        xbc[:, inner:] *= 2.0 ** -4
        skip *= 2.0 ** -3
        xbc[6, 5], xbc[18, vdim + 40] = 3.4e38, -3.395e38
    else:                                           # below the largest number by the numbers, above it by their first pieces
        xbc[:, inner + n_state:] = 0
        xbc[0, inner + n_state + 3], S[0, 3, 5], dt_bias[0], skip[0] = 2.0, 1.999 * 2.0 ** 126, -30.0, 0.0
    state = S.transpose(1, 2).reshape(1, -1).to(DEV)
    y = torch.empty(n, inner, device=DEV)
    o.ssd_chunks(xbc.to(DEV), proj.to(DEV), 0, dt_bias.to(DEV), a_log.to(DEV), skip.to(DEV), heads, groups, vdim, n_state, state,
                 torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV), y)
    want_S = S.double()
    want = in_chunks(xbc, proj, dt_bias, a_log, skip, heads, groups, vdim, n_state, want_S)
    assert where[:5] != "large" or bool(want.isfinite().all())
    for got, ref in ((y.cpu(), want), (state.cpu().view(heads, vdim, n_state).transpose(1, 2), want_S)):
        ref32 = ref.float()
        assert torch.equal(got.isnan(), ref32.isnan()) and torch.equal(got.isinf(), ref32.isinf())
        assert torch.equal(got[got.isinf()], ref32[ref32.isinf()])
        fine = ref32.isfinite()
        size = ref[fine].abs().reshape(-1)
        # what meets a large number is as large, the rest as above: an element's error against its own size or that of its row
        assert bool(((got[fine].double() - ref[fine]).abs().reshape(-1) <= 1e-4 * size + 1e-4 * (1.0 + size)).all())


@pytest.mark.parametrize("heads,groups,lengths", [(16, 1, [2048]), (64, 8, [1905, 1096]), (64, 8, [300])])
def test_error_of_outputs_and_states(heads, groups, lengths):
    """Pieces on the tensor cores against plain multiply-adds token by token, both against 64 bits, at memories of tens to
    hundreds of tokens: measured 1.11 to 1.13 times its error in the outputs and 0.95 to 1.03 times in the matrix (with one sum
    for all products of pieces 1.18 to 1.25 and 1.06 to 1.18)."""
    from tokenizer_b200.kernels import ops as o
    vdim, n_state, rows = 64, 128, sum(lengths)
    inner, share = heads * vdim, heads // groups
    g = torch.Generator(device=DEV).manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    dt_bias, a_log, skip = 0.5 * rnd(heads) - 3.5, 0.5 * rnd(heads), 1 + 0.2 * rnd(heads)
    xbc, proj = torch.nn.functional.silu(rnd(rows, inner + 2 * groups * n_state)), rnd(rows, heads)
    starts = [sum(lengths[:r]) for r in range(len(lengths) + 1)]
    first = 0.3 * rnd(len(lengths), heads, vdim, n_state)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    found = []
    for scan in (o.ssd_chunks, o.mamba2_scan):
        state, y = first.reshape(len(lengths), -1).clone(), torch.empty(rows, inner, device=DEV)
        scan(xbc, proj, 0, dt_bias, a_log, skip, heads, groups, vdim, n_state, state, ints(starts), ints(range(len(lengths))), y)
        found.append((y, state))
    dt = torch.nn.functional.softplus(proj.double() + dt_bias.double())
    keep = torch.exp(-torch.exp(a_log.double()) * dt)
    x = xbc[:, :inner].double().view(rows, heads, vdim)
    b, c = (t.reshape(rows, groups, n_state).double().repeat_interleave(share, 1)
            for t in torch.split(xbc[:, inner:], groups * n_state, dim=1))
    want, states = torch.empty(rows, heads, vdim, dtype=torch.float64, device=DEV), []
    for r in range(len(lengths)):
        S = first[r].double()
        for t in range(starts[r], starts[r + 1]):
            S = keep[t][:, None, None] * S + (dt[t][:, None] * x[t])[:, :, None] * b[t][:, None, :]
            want[t] = (S * c[t][:, None, :]).sum(-1) + skip.double()[:, None] * x[t]
        states.append(S.reshape(-1))
    want = (want.reshape(rows, -1), torch.stack(states))
    chunks, tokens = ([float((got.double() - ref).norm() / ref.norm()) for got, ref in zip(pair, want)] for pair in found)
    assert chunks[0] <= 1.16 * tokens[0] and chunks[1] <= 1.05 * tokens[1]
