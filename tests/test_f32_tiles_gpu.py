"""The 32-bit kernels for prompts: the product's bits do not depend on the form a tile count picks, and attention over
tiles of rows gives the bits of the kernel for single rows."""
import pytest
import torch

from test_kernels_gpu import DEV, ops, paged_setup, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (3, 33, 7), (16, 896, 64), (33, 130, 36), (65, 129, 100), (777, 1152, 896),
                                   (130, 4100, 33), (2100, 896, 130), (513, 2570, 31)])
def test_product_rows_do_not_depend_on_the_batch(M, N, K):
    o = ops()
    a, w, bias = rnd(M, K, seed=1), rnd(N, K, seed=2), rnd(N, seed=3)
    out = torch.full((M, N), 9.0, device=DEV)
    o.gemm_f32(a, w, bias, out)
    want = a.double() @ w.double().t() + bias.double()
    # a chain of K roundings, each of a partial sum that stays below sum |a w|
    bound = (K + 2) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t() + bias.double().abs())
    assert bool(((out.double() - want).abs() <= bound + 1e-30).all())
    for rows in (slice(0, 1), slice(M // 2, min(M, M // 2 + 5)), slice(max(0, M - 40), M)):
        part = torch.empty(a[rows].shape[0], N, device=DEV)
        o.gemm_f32(a[rows].contiguous(), w, bias, part)
        assert torch.equal(part, out[rows])
    few = torch.empty(M, min(N, 40), device=DEV)
    o.gemm_f32(a, w[:min(N, 40)].contiguous(), bias[:min(N, 40)].contiguous(), few)
    assert torch.equal(few, out[:, :min(N, 40)])


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (5, 33, 7), (64, 128, 16), (129, 257, 100), (300, 130, 36)])
def test_every_form_of_the_product_gives_the_same_bits(M, N, K):
    o = ops()
    a, w, bias = rnd(M, K, seed=4), rnd(N, K, seed=5), rnd(N, seed=6)
    outs = [torch.full((M, N), 9.0, device=DEV) for _ in range(6)]
    for form, out in enumerate(outs):
        o.gemm_f32(a, w, bias, out, form=form)
    assert all(torch.equal(out, outs[0]) for out in outs)
    with pytest.raises(Exception):
        o.gemm_f32(a, w, bias, outs[0], form=6)


@pytest.mark.parametrize("nh,nkv,d,page,sink,softcap", [
    (4, 2, 64, 16, False, None), (3, 1, 128, 5, True, None), (2, 2, 64, 64, True, 20.0), (7, 1, 64, 16, False, None)])
def test_attention_tiles_give_the_bits_of_single_rows(nh, nkv, d, page, sink, softcap):
    o = ops()
    spans = [(1, 0), (64, 0), (65, 3), (128, 100), (130, 0), (400, 250)]
    k_pool, v_pool, tables, _ = paged_setup([n for n, _ in spans], nh, nkv, d, page, torch.float32, seed=4)
    row_req, pos, tiles = [], [], []
    for r, (n, start) in enumerate(spans):
        first = len(pos)
        row_req += [r] * (n - start)
        pos += list(range(start, n))
        tiles += [[first + off, min(64, n - start - off)] for off in range(0, n - start, 64)]
    tiles.append([0, 0])
    q = rnd(len(pos), nh * d, seed=5)
    args = [torch.tensor(x, dtype=torch.int32, device=DEV) for x in (row_req, pos, tiles)]
    sinks = rnd(nh, seed=6) if sink else None
    want, got = torch.empty_like(q), torch.full_like(q, 9.0)
    o.paged_attention_generic(q, k_pool, v_pool, want, tables, args[0], args[1], nh, nkv, d, page, None, d ** -0.5,
                              sink=sinks, softcap=softcap)
    o.paged_attention_f32_tiles(q, k_pool, v_pool, got, tables, *args, len(tiles), nh, nkv, d, page, d ** -0.5, sink=sinks,
                                softcap=softcap)
    assert torch.isfinite(want).all() and torch.equal(got, want)
