"""The 32-bit product on the tensor cores: one result whatever the tile and the cut of k, no further from 64 bits than a
chain of multiply-adds, and infinities, NaNs and the largest numbers as that chain has them."""
import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (1, 896, 896), (16, 127, 64), (17, 129, 68), (33, 128, 1020), (96, 300, 1028),
                                   (97, 257, 2048), (130, 640, 4864), (257, 128, 260), (500, 385, 3100)])
def test_tile_and_cut_change_no_bit(M, N, K):
    o = ops()
    a, w, bias = rnd(M, K, seed=1), rnd(N, K, seed=2), rnd(N, seed=3)
    outs = []
    for tile in range(5):
        for split in (False, True):
            outs.append(torch.full((M, N), 9.0, device=DEV))
            o.gemm_f32_tcgen05(a, w, bias, outs[-1], tile=tile, split=split)
    assert all(torch.equal(out, outs[0]) for out in outs)
    want = a.double() @ w.double().t() + bias.double()
    scale = a.double().abs() @ w.double().abs().t() + bias.double().abs()
    # pieces left out: 2^-24 of a product; a chunk's accumulator cuts at most a unit in the last place off 16 times,
    # those of the next orders at 2^-8; the K / 256 chunks, the groups and the bias round once each
    bound = (1 + 2 * 16 + 1 + K / 256 + K / 640 + 4) * 2.0 ** -24 * scale
    assert bool(((outs[0].double() - want).abs() <= bound).all())
    chain = torch.empty(M, N, device=DEV)
    o.gemm_f32(a, w, bias, chain, form=0)
    if K >= 768:
        assert float((outs[0].double() - want).norm()) <= float((chain.double() - want).norm())


@pytest.mark.parametrize("M,N,K", [(5, 130, 256), (70, 40, 2000)])
def test_numbers_without_pieces(M, N, K):
    o = ops()
    a, w = rnd(M, K, seed=4), rnd(N, K, seed=5)
    clean = torch.empty(M, N, device=DEV)
    o.gemm_f32_tcgen05(a, w, None, clean)
    inf = float("inf")
    a[1, 3], a[2, K - 1], a[3, 7] = inf, float("nan"), 3.4028e38
    w[9, 5], w[11, 3], w[20, 70] = -inf, 0.0, 3.4e38
    for tile in range(5):
        for split in (False, True):
            got, chain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
            o.gemm_f32_tcgen05(a, w, None, got, tile=tile, split=split)
            o.gemm_f32(a, w, None, chain, form=1)
            assert torch.equal(got.isnan(), chain.isnan()) and torch.equal(got.isinf(), chain.isinf())
            assert torch.equal(got[got.isinf()], chain[chain.isinf()])
            rows = [r for r in range(M) if r not in (1, 2, 3)]
            columns = [n for n in range(N) if n not in (9, 11, 20)]
            assert torch.equal(got[rows][:, columns], clean[rows][:, columns])
            assert torch.allclose(got[3][columns], chain[3][columns], rtol=1e-5)


def test_small_numbers_keep_their_bits():
    o = ops()
    a, w = rnd(8, 512, seed=6) * 2.0 ** -100, rnd(64, 512, seed=7)
    out = torch.empty(8, 64, device=DEV)
    o.gemm_f32_tcgen05(a, w, None, out)
    want = a.double() @ w.double().t()
    assert float((out.double() - want).abs().max()) <= 20 * 2.0 ** -24 * float((a.double().abs() @ w.double().abs().t()).max())


@pytest.mark.parametrize("K", [768, 2000])
def test_products_just_below_the_largest_number(K):
    """The first pieces of two numbers are rounded up: their product, or a sum of such products, may lie above the largest
    number where the numbers' own does not."""
    o = ops()
    M, N = 20, 130
    a, w = torch.zeros(M, K, device=DEV), torch.zeros(N, K, device=DEV)
    a[:, 5], w[:, 5] = 1.999 * 2.0 ** 63, 2.0 ** 64                      # 1.999 is 2 in sixteen bits
    a[3, 6], w[:, 6] = -1.999 * 2.0 ** 63, 2.0 ** 63                     # half of it off again
    w[7, 5], w[7, 6] = -1.9999 * 2.0 ** 63, 0.0
    w[9, 5] = 2.0 ** 66                                                  # truly above
    want = a.double() @ w.double().t()
    for tile in range(5):
        for split in (False, True):
            got = torch.empty(M, N, device=DEV)
            o.gemm_f32_tcgen05(a, w, None, got, tile=tile, split=split)
            columns = [n for n in range(N) if n != 9]
            assert bool(torch.isfinite(got[:, columns]).all()) and bool(got[:, 9].isinf().all())
            assert float(((got[:, columns].double() - want[:, columns]) / want[:, columns]).abs().max()) < 1e-6


@pytest.mark.parametrize("K", [768, 772, 896, 1024])
@pytest.mark.parametrize("M,N", [(1, 300), (65, 257)])
def test_numbers_of_one_sign(K, M, N):
    """What the tensor core cuts off instead of rounding adds up where all products have one sign: from 768 of k on it is still
    closer to 64 bits than a chain of multiply-adds."""
    o = ops()
    a, w = rnd(M, K, seed=21).abs(), rnd(N, K, seed=22).abs()
    got, chain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    o.gemm_f32_tcgen05(a, w, None, got)
    o.gemm_f32(a, w, None, chain, form=0)
    want = a.double() @ w.double().t()
    assert float((got.double() - want).norm()) <= float((chain.double() - want).norm())


@pytest.mark.parametrize("M", [1, 7, 100])
def test_where_the_tensor_cores_take_over(M):
    """By k and the operands' place alone, whatever the rows: 768 of k on 16 bytes and more."""
    o = ops()
    for K, off, tensor in ((764, 0, False), (768, 0, True), (770, 0, False), (772, 0, True), (768, 1, False)):
        room = rnd(M * K + 4, seed=23)
        a, w = room[off:off + M * K].view(M, K), rnd(90, K, seed=24)
        got, own, chain = (torch.empty(M, 90, device=DEV) for _ in range(3))
        o.gemm_f32(a, w, None, got)
        o.gemm_f32(a, w, None, chain, form=0)
        if tensor:
            o.gemm_f32_tcgen05(a, w, None, own)
        assert torch.equal(got, own if tensor else chain)
        assert not tensor or not torch.equal(own, chain)
