"""Products on tcgen05 whose weight ends inside a warp's 32 rows, in blocks that have more to do behind that tile: the lanes
past the last row store nothing and are back for the next tile's loads from tensor memory, which a warp makes as a whole."""
import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [3, 17, 64])
@pytest.mark.parametrize("N,K,S", [(128 * 75 + 4, 512, 4), (128 * 74 + 20, 1024, 8), (128 * 148 + 60, 256, 2)])
def test_few_rows_in_pieces_of_k(M, N, K, S):
    o = ops()
    a, w = rnd(M, K, seed=91, dtype=torch.bfloat16), rnd(N, K, seed=92, dtype=torch.bfloat16, scale=0.1)
    room = torch.full((S * M * N + 64,), 7.0, device=DEV)
    o.gemm_tcgen05_partials(a, w, room[:S * M * N].view(S, M, N))
    o.gemm_tcgen05_check()
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    # a 2^-23 of the products' sizes at each of K / 16 steps
    assert bool(((room[:S * M * N].view(S, M, N).double().sum(0) - want).abs() <= size * (K / 16 + 2) * 2.0 ** -23).all())
    assert bool((room[S * M * N:] == 7.0).all())


@pytest.mark.parametrize("M,N,K,tile", [(160, 128 * 74 + 1, 1300, 4), (97, 128 * 150 + 31, 700, 2), (16, 33, 2600, 0), (40, 97, 1920, 1)])
def test_32_bit_rows_with_groups_of_k_one_after_another(M, N, K, tile):
    o = ops()
    a, w, bias = rnd(M, K, seed=93), rnd(N, K, seed=94), rnd(N, seed=95)
    room = torch.full((M * N + 64,), 7.0, device=DEV)
    o.gemm_f32_tcgen05(a, w, bias, room[:M * N].view(M, N), tile=tile, split=False)
    want = a.double() @ w.double().t() + bias.double()
    size = a.double().abs() @ w.double().abs().t() + bias.double().abs()
    # the bound of test_gemm_f32_tcgen05_gpu.py, where it is derived
    bound = (1 + 2 * 16 + 1 + K / 256 + K / 640 + 4) * 2.0 ** -24 * size
    assert bool(((room[:M * N].view(M, N).double() - want).abs() <= bound).all())
    assert bool((room[M * N:] == 7.0).all())
    o.raise_if_error()


@pytest.mark.parametrize("M,N,K", [(70, 131, 64), (129, 1, 72), (100, 40, 640)])
def test_rows_of_no_whole_pitch(M, N, K):
    """More than 64 rows into an output whose rows are no multiple of 16 bytes: lanes behind the last row and columns behind the last."""
    o = ops()
    a, w = rnd(M, K, seed=96, dtype=torch.bfloat16), rnd(N, K, seed=97, dtype=torch.bfloat16, scale=0.1)
    out = torch.full((M, N), 9.0, device=DEV)
    o.gemm_tcgen05(a, w, None, out)
    o.gemm_tcgen05_check()
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    assert bool(((out.double() - want).abs() <= size * (K / 16 + 2) * 2.0 ** -23).all())
