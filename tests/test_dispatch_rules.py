"""The host-side rules that choose how a product is cut: whatever the sizes, the pieces of k they
ask for are ones the kernels accept (no empty piece, whole 64-element blocks), and the rules stay
within the bounds their comments state.  Pure arithmetic: runs without a GPU."""
import itertools

import pytest

torch = pytest.importorskip("torch")

from tokenizer_b200.parts import gemm_bf16 as rules

ROWS = [1, 7, 16, 17, 33, 64, 100, 128, 129, 256, 300, 512, 777, 1024, 1536, 2048, 3000, 4096, 9000]
WIDTHS = [8, 64, 100, 128, 132, 256, 896, 1152, 1536, 4864, 9728, 20000]
DEPTHS = [8, 64, 72, 128, 264, 896, 1032, 2048, 4864, 8192]


def pieces_are_whole(K, pieces):
    """What the tile kernels check: with pieces of ceil(k_blocks / pieces) blocks, none is empty."""
    k_blocks = -(-K // 64)
    per = -(-k_blocks // pieces)
    return pieces >= 1 and (pieces - 1) * per < k_blocks


SIZES = list(itertools.product(ROWS, WIDTHS, DEPTHS))


def test_pieces_of_k_for_tile_products():
    cut = 0
    for M, N, K in SIZES:
        pieces = rules.choose_tile_k_splits(M, N, K)
        assert 1 <= pieces <= 8 and pieces_are_whole(K, pieces), (M, N, K, pieces)
        if pieces > 1:
            cut += 1
            # the consumer adds every plane: at most 8 MB of them, none of more than 4 MB
            assert M * N * 4 <= 4_000_000 and pieces * M * N * 4 <= 8_000_000, (M, N, K, pieces)
            assert N % 4 == 0                                    # planes are stored in 16-byte TMA rows
            assert -(-M // 128) * -(-N // 128) * 2 <= 148        # only when the tiles leave SMs idle
    assert cut > 100


def test_pieces_of_k_for_few_rows():
    for M, N, K in SIZES:
        pieces = rules.choose_k_splits(M, N, K)
        assert 1 <= pieces <= 16, (M, N, K, pieces)
        if pieces > 1:
            assert K // 256 >= pieces                            # a piece keeps at least 256 elements of k


def test_the_pair_rules_exclude_each_other():
    for M, N, K in SIZES:
        whole, halves = rules.use_pair(M, N, K), rules.use_pair_halves(M, N, K)
        assert not (whole and halves), (M, N, K)
        if halves:
            assert pieces_are_whole(K, 2) and N % 4 == 0 and M >= 1536
        if whole:
            assert N % 8 == 0 and -(-M // 256) * -(-N // 256) >= 44


def test_the_sizes_the_rules_were_measured_at():
    """Qwen2.5-0.5B: the down projection (N=896, K=4864) and the output projection (N=896, K=896)."""
    assert rules.choose_tile_k_splits(64, 896, 4864) == 8
    assert rules.choose_tile_k_splits(512, 896, 896) == 4            # 4 planes of 1.8 MB
    assert rules.choose_tile_k_splits(2048, 896, 4864) == 1          # planes of 7.3 MB: not on lone CTAs
    assert rules.use_pair_halves(2048, 896, 4864) and not rules.use_pair(2048, 896, 4864)
    assert rules.use_pair(4096, 896, 4864) and not rules.use_pair_halves(4096, 896, 4864)
    assert not rules.use_pair(1, 22528, 2048) and not rules.use_pair(128, 22528, 2048) and rules.use_pair(256, 22528, 2048)
    assert not rules.use_pair(2048, 896, 896) and not rules.use_pair_halves(2048, 1152, 896)


class Launches:
    """Stands for the libraries: notes the launchers that are called, answers every one of them with success."""

    def __init__(self, monkeypatch):
        from tokenizer_b200.kernels import ops
        self.names = []
        monkeypatch.setattr(ops, "_lib", lambda name: self)
        monkeypatch.setattr(ops, "_ptr", lambda t: None)
        monkeypatch.setattr(ops, "_stream", lambda: None)
        monkeypatch.setattr(ops, "linear_ring_supported", lambda M, N, K, k_splits=1, gated=False:
                            M <= ops.RING_MAX_ROWS and K // k_splits <= (4096 if M <= 16 else 1536))

    def __getattr__(self, name):
        return lambda *args: self.names.append(name.replace("tokb200_", "")) or 0


BF16 = dict(dtype=torch.bfloat16, device="meta")


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("on", [True, False])
def test_large_weights_of_few_rows(monkeypatch, M, on):
    """On rings up to 8 rows and on the tensor cores from 9 on; with the switch off on the kernel of small weights throughout."""
    from tokenizer_b200.kernels import ops
    launches = Launches(monkeypatch)
    monkeypatch.setattr(ops, "_RING", on)
    ops.gated_linear(torch.empty(M, 1536, **BF16), torch.empty(17920, 1536, **BF16), torch.empty(M, 8960, **BF16))
    rules.linear_bf16(torch.empty(M, 8192, **BF16), torch.empty(2048, 8192, **BF16), None, torch.bfloat16, partials_ok=True)
    rules.linear_bf16(torch.empty(M, 3584, **BF16), torch.empty(4608, 3584, **BF16), torch.empty(4608, device="meta"),
                      torch.bfloat16)
    want = ["linear_small_m_gated", "linear_small_m", "linear_small_m"] if not on else \
        ["linear_ring_gated", "linear_ring", "linear_ring"] if M <= 8 else \
        ["gemm_tcgen05_gated", "gemm_tcgen05_partials", "linear_ring"]
    assert launches.names == want


@pytest.mark.parametrize("M,N,K,want", [
    # tiles that fill their turns of 148, that do not, and k so short that it does not matter
    (9, 37888, 3584, "gemm_tcgen05"), (16, 28672, 2048, "gemm_tcgen05"), (9, 14336, 2048, "gemm_tcgen05"),
    (9, 8192, 4096, "linear_ring"), (16, 11264, 2048, "linear_ring"), (9, 20480, 3584, "linear_ring"), (9, 40960, 2560, "linear_ring"),
    (9, 20480, 896, "gemm_tcgen05"), (16, 22528, 1024, "gemm_tcgen05"), (9, 20480, 1024, "linear_ring"),
    # k beyond the ring kernel's
    (9, 4096, 5120, "linear_small_m"), (16, 8192, 5120, "linear_small_m"), (9, 11264, 5120, "gemm_tcgen05"),
    # a small weight: never; 17 to 32 rows: the ring where tiles are few
    (16, 9728, 896, "linear_small_m"), (17, 1024, 1024, "linear_ring"), (32, 4096, 1536, "linear_ring"),
    (17, 9728, 896, "gemm_tcgen05"), (33, 1024, 1024, "gemm_tcgen05"), (24, 4096, 2048, "gemm_tcgen05")])
def test_gated_products_of_few_rows(monkeypatch, M, N, K, want):
    from tokenizer_b200.kernels import ops
    launches = Launches(monkeypatch)
    ops.gated_linear(torch.empty(M, K, **BF16), torch.empty(N, K, **BF16), torch.empty(M, N // 2, **BF16))
    assert launches.names == [want + "_gated"]


@pytest.mark.parametrize("M,N,K,want", [
    (9, 1024, 13312, "linear_ring"), (16, 1024, 13312, "linear_ring"), (17, 1024, 13312, "gemm_tcgen05_partials"),
    (9, 1536, 8960, "gemm_tcgen05_partials"), (9, 4096, 12288, "gemm_tcgen05_partials"), (8, 4096, 12288, "linear_ring")])
def test_partial_sums_of_few_rows(monkeypatch, M, N, K, want):
    launches = Launches(monkeypatch)
    rules.linear_bf16(torch.empty(M, K, **BF16), torch.empty(N, K, **BF16), None, torch.bfloat16, partials_ok=True)
    assert launches.names == [want]


def test_what_is_no_integer_is_refused():
    """A float or a text that reaches a launcher as a size is an error, never another size."""
    from tokenizer_b200.kernels import ops
    for bad in (3.7, 4.0, "12", None):
        with pytest.raises(TypeError):
            ops._i(bad)
    assert [ops._i(v) for v in (3, True, -1)] == [3, 1, -1]
