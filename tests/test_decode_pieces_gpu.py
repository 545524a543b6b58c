"""Decode attention where the launch's choice of pieces turns: clusters of as many blocks as the device's groups of
multiprocessors hold and one pair more, rows left whole, rows cut."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, attention_reference, close_tensor_core_attention, ops, paged_setup, rnd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh,nkv,d,rows,longest", [
    (28, 4, 128, 4, 2000), (28, 4, 128, 3, 2000), (12, 2, 128, 12, 1500), (14, 2, 64, 24, 1500),      # clusters or scratch
    (8, 8, 128, 19, 4400), (8, 8, 128, 18, 4400)])                                                     # whole from 148 pairs on
def test_against_the_reference(nh, nkv, d, rows, longest):
    lengths = [max(1, longest - 37 * i) for i in range(rows)]
    k_pool, v_pool, tables, dense = paged_setup(lengths, nh, nkv, d, 16, torch.bfloat16, seed=41)
    pos = [n - 1 for n in lengths]
    q = rnd(rows, nh, d, seed=42, dtype=torch.bfloat16)
    out = torch.full_like(q, 9.0)
    scale = 1.0 / math.sqrt(d)
    want = attention_reference(q.float().cpu(), dense, list(range(rows)), pos, nh, nkv, None, scale)
    for _ in range(2):          # twice: counters of a merge are left ready
        ops().decode_attention(q.view(rows, nh * d), k_pool, v_pool, out.view(rows, nh * d), tables,
                               torch.arange(rows, dtype=torch.int32, device=DEV),
                               torch.tensor(pos, dtype=torch.int32, device=DEV), nh, nkv, d, 16, None, scale)
        close_tensor_core_attention(out, want)
        out.fill_(9.0)


@pytest.mark.parametrize("nh,nkv,rows,longest,skewed", [(8, 8, 20, 5000, False), (8, 8, 20, 5000, True), (4, 2, 80, 4600, False),
                                                        (8, 8, 19, 9300, True), (8, 8, 19, 9300, False)])
@pytest.mark.parametrize("even", [None, 0, 1])
def test_long_rows_whole_or_cut(nh, nkv, rows, longest, skewed, even):
    """Rows beyond 4,096 keys in one piece, in two, or in the short pieces of a launch that says nothing: the same attention, in
    any order of the rows, idle ones among them; counters are left ready."""
    d = 128
    lengths = [longest if not i % 19 else 700 + 13 * i for i in range(rows)] if skewed else [longest - 29 * i for i in range(rows)]
    k_pool, v_pool, tables, dense = paged_setup(lengths, nh, nkv, d, 16, torch.bfloat16, seed=43)
    pos = [n - 1 for n in lengths]
    q = rnd(rows, nh, d, seed=44, dtype=torch.bfloat16)
    scale = 1.0 / math.sqrt(d)
    want = attention_reference(q.float().cpu(), dense, list(range(rows)), pos, nh, nkv, None, scale)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    order = sorted(range(rows), key=lambda i: -lengths[i])
    order[3] = -1
    idle = [i for i in range(rows) if i not in order]
    for served in (None, order):
        out = torch.full_like(q, 9.0)
        for _ in range(2):
            ops().decode_attention(q.view(rows, nh * d), k_pool, v_pool, out.view(rows, nh * d), tables, ints(range(rows)), ints(pos),
                                   nh, nkv, d, 16, None, scale, rows=None if served is None else ints(served),
                                   even=None if even is None else ints([even]))
            if served is not None:
                assert bool((out[idle] == 9.0).all())
                out[idle] = want[idle].to(out)
            close_tensor_core_attention(out, want)
            out.fill_(9.0)
