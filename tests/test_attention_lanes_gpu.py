"""The prompt-attention kernel on tensor cores where its two lanes of work can go wrong: heads side by side and keys
split, a group's odd head, one to three key blocks (a lane without a step), page sizes that TMA takes and that it does
not, values seen in part beside whatever the cache holds (NaN and infinities), kept first keys."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, close_tensor_core_attention, ops, paged_setup, rnd

pytestmark = pytest.mark.gpu


def reference(q, dense, row_req, pos, nh, nkv, window, keep, scale):
    out = torch.zeros_like(q)
    for t in range(q.shape[0]):
        k, v = dense[row_req[t]]
        p = pos[t]
        lo = 0 if window is None else max(0, p - window)
        seen = [i for i in range(p + 1) if i >= lo or i < keep]
        for h in range(nh):
            g = h // (nh // nkv)
            out[t, h] = torch.softmax((k[seen][:, g] @ q[t, h]) * scale, 0) @ v[seen][:, g]
    return out


@pytest.mark.parametrize("split", [True, False, None])
@pytest.mark.parametrize("nh,nkv,d,page,window,keep", [
    (3, 1, 64, 16, None, 0), (2, 1, 128, 16, None, 0), (4, 4, 128, 128, None, 0), (5, 1, 64, 5, None, 0),
    (2, 2, 64, 256, 150, 20), (3, 1, 128, 24, 130, 0), (7, 1, 128, 12, 140, 33), (2, 1, 64, 8, 3, 1)])
def test_two_lanes(nh, nkv, d, page, window, keep, split):
    # (keys, first position of the portion): one to six key blocks, from an edge and from the middle of a block
    spans = [(1, 0), (127, 0), (128, 100), (129, 1), (257, 128), (400, 300), (700, 560)]
    k_pool, v_pool, tables, dense = paged_setup([n for n, _ in spans], nh, nkv, d, page, torch.bfloat16, seed=7)
    # what no row sees is not to be read as a number: infinities beside the NaN of the free rows
    v_pool[torch.isnan(v_pool).all(-1).all(-1).nonzero()[::2, 0]] = float("inf")
    row_req, pos, tiles = [], [], []
    for r, (n, start) in enumerate(spans):
        first = len(pos)
        row_req += [r] * (n - start)
        pos += list(range(start, n))
        tiles += [[first + off, min(128, n - start - off)] for off in range(0, n - start, 128)]
    tiles.append([0, 0])                                      # an idle tile of a padded step
    q = rnd(len(pos), nh, d, seed=8, dtype=torch.bfloat16)
    out = torch.full_like(q, 9.0)
    scale = 1.0 / math.sqrt(d)
    ops().attention_tcgen05(q.view(len(pos), -1), k_pool, v_pool, out.view(len(pos), -1), tables,
                            torch.tensor(row_req, dtype=torch.int32, device=DEV),
                            torch.tensor(pos, dtype=torch.int32, device=DEV),
                            torch.tensor(tiles, dtype=torch.int32, device=DEV), len(tiles), nh, nkv, d, page, window,
                            scale, keep_first=keep, split=split)
    torch.cuda.synchronize()
    ops().attention_tcgen05_check(d)
    assert torch.isfinite(out.float()).all()
    want = reference(q.float().cpu(), dense, row_req, pos, nh, nkv, window, keep, scale)
    close_tensor_core_attention(out, want)


def test_repeats_are_bitwise_equal():
    """The same launch many times over: a race between the lanes' products and the softmax would show."""
    nh, nkv, d, page, n = 7, 1, 128, 16, 1500
    k_pool, v_pool, tables, _ = paged_setup([n], nh, nkv, d, page, torch.bfloat16, seed=9)
    q = rnd(n, nh, d, seed=10, dtype=torch.bfloat16)
    tiles = [[off, min(128, n - off)] for off in range(0, n, 128)][::-1]
    args = [torch.zeros(n, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV),
            torch.tensor(tiles, dtype=torch.int32, device=DEV)]
    for split in (True, False):
        first = None
        for _ in range(40):
            out = torch.empty_like(q)
            ops().attention_tcgen05(q.view(n, -1), k_pool, v_pool, out.view(n, -1), tables, *args, len(tiles), nh, nkv, d,
                                    page, None, d ** -0.5, split=split)
            first = out if first is None else first
            assert torch.equal(out, first)
    ops().attention_tcgen05_check(d)
