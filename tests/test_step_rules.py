"""The rules that pick a kernel by a step's portions, on the measured sides of their lines, and that a captured step's key
tells apart what they tell apart."""
from types import SimpleNamespace

import pytest

torch = pytest.importorskip("torch")

from tokenizer_b200.parts import attention, part_class, recurrent


def delta(kind, heads, chunked=True):
    part = kind.__new__(kind)
    part.heads, part.chunked = heads, chunked
    return part


@pytest.mark.parametrize("q_lens,by_head,by_channel", [
    ([2048], True, True), ([512] + [1] * 15, True, True), ([512] + [1] * 63, False, False), ([31], False, False),
    ([64], True, False), ([128] * 4 + [8] * 28, False, False), ([512] * 8, True, True), ([1], False, False), ([], False, False)])
def test_delta_rules(q_lens, by_head, by_channel):
    for kind, want in ((recurrent.GatedDeltaNet, by_head), (recurrent.ChannelDeltaNet, by_channel)):
        assert delta(kind, 16)._in_chunks(q_lens) is want
        assert not delta(kind, 16, chunked=False)._in_chunks(q_lens)
        if q_lens:
            assert (delta(kind, 16).shape_key(q_lens) == "delta_chunks") is want


@pytest.mark.parametrize("heads,groups,q_lens,want", [
    (64, 8, [2048], True), (64, 8, [1905, 1096], True), (64, 8, [128], True), (64, 8, [127], False), (64, 8, [1], False),
    (64, 8, [], False), (128, 8, [255], True), (128, 8, [128], True), (48, 1, [1024], True), (32, 1, [2048], True),
    (24, 1, [2048], False), (16, 1, [2048], False), (16, 1, [1905, 1096], True), (16, 1, [128, 128], True),
    (64, 8, [622, 357, 1021], True), (64, 8, [512] * 4, True), (64, 8, [1200] * 4, True), (64, 8, [128] * 16, True),
    (64, 8, [64] * 16, False), (64, 8, [100] * 8, False), (64, 8, [2048] + [1] * 15, True), (64, 8, [1024, 600] + [1] * 20, True),
    (64, 8, [400, 1, 1, 1], True), (64, 8, [128, 1, 1, 1], True), (64, 8, [300] + [1] * 31, False), (64, 8, [1024] + [1] * 63, False),
    (64, 8, [256] * 4 + [1] * 60, False), (128, 8, [512] + [1] * 31, False), (64, 8, [130] * 16 + [2] * 16, False),
    (32, 1, [140] * 16 + [2] * 10, False),
    # B and C in pieces for every head or two: while the blocks fill one or two turns
    (64, 64, [2048], True), (64, 64, [1905, 1096], True), (64, 64, [512] * 4, False), (64, 64, [128] * 8, False),
    (64, 32, [128] * 4, False), (64, 16, [512] * 4, True), (32, 32, [128] * 3, False), (16, 16, [1905, 1096], False)])
def test_state_space_rule(heads, groups, q_lens, want):
    part = delta(part_class("mixer", "mamba2"), heads)
    part.vdim, part.groups = 64, groups
    assert part._in_chunks(q_lens) is want
    part.chunked = False
    assert not part._in_chunks(q_lens)
    part.chunked = True
    if q_lens:
        assert (part.shape_key(q_lens) == "ssm_chunks") is want


@pytest.mark.parametrize("longest,tokens,reach,d,want", [
    (128, 128, 128, 64, True), (384, 384, 512, 64, True), (385, 385, 512, 64, False), (256, 1024, 256, 64, True),
    (256, 1152, 256, 64, False), (200, 256, 1024, 64, False), (128, 128, 128, 128, False)])
def test_short_portions_of_near_keys(monkeypatch, longest, tokens, reach, d, want):
    monkeypatch.setattr(attention.ops, "prefill_attention_supported", lambda *a: True)
    part = attention.PagedAttention()
    part.nh, part.nkv, part.d = 14, 2, d
    ctx = SimpleNamespace(max_q_len=longest, n_tokens=tokens)
    group = SimpleNamespace(block_table=torch.empty(1, reach // 16), page_size=16)
    assert part._near(ctx, group, (None, 1)) is want and part._near(ctx, group, None) is False
    assert (part.shape_key([longest]) == "middle") is (longest < attention._WIDE_ALWAYS)


@pytest.mark.parametrize("heads,q_lens,want", [(4, [32], False), (4, [48], False), (4, [64], True), (8, [32], True)])
def test_delta_rule_of_few_heads(heads, q_lens, want):
    part = delta(recurrent.GatedDeltaNet, heads)
    assert part._in_chunks(q_lens) is want and (part.shape_key(q_lens) == "delta_chunks") is want


@pytest.mark.parametrize("heads,vdim,q_lens,want", [
    (8, 128, [128] * 16, False), (16, 64, [128] * 16, False), (16, 128, [128] * 16, True), (16, 32, [128] * 16, True),
    (4, 128, [128] * 16, True), (16, 16, [128] * 16, True), (8, 128, [512] * 8, True), (16, 128, [128], True)])
def test_channel_delta_rule_of_short_portions(heads, vdim, q_lens, want):
    part = delta(recurrent.ChannelDeltaNet, heads)
    part.vdim = vdim
    assert part._in_chunks(q_lens) is want and (part.shape_key(q_lens) == "delta_chunks") is want


def heads_of(nh, nkv, d=64, window=None, chunk=None):
    part = attention.PagedAttention()
    part.nh, part.nkv, part.d, part.window, part.chunk = nh, nkv, d, window, chunk
    return part


@pytest.mark.parametrize("nh,nkv,q_lens,window,cut", [
    (14, 2, [512], None, True), (14, 2, [2048], None, True), (14, 2, [384] * 4, None, False), (14, 2, [500] * 3, None, False),
    (14, 2, [700] * 2, None, True), (14, 2, [2048], 256, False), (14, 2, [480] + [1] * 31, None, True), (32, 8, [640], None, True),
    (32, 8, [500] * 2, None, False), (32, 8, [1536], None, False), (28, 4, [200] * 5, None, True), (28, 4, [2048], None, False),
    (4, 4, [4096], None, True)])
def test_where_keys_are_cut(nh, nkv, q_lens, window, cut):
    part = heads_of(nh, nkv, window=window)
    assert part._cut_keys(q_lens) is cut
    # a captured step's key tells the two apart, in whatever order the requests come
    assert part.shape_key(q_lens).endswith("two heads a block" + ("+1" if 1 in q_lens else "")) is not cut
    assert part.shape_key(q_lens) == part.shape_key(q_lens[::-1])
    assert part.shape_key([n for n in q_lens if n > 1]).endswith("two heads a block") is not cut


@pytest.mark.parametrize("nh,nkv,tokens,reach,want", [
    (14, 2, 1024, 256, True), (32, 8, 256, 256, True), (32, 8, 384, 512, False), (32, 8, 512, 256, False), (64, 8, 128, 128, True),
    (64, 8, 256, 256, False)])
def test_near_keys_of_many_heads(monkeypatch, nh, nkv, tokens, reach, want):
    monkeypatch.setattr(attention.ops, "prefill_attention_supported", lambda *a: True)
    ctx = SimpleNamespace(max_q_len=96, n_tokens=tokens)
    group = SimpleNamespace(block_table=torch.empty(1, reach // 16), page_size=16)
    assert heads_of(nh, nkv)._near(ctx, group, (None, 1)) is want
