"""Decode attention left to choose its kernel (quic_attn_decode, splits 0) against an fp32 softmax:
tile and split boundaries, ragged starts and ends, rows without tokens, strided planes, large values in
every place that no row attends to."""

from __future__ import annotations

import pytest
import torch

from quic_cu_b200 import kernels

pytestmark = pytest.mark.gpu

HEADS, KV, HD = kernels.HEADS, kernels.KV_HEADS, kernels.HEAD_DIM


@pytest.mark.parametrize("rows,tokens", [(1, 1), (1, 64), (2, 65), (1, 1279), (1, 1281), (3, 5121), (37, 1290), (49, 2000),
                                         (74, 1300), (148, 256), (149, 256), (149, 257), (300, 700)])
def test_attention_over_row_ranges(rows, tokens):
    gen = torch.Generator(device="cuda").manual_seed(rows * 10007 + tokens)
    q = torch.randn(rows, HEADS, HD, device="cuda", generator=gen).half()
    k, v = (torch.randn(rows, KV, tokens + 5, HD, device="cuda", generator=gen).half() for _ in range(2))
    start = torch.randint(0, tokens // 3 + 1, (rows,), device="cuda", generator=gen).int()
    end = torch.randint(2 * tokens // 3, tokens + 1, (rows,), device="cuda", generator=gen).int()
    start[-1], end[-1] = 0, tokens
    if rows > 2:
        start[0], end[0] = tokens // 2, tokens // 2  # nothing to attend to
        start[1], end[1] = tokens - 1, tokens + 3    # clamped at the cache's end
    at = torch.arange(tokens + 5, device="cuda")
    live = (at >= start[:, None]) & (at < end[:, None].clamp(max=tokens))
    for t in (k, v):
        t.masked_fill_(~live[:, None, :, None], 1e4)
    out = torch.empty_like(q)
    scratch = torch.zeros(kernels.lib().quic_attn_scratch_bytes(rows, kernels.lib().quic_attn_pick_splits(rows, tokens)),
                          dtype=torch.uint8, device="cuda")
    kernels.check(kernels.lib().quic_attn_decode(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), k.stride(0), k.stride(1), start.data_ptr(), end.data_ptr(), tokens,
        0.125, out.data_ptr(), rows, 0, scratch.data_ptr(), kernels.stream_ptr()), "attn_decode")
    kf, vf = (t.float().repeat_interleave(HEADS // KV, 1) for t in (k, v))
    score = torch.einsum("bhd,bhtd->bht", q.float(), kf) * 0.125
    prob = torch.softmax(score.masked_fill(~live[:, None], float("-inf")), -1).nan_to_num(0.0)
    want = torch.einsum("bht,bhtd->bhd", prob, vf)
    assert torch.isfinite(out).all()
    assert (out.float() - want).norm() <= 2e-3 * want.norm()


@pytest.mark.parametrize("rows,tokens,offset", [(1, 4096, 1), (3, 2500, 1), (2, 3000, 3), (1, 700, 2), (20, 900, 2), (1, 4096, 2)])
def test_queries_at_any_address_that_was_taken(rows, tokens, offset):
    """q starts `offset` values into its allocation; keys and values outside the rows' tokens are NaN."""
    gen = torch.Generator(device="cuda").manual_seed(rows + tokens)
    buf = torch.randn(rows * HEADS * HD + 8, device="cuda", generator=gen).half()
    q = buf[offset:offset + rows * HEADS * HD].view(rows, HEADS, 1, HD)
    k, v = (torch.randn(rows, KV, tokens, HD, device="cuda", generator=gen).half() for _ in range(2))
    pads = torch.tensor([(37 * i + 5) % (tokens // 2) for i in range(rows)], dtype=torch.int32, device="cuda")
    dead = torch.arange(tokens, device="cuda") < pads[:, None]
    if offset % 2 == 0:  # (the scalar kernel multiplies what it masks)
        for t in (k, v):
            t.masked_fill_(dead[:, None, :, None], float("nan"))
    got = kernels.flash_attn_decode().forward(q, k, v, 0.125, pads)
    kf, vf = (t.float().masked_fill(dead[:, None, :, None], 0).repeat_interleave(HEADS // KV, 1) for t in (k, v))
    score = torch.einsum("bhod,bhtd->bhot", q.float(), kf) * 0.125
    want = torch.softmax(score.masked_fill(dead[:, None, None], float("-inf")), -1) @ vf
    assert (got.float() - want).norm() <= 2e-3 * want.norm()


@pytest.mark.parametrize("rows,tokens", [(1, 100), (16, 1024)])
def test_queries_at_an_odd_address_are_refused_where_they_are_read_in_pairs(rows, tokens):
    buf = torch.zeros(rows * HEADS * HD + 8, device="cuda").half()
    k = torch.zeros(rows, KV, tokens, HD, device="cuda").half()
    with pytest.raises(RuntimeError, match="aligned"):
        kernels.flash_attn_decode().forward(buf[1:1 + rows * HEADS * HD].view(rows, HEADS, 1, HD), k, k)


@pytest.mark.parametrize("rows,longest", [(1, 4200), (2, 4161), (3, 4500), (9, 4097), (16, 3300), (17, 4200), (20, 3500), (21, 1990), (40, 2100)])
def test_decode_steps_over_long_rows_match_a_prefill_of_the_same_tokens(tiny_model, rows, longest):
    """The attention over ranges of a cluster inside a decode step (rows beyond 4096 tokens, more CTAs of 512 tokens than
    SMs, 21 rows and more from three ranges on): what the step appends in the second layer went through its attention.  A prefill of
    prompt + token leaves the same there, up to the roundings to fp16 (34 of 2^-11 / sqrt(3), see test_rows_chain_gpu.py)."""
    from quic_cu_b200 import model as qmodel

    _, _, state, config = tiny_model
    state = {k: v * 0.25 if k.endswith("weight_scale") else v for k, v in state.items()}
    net = qmodel.from_state_dict(state, config)
    net.use_persist = False
    bound = min(qmodel._ctx_bucket(longest + 1, rows), 4608)
    assert kernels.lib().quic_decode_attention_form(rows, bound) == kernels.ATTN_FLOW
    gen = torch.Generator().manual_seed(rows)
    lens = torch.randint(1, longest, (rows,), generator=gen).tolist()
    lens[0] = longest
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    slots = torch.randperm(rows, generator=gen).tolist()
    cache, other = (net.new_cache(n_slots=rows, s_max=4608) for _ in range(2))
    first, _ = net.prefill(cache, slots, prompts)
    net.decode(cache, slots, 1)
    net.prefill(other, slots, [torch.cat([p, first[i:i + 1].cpu()]) for i, p in enumerate(prompts)])
    for i, (slot, n) in enumerate(zip(slots, lens)):
        got, want = cache.kv[1, :, slot, :, n].float(), other.kv[1, :, slot, :, n].float()
        worst = ((got - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)).max().item()
        assert worst < 2 * (34 / 3) ** 0.5 * 2 ** -11, (i, n, worst)
