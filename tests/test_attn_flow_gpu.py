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
