"""quic_attn_prefill on the tensor cores, both forms (by the grid's size), against an fp32 softmax: ragged
ends of tiles, prompts that continue a cached one, and scores whose maxima keep growing."""

import pytest
import torch

from quic_cu_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,offs", [([128], [0]), ([129], [0]), ([193, 1, 64], [0, 0, 0]), ([257, 130], [63, 200]),
                                       ([130] * 45, [0] * 45), ([640, 200] * 6, [0, 65] * 6)], ids=lambda v: f"{len(v)}x{v[0]}")
@pytest.mark.parametrize("gain", [1.0, 8.0])
def test_prefill_attention_forms(lens, offs, gain):
    rows, n_seq, s_max = sum(lens), len(lens), max(n + o for n, o in zip(lens, offs)) + 7
    gen = torch.Generator(device="cuda").manual_seed(rows)
    q = torch.randn(14, rows, 64, device="cuda", generator=gen).half()
    ramp = torch.linspace(0.1, gain, s_max, device="cuda")[:, None]  # later keys score higher
    k = (torch.randn(n_seq, 2, s_max, 64, device="cuda", generator=gen) * ramp).half()
    v = torch.randn(n_seq, 2, s_max, 64, device="cuda", generator=gen).half()
    starts = [sum(lens[:i]) for i in range(n_seq)]
    table = torch.tensor([starts, lens, list(range(n_seq)), offs], dtype=torch.int32, device="cuda")
    out = torch.empty(rows, 896, device="cuda", dtype=torch.float16)
    kernels.check(kernels.lib().quic_attn_prefill(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), table[0].data_ptr(), table[1].data_ptr(), table[2].data_ptr(),
        table[3].data_ptr(), n_seq, max(lens), rows, s_max, n_seq, 0.125, out.data_ptr(), kernels.stream_ptr()), "attn_prefill")
    for i, (r0, n, o) in enumerate(zip(starts, lens, offs)):
        kk, vv = (t[i, :, :n + o].float().repeat_interleave(7, 0) for t in (k, v))
        score = q[:, r0:r0 + n].float() @ kk.transpose(1, 2) * 0.125
        seen = torch.arange(n + o, device="cuda") <= torch.arange(n, device="cuda")[:, None] + o
        want = torch.softmax(score.masked_fill(~seen, float("-inf")), -1) @ vv
        got = out[r0:r0 + n].view(n, 14, 64).transpose(0, 1).float()
        assert (got - want).norm() <= 2e-3 * want.norm()
    assert kernels.lib().quic_w4a16_tensor_status() == 0
