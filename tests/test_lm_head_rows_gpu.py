"""quic_lm_head_argmax around the row counts where its kernel, its chunks and its scratch change."""

import pytest
import torch

from quic_cu_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 16, 17, 31, 32, 33, 128, 129, 257])
@pytest.mark.parametrize("vocab", [2048, 1000])
def test_logits_and_tokens_by_row_count(rows, vocab):
    gen = torch.Generator(device="cuda").manual_seed(rows + vocab)
    embed = torch.randn(vocab, kernels.HIDDEN, device="cuda", generator=gen).half()
    for _ in range(2):  # again on the scratch that the first call left
        x = torch.randn(rows, kernels.HIDDEN, device="cuda", generator=gen).half()
        tokens, logits = kernels.lm_head_argmax(x, embed, want_logits=True)
        want = x.float() @ embed.float().T
        assert (logits.float() - want).norm() <= 1e-3 * want.norm()
        assert torch.equal(tokens, logits.float().argmax(-1))
