"""A serving queue whose steps of more than 16 rows run beside prefills of every form on another stream."""

from types import SimpleNamespace

import pytest
import torch

from quic_cu_b200 import kernels as K
from quic_cu_b200.config import EngineConfig
from quic_cu_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net(tiny_model):
    """The tiny model with its tokens paired: the final norm's signs make the best next token of t the one paired with it by a
    wide margin, so that a rounding (prompts admitted together or one by one) changes no token."""
    from quic_cu_b200 import model as qmodel

    _, _, state, config = tiny_model
    gen = torch.Generator().manual_seed(3)
    signs = torch.where(torch.rand(896, generator=gen) < 0.5, -1.0, 1.0)
    half = torch.randn(1024, 896, generator=gen)
    state = {k: v * 0.1 if k.endswith("weight_scale") else v for k, v in state.items()}
    state["model.embed_tokens.weight"] = torch.stack([half, half * signs], dim=1).view(2048, 896).half()
    state["model.norm.weight"] = (signs * 0.5).half()
    return qmodel.from_state_dict(state, config)


# prompt lengths, and rows of a prefill: the rows chain; the W4A16 GEMM; SM pairs and the tcgen05 attention
@pytest.mark.parametrize("shortest,longest,low,high", [(8, 17, 64, 128), (16, 80, 129, 767), (64, 1000, 768, 1 << 20)])
def test_steps_of_many_rows_beside_prefills_of_every_form(net, shortest, longest, low, high):
    """64 slots, 160 requests whose ends are spread over the steps: decode steps of 17..64 rows on a stream of high priority beside
    prefills on another.  Two runs on one engine give the same tokens, a run on another engine leaves the same bits in the
    cache, and with the prefills in line the tokens are the same too."""
    gen = torch.Generator().manual_seed(longest)
    lens = [shortest + int((longest - shortest) * ((i * 0.618034) % 1.0)) for i in range(160)]
    limits = [24 + (i * 37) % 72 for i in range(160)]
    prompts = [torch.randint(0, 2048, (n,), generator=gen).tolist() for n in lens]
    beside = []

    def engine(overlap):
        e = Engine(config=EngineConfig(batching="continuous", max_context=1280, decode_burst=8, overlap_prefill=overlap),
                   max_batch_size=64, model_module=SimpleNamespace(load=lambda **options: (net, None)))
        begin = e._prefill_begin

        def watched(sequences, stream=None):
            if stream is not None and sum(not s.is_finished for s in e.running) > 16:
                beside.append(sum(s.prompt_tokens.numel() for s in sequences))
            return begin(sequences, stream)

        e._prefill_begin = watched
        return e

    def serve(e):
        for p, lim in zip(prompts, limits):
            e.add_request_ids(p, max_tokens=lim)
        return e.run()

    first, other = engine(True), engine(True)
    tokens = serve(first)
    torch.cuda.synchronize()
    kv = first.cache.kv.clone()
    assert [len(o) for o in tokens] == limits
    assert sum(low <= n <= high for n in beside) >= 5, beside
    assert serve(first) == tokens
    assert serve(other) == tokens
    assert torch.equal(other.cache.kv, kv)
    assert serve(engine(False)) == tokens
    assert K.lib().quic_w4a16_tensor_status() == 0
