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


def test_prefills_on_sm_pairs_beside_decode_steps_keep_their_bits(net):
    """Prefills of 770..1250 rows, eight launches on CTA pairs each, on one stream beside bursts of 62 rows on another of high
    priority: one-CTA and two-CTA allocations of tensor memory take turns on every SM.  Every prefill leaves the bits that it
    leaves alone."""
    gen = torch.Generator().manual_seed(11)
    lens = [(406, 773), (770,), (500, 300, 450), (1200,), (900, 33)]
    prompts = [[torch.randint(0, 2048, (n,), generator=gen) for n in group] for group in lens]
    rows = list(range(62))
    cache = net.new_cache(n_slots=65, s_max=1280)
    net.prefill(cache, rows, [torch.randint(0, 2048, (20 + i,), generator=gen) for i in rows])
    want = []
    for group in prompts:
        first, logits = net.prefill(cache, [62, 63, 64][:len(group)], group)
        want.append((first.clone(), logits.clone()))
    tok, pos, length = cache.tok.clone(), cache.pos.clone(), list(cache.host_len)
    alone = net.decode(cache, rows, 16)
    main, side = torch.cuda.Stream(priority=-1), torch.cuda.Stream()
    torch.cuda.synchronize()
    for i in range(150):
        with torch.cuda.stream(main):
            cache.tok[:62].copy_(tok[:62])
            cache.pos[:62].copy_(pos[:62])
        cache.host_len[:62] = length[:62]
        got = []
        with torch.cuda.stream(side):
            for group in prompts:
                got.append(net.prefill(cache, [62, 63, 64][:len(group)], group))
        with torch.cuda.stream(main):
            assert net.decode(cache, rows, 16) == alone
        side.synchronize()
        cache.raise_errors()
        for (first, logits), (first_alone, logits_alone) in zip(got, want):
            assert torch.equal(first, first_alone) and torch.equal(logits, logits_alone)
