"""The persistent decode kernel over its row counts, weight types and context edges: logits against
the kernel chain on the same cache, and the same bits on every run."""

import pytest
import torch

pytestmark = pytest.mark.gpu
RTOL, ATOL = 2e-2, 5e-2


@pytest.fixture(scope="module")
def dense_model():
    from quic_cu_b200 import model as qmodel
    from quic_cu_b200.checkpoint import qwen_config_dict, synthetic_dense_checkpoint

    config = qwen_config_dict(2, 2048)
    config.pop("quantization_config")
    return qmodel.from_state_dict(synthetic_dense_checkpoint(n_layers=2, vocab=2048, seed=4), config)


@pytest.mark.parametrize("persist", [True, False])
@pytest.mark.parametrize("rows", [1, 4])
def test_two_models_on_one_cache(tiny_model, dense_model, persist, rows):
    """Launch plans and graphs that a cache keeps are those of the model that made them, and of its choice of kernel."""
    nets = (tiny_model[0], dense_model)
    old = [net.use_persist for net in nets]
    gen = torch.Generator().manual_seed(rows)
    prompts = [torch.randint(0, 2048, (20 + i,), generator=gen) for i in range(rows)]
    slots = list(range(rows))

    def answer(net, cache):
        net.prefill(cache, slots, prompts)
        return net.decode(cache, slots, 8)

    try:
        for net in nets:
            net.use_persist = persist
        want = [answer(net, net.new_cache(n_slots=4, s_max=128)) for net in nets]
        cache = nets[0].new_cache(n_slots=4, s_max=128)
        for _ in range(2):
            assert [answer(net, cache) for net in nets] == want
        kinds = {type(p.handle) for p in cache._plans.values()}
        for net in nets:
            net.use_persist = not persist
            answer(net, cache)
        assert len({type(p.handle) for p in cache._plans.values()}) == 2 and len(kinds) == 1
    finally:
        for net, flag in zip(nets, old):
            net.use_persist = flag


# tokens cached before the step: the step's own token opens or closes a 32-token half tile (31, 32, 63),
# falls to the first warp's second half tile (448), lies beyond what stays in shared memory (1000 at 16
# rows, one split) or in a later split (800 at one row, 1700 at two)
@pytest.mark.parametrize("lens", [
    [1], [31], [447], [448], [800], [32, 1700], [63, 5, 900], [5, 64, 300, 31], [700, 90, 33, 1, 480],
    [96] * 8, [20, 300, 7, 64, 65, 511, 512, 1, 30], [17 * (i + 1) for i in range(12)], [1000] + [40] * 15,
], ids=lambda v: f"{len(v)}x{max(v)}")
@pytest.mark.parametrize("dense", [False, True], ids=["w4", "fp16"])
def test_logits_match_the_kernel_chain_and_repeat(tiny_model, dense_model, dense, lens):
    net = dense_model if dense else tiny_model[0]
    rows, old = len(lens), net.use_persist
    gen = torch.Generator().manual_seed(sum(lens))
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    cache = net.new_cache(n_slots=16, s_max=2048)
    slots = torch.randperm(16, generator=gen)[:rows].tolist()
    net.prefill(cache, slots, prompts)
    state = [t.clone() for t in (cache.kv, cache.tok, cache.pos)]
    host_len = list(cache.host_len)

    def step(persist, steps):
        for t, s in zip((cache.kv, cache.tok, cache.pos), state):
            t.copy_(s)
        cache.host_len[:] = host_len
        net.use_persist = persist
        try:
            burst = net.decode(cache, slots, steps) if steps else None
            logits = torch.empty(rows, 2048, dtype=torch.float16, device="cuda")
            net.decode_async(cache, slots, 1, logits=logits)
            if persist:
                assert net.persist_status(cache) == 0
        finally:
            net.use_persist = old
        return logits, burst, cache.kv.clone()

    got, want = step(True, 0), step(False, 0)
    a, b = got[0].float(), want[0].float()
    assert ((a - b).abs() <= ATOL + RTOL * b.abs()).all(), (a - b).abs().max().item()
    assert (got[2].float() - want[2].float()).abs().max() <= 5e-2
    first = step(True, 3)
    for _ in range(4):
        again = step(True, 3)
        assert again[1] == first[1] and torch.equal(again[0], first[0]) and torch.equal(again[2], first[2])
