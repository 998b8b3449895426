"""The bounded waits of the tcgen05 kernels, one operator at a time: operands that come late but within the limit change
nothing, operands that come too late or never set the error word, the CTAs leave in order (MMAs and copies complete,
tensor memory free), and the next call is right."""

import pytest
import torch

from quic_cu_b200 import kernels as K

pytestmark = pytest.mark.gpu


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _linear(weight, m):
    x = torch.randn(m, weight.size_k, device="cuda", generator=_gen(m)).half()
    return lambda: K.w4a16_linear(weight, x)


def _packed(n, k):
    w = K.W4Weight(n, k, torch.device("cuda"))
    w.qw.random_(-2 ** 31, 2 ** 31 - 1, generator=_gen(1))
    w.zp.random_(0, 255, generator=_gen(2))
    w.sc.copy_(torch.rand(w.sc.shape, device="cuda", generator=_gen(3)) * 0.02)
    return w


def _dense(n, k):
    w = K.F16Weight(n, k, torch.device("cuda"))
    w.w.copy_(torch.randn(n, k, device="cuda", generator=_gen(4)) * 0.05)
    return w


def _lm_head(rows):
    x = torch.randn(rows, K.HIDDEN, device="cuda", generator=_gen(5)).half()
    table = torch.randn(2048, K.HIDDEN, device="cuda", generator=_gen(6)).half()
    return lambda: K.lm_head_argmax(x, table, want_logits=True)[1]


def _attention(n_seq):
    """130 rows a sequence behind 70 cached tokens; 45 sequences are more CTAs than the form with scores a tile ahead takes."""
    rows, s_max = 130 * n_seq, 256
    q = torch.randn(14, rows, 64, device="cuda", generator=_gen(7)).half()
    k, v = (torch.randn(n_seq, 2, s_max, 64, device="cuda", generator=_gen(s)).half() for s in (8, 9))
    table = torch.tensor([[130 * i for i in range(n_seq)], [130] * n_seq, list(range(n_seq)), [70] * n_seq], dtype=torch.int32,
                         device="cuda")
    return lambda: K.attn_prefill(q, k, v, table[0], table[1], table[2], 130, seq_off=table[3])


CALLS = {
    "w4a16, one wave": lambda: _linear(_packed(1152, 896), 64),
    "w4a16, split K": lambda: _linear(_packed(896, 4864), 100),
    "w4a16, two row tiles": lambda: _linear(_packed(9728, 896), 500),
    "fp16": lambda: _linear(_dense(1152, 896), 64),
    "fp16, split K": lambda: _linear(_dense(896, 4864), 20),
    "pair": lambda: _linear(_dense(1152, 896), 700),
    "pair, more tiles than pairs": lambda: _linear(_dense(9728, 896), 700),
    "lm_head, 3 rows": lambda: _lm_head(3),
    "lm_head, 128 rows": lambda: _lm_head(128),
    "attention, ahead": lambda: _attention(1),
    "attention": lambda: _attention(45),
}


# (limit, late): pauses of 0.6 ms a k block against limits of 1.5 and 0.3 ms; a first k block that never comes
@pytest.mark.parametrize("name", list(CALLS))
def test_late_operands(name):
    call, lib = CALLS[name](), K.lib()

    def run(limit, late):
        lib.quic_w4a16_tensor_test_hook(limit, late)
        try:
            y = call().clone()
        finally:
            lib.quic_w4a16_tensor_test_hook(0, -1)
        return y, lib.quic_w4a16_tensor_status()

    want = call().clone()
    assert lib.quic_w4a16_tensor_status() == 0
    late, status = run(1500, -600)
    assert status == 0 and torch.equal(late, want)
    for limit, how in ((300, -600), (1500, 0)):
        assert run(limit, how)[1] != 0
        assert torch.equal(call(), want)
        assert lib.quic_w4a16_tensor_status() == 0


def test_an_early_tile_of_the_streamed_attention_that_never_lands(tiny_model):
    """Tiles requested before the dependency wait that count as too early are requested again once the first copies have
    landed.  Where that of the first tile never does, those of the others are on their way when the wait gives up."""
    net, _, _, _ = tiny_model
    lib, slots = K.lib(), list(range(24))
    prompts = [torch.randint(0, 2048, (70 + 8 * i,), generator=torch.Generator().manual_seed(i)) for i in slots]

    def decode():
        cache = net.new_cache(n_slots=24, s_max=320)
        net.prefill(cache, slots, prompts)
        return net.decode(cache, slots, 2)

    want = decode()
    lib.quic_attn_stream_test_hook(3)
    try:
        with pytest.raises(RuntimeError, match="bounded wait"):
            decode()
    finally:
        lib.quic_attn_stream_test_hook(0)
    assert decode() == want
    assert lib.quic_w4a16_tensor_status() == 0


def _prompts(count, length):
    return [torch.randint(0, 2048, (length,), generator=torch.Generator().manual_seed(i)) for i in range(count)]


class _Hook:
    """Operands that never come, for what is launched or captured meanwhile."""

    def __enter__(self):
        K.lib().quic_w4a16_tensor_test_hook(2000, 0)

    def __exit__(self, *_):
        K.lib().quic_w4a16_tensor_test_hook(0, -1)


@pytest.mark.parametrize("length", [40, 200])
def test_a_prefill_that_gave_up_is_heard_of_by_its_own_cache(tiny_model, length):
    """Both chains of a short prefill.  The error is raised where its results are first waited for: by raise_errors() after a
    synchronisation, by the next decode() or forward() of the same cache; not by a decode() of another."""
    net, slots = tiny_model[0], [0, 1]
    good, bad = (net.new_cache(n_slots=2, s_max=256) for _ in range(2))
    net.prefill(good, slots, _prompts(2, length))
    for hears in ("decode", "forward", "raise_errors"):
        with _Hook():
            net.prefill(bad, slots, _prompts(2, length))
        net.decode(good, slots, 2)
        torch.cuda.synchronize()
        good.raise_errors()
        bad.batch_slots = slots
        with pytest.raises(RuntimeError, match="bounded wait.*in a prefill"):
            net.decode(bad, slots, 2) if hears == "decode" else bad.raise_errors() if hears == "raise_errors" else net(
                torch.zeros(2, 1, dtype=torch.long), past_key_values=bad)
        bad.raise_errors()  # (heard of once)
    first, _ = net.prefill(bad, slots, _prompts(2, length))
    again, _ = net.prefill(good, slots, _prompts(2, length))
    assert torch.equal(first, again) and net.decode(bad, slots, 3) == net.decode(good, slots, 3)
    assert K.lib().quic_w4a16_tensor_status() == 0


def test_a_forward_step_that_gave_up_is_heard_of_by_the_next(tiny_model):
    """forward() does not wait for its step: the next one raises, or raise_errors() after a synchronisation."""
    net, rows = tiny_model[0], 20
    ids = torch.stack(_prompts(rows, 30))
    good, bad = net(ids).past_key_values, net(ids).past_key_values
    token = torch.zeros(rows, 1, dtype=torch.long)
    for hears in ("forward", "raise_errors"):
        bad.release_graphs()
        with _Hook():
            net(token, past_key_values=bad)
        torch.cuda.synchronize()
        net.decode(good, good.batch_slots, 1)
        with pytest.raises(RuntimeError, match="bounded wait.*in a step"):
            net(token, past_key_values=bad) if hears == "forward" else bad.raise_errors()
    assert K.lib().quic_w4a16_tensor_status() == 0


def test_the_engine_hears_of_a_prefill_that_gave_up(tiny_model):
    from types import SimpleNamespace

    from quic_cu_b200.config import EngineConfig
    from quic_cu_b200.engine import Engine

    net = tiny_model[0]
    engine = Engine(config=EngineConfig(batching="continuous", max_context=256, decode_burst=4), max_batch_size=4,
                    model_module=SimpleNamespace(load=lambda **options: (net, None)))
    engine.add_request_ids(_prompts(1, 60)[0], max_tokens=4)
    with _Hook(), pytest.raises(RuntimeError, match="bounded wait.*in a prefill"):
        engine.run()
    assert K.lib().quic_w4a16_tensor_status() == 0
