"""The decode step of 16..128 rows (un-quantised from 3): one launch per linear with norm, RoPE + KV
append, residual or SwiGLU inside, `down` over clusters of eight CTAs; and the step of more rows, a GEMM per linear."""

import pytest
import torch
from torch.linalg import vector_norm as norm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nets(tiny_model):
    from quic_cu_b200 import model as qmodel
    from quic_cu_b200.checkpoint import qwen_config_dict, synthetic_dense_checkpoint

    config = qwen_config_dict(2, 2048)
    config.pop("quantization_config", None)
    # packed weights of the spread of the un-quantised ones: with the checkpoint's own, gates of 30 and more turn a
    # rounding of theirs into thirty
    _, _, state, packed_config = tiny_model
    state = {k: v * 0.25 if k.endswith("weight_scale") else v for k, v in state.items()}
    return {"w4": qmodel.from_state_dict(state, packed_config),
            "fp16": qmodel.from_state_dict(synthetic_dense_checkpoint(n_layers=2, vocab=2048, seed=99), config)}


@pytest.mark.parametrize("weights,rows", [("w4", n) for n in (16, 17, 63, 64, 65, 127, 128, 129, 201)] +
                         [("fp16", n) for n in (3, 16, 64, 65, 128, 129, 201)])
def test_appended_keys_and_values_match_a_prefill_of_the_same_tokens(nets, monkeypatch, weights, rows):
    """Edges of the row tiles (64, 128) and of what the path takes (beyond: GEMMs, the attention finishes the QKV linear).  A step appends K and V of the token it feeds
    in every layer; a prefill of prompt + token, other kernels, has to leave the same there.  On the way to K and V of
    the second layer lie 17 roundings to fp16 (two norms and the third, four linears with their sums, bias, rotation,
    probabilities, activation), each 2^-11 / sqrt(3) in the root mean square, on either side; the worst of up to
    512 (row, plane) pairs is allowed twice their root of 34."""
    from quic_cu_b200 import kernels as K

    net = nets[weights]
    monkeypatch.setattr(net, "use_persist", False)
    gen = torch.Generator().manual_seed(rows)
    lens = torch.randint(8, 90, (rows,), generator=gen).tolist()
    lens[0] = 300  # (more rows in the prefills than any of the forms under test takes)
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    slots = torch.randperm(rows + 2, generator=gen)[:rows].tolist()  # rows need not sit in slot order, nor fill the cache
    cache, other = (net.new_cache(n_slots=rows + 2, s_max=320) for _ in range(2))
    first, _ = net.prefill(cache, slots, prompts)
    per_layer = 5 if rows <= 128 else 7 if weights == "w4" else 8
    assert net.launches_per_step(cache, rows, 320) == per_layer * net.n_layers + 3
    idle = [s for s in range(rows + 2) if s not in slots]
    before = cache.kv[:, :, idle].clone()
    net.decode(cache, slots, 1)
    net.prefill(other, slots, [torch.cat([p, first[i:i + 1].cpu()]) for i, p in enumerate(prompts)])
    at = torch.tensor(lens, device="cuda")
    got, want = (c.kv[:, :, slots].float().gather(4, at.view(1, 1, rows, 1, 1, 1).expand(2, 2, rows, 2, 1, 64)) for c in (cache, other))
    worst = (norm(got - want, dim=(3, 4, 5)) / norm(want, dim=(3, 4, 5))).max().item()
    assert worst < 2 * (34 / 3) ** 0.5 * 2 ** -11, worst
    assert torch.equal(cache.kv[:, :, idle], before)
    assert K.lib().quic_w4a16_tensor_status() == 0


def test_rows_of_very_small_and_large_norm(nets):
    """The rows' factors are a power of two, applied before the product, and a rest of 1 to 2, after it: rows far from 1 in
    size must come out as a norm in 32 bits gives them, that of the per-operator prefill.  In the decode step and in a
    short prefill."""
    net = nets["w4"]
    embed = net.embed.clone()
    try:
        scale = torch.tensor([2.0 ** -14, 2.0 ** -7, 1.0, 37.0, 1500.0], device="cuda", dtype=torch.float32)
        net.embed[:40] = (embed[:40].float().sign() * scale.repeat(8).view(40, 1) *
                          (0.5 + torch.rand(40, 896, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3)))).half()
        ids, slots = torch.arange(40).view(40, 1), list(range(40))
        step, short, other = (net.new_cache(n_slots=40, s_max=64) for _ in range(3))
        for c in (step, short, other):
            net.prefill(c, slots, [torch.tensor([5])] * 40)
        step.tok.copy_(ids.view(-1))
        net.decode(step, slots, 1)
        net.prefill(short, slots, list(ids), offsets=[1] * 40)
        net.prefill(other, slots, list(ids), offsets=[1] * 40, all_logits=True)
        want = other.kv[0, :, :, :, 1].float()
        for c in (step, short):
            got = c.kv[0, :, :, :, 1].float()
            worst = (norm(got - want, dim=(2, 3)) / norm(want, dim=(2, 3))).max().item()
            assert worst < 2 * 3 ** 0.5 * 2 ** -12, worst  # three roundings on either side
    finally:
        net.embed.copy_(embed)


def test_a_row_with_an_infinity(nets):
    """Its keys and values are NaN, as the per-operator prefill leaves them; the other rows keep their bits."""
    net, prompts, slots = nets["w4"], [torch.tensor([i]) for i in range(20)], list(range(20))
    clean, spoilt, other = (net.new_cache(n_slots=20, s_max=64) for _ in range(3))
    net.prefill(clean, slots, prompts)
    before = net.embed[7, 100].clone()
    try:
        net.embed[7, 100] = float("inf")
        net.prefill(spoilt, slots, prompts)
        net.prefill(other, slots, prompts, all_logits=True)
    finally:
        net.embed[7, 100] = before
    for c in (spoilt, other):
        assert torch.isnan(c.kv[:, :, 7, :, 0]).all()
    others = [i for i in slots if i != 7]
    assert torch.equal(spoilt.kv[:, :, others], clean.kv[:, :, others])


@pytest.mark.parametrize("weights", ["w4", "fp16"])
def test_a_row_of_zeros_under_a_small_eps(nets, weights):
    """eps 1e-12: 1 / rms of a row of zeros is 1e6, and of a row of fp16's smallest values 7.8e5, more than fp16 holds.  The
    chain of a short prefill against the per-operator one, whose factor is in 32 bits."""
    net = nets[weights]
    embed, eps = net.embed.clone(), net.eps
    try:
        net.eps = net._c_model.eps = 1e-12
        net.embed[0], net.embed[1] = 0, 2.0 ** -24
        cache, other = (net.new_cache(n_slots=20, s_max=64) for _ in range(2))
        prompts = [torch.tensor([i]) for i in range(20)]
        net.prefill(cache, list(range(20)), prompts)
        net.prefill(other, list(range(20)), prompts, all_logits=True)
        got, want = cache.kv[0, :, :, :, 0].float(), other.kv[0, :, :, :, 0].float()
        assert torch.isfinite(want).all()
        worst = (norm(got - want, dim=(2, 3)) / norm(want, dim=(2, 3))).max().item()
        assert worst < 2 * 3 ** 0.5 * 2 ** -12, worst  # three roundings on either side
    finally:
        net.embed.copy_(embed)
        net.eps = net._c_model.eps = eps


@pytest.mark.parametrize("weights,lens", [("w4", [2]), ("w4", [64]), ("w4", [40, 25]), ("w4", [128]), ("w4", [1] * 20), ("fp16", [3]),
                                          ("fp16", [65]), ("fp16", [129]), ("fp16", [200, 120])])
def test_a_short_prefill_matches_the_operators_one_by_one(nets, weights, lens):
    """Edges of the row tiles and of what the chain takes of prompts (128 rows, un-quantised 320): keys, values and the last
    rows' logits against the per-operator prefill.  Roundings as above, three more for a logit."""
    net = nets[weights]
    gen = torch.Generator().manual_seed(sum(lens))
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    slots = torch.randperm(len(lens) + 1, generator=gen)[:len(lens)].tolist()
    cache, other = (net.new_cache(n_slots=len(lens) + 1, s_max=256) for _ in range(2))
    first, logits = net.prefill(cache, slots, prompts)
    _, want = net.prefill(other, slots, prompts, all_logits=True)
    last = torch.tensor(lens).cumsum(0) - 1
    worst = (norm(logits.float() - want.view(-1, 2048)[last].float(), dim=1) / norm(want.view(-1, 2048)[last].float(), dim=1)).max().item()
    assert worst < 2 * (40 / 3) ** 0.5 * 2 ** -11, worst
    for slot, n in zip(slots, lens):
        got, ref = cache.kv[:, :, slot, :, :n].float(), other.kv[:, :, slot, :, :n].float()
        worst = (norm(got - ref, dim=(2, 4)) / norm(ref, dim=(2, 4))).max().item()
        assert worst < 2 * (34 / 3) ** 0.5 * 2 ** -11, worst
    assert cache.pos[slots].tolist() == lens and cache.tok[slots].tolist() == first.tolist()


def test_the_limit_of_a_wait_is_not_for_the_kernel_in_front(nets):
    """The attention of 64 rows of 32000 tokens (1 GB a layer; no memory is faster than 8 TB/s, so 130 us and more) stands
    before o_proj, whose CTAs are there from its start.  A limit of 60 us, enough for any wait of theirs once the attention has
    ended, must not run out over it."""
    from quic_cu_b200 import kernels as K

    net, lib, rows, length = nets["w4"], K.lib(), 64, 32000
    cache = net.new_cache(n_slots=rows, s_max=32064)
    cache.kv.normal_(generator=torch.Generator(device="cuda").manual_seed(1))
    tokens = torch.arange(rows, dtype=torch.int32, device="cuda")

    def step():
        cache.release_graphs()  # a graph holds the limit that it was captured with
        cache.tok.copy_(tokens)
        cache.pos.fill_(length)
        cache.host_len[:] = [length] * rows
        return net.decode(cache, list(range(rows)), 1)

    want = step()
    lib.quic_w4a16_tensor_test_hook(60, -1)
    try:
        assert step() == want
    finally:
        lib.quic_w4a16_tensor_test_hook(0, -1)
    assert lib.quic_w4a16_tensor_status() == 0


@pytest.mark.parametrize("weights,rows", [("w4", 20), ("w4", 100), ("fp16", 20), ("fp16", 100)])
def test_stages_that_come_late_and_too_late(nets, weights, rows):
    """Every stage of the rows 2 ms late, with a limit of 3 ms a wait: the whole accumulation takes 14 ms, and nobody who waits
    for all of it may give up before the issuer of the MMAs does.  With a limit of 1 ms the issuer gives up: decode() raises, the
    CTAs leave in order, and the next decode() is right."""
    from quic_cu_b200 import kernels as K

    net, lib = nets[weights], K.lib()
    gen = torch.Generator().manual_seed(rows)
    prompts = [torch.randint(0, 2048, (int(n),), generator=gen) for n in torch.randint(4, 30, (rows,), generator=gen)]
    slots = list(range(rows))

    def step(limit, late):
        cache = net.new_cache(n_slots=rows, s_max=64)
        net.prefill(cache, slots, prompts)
        torch.cuda.synchronize()
        lib.quic_w4a16_tensor_test_hook(limit, late)
        try:
            return net.decode(cache, slots, 1), cache.kv
        finally:
            lib.quic_w4a16_tensor_test_hook(0, -1)

    tokens, kv = step(0, -1)
    late = step(3000, -2000)
    assert late[0] == tokens and torch.equal(late[1], kv)
    with pytest.raises(RuntimeError, match="bounded wait"):
        step(1000, -2000)
    again = step(0, -1)
    assert again[0] == tokens and torch.equal(again[1], kv)
    assert lib.quic_w4a16_tensor_status() == 0


@pytest.mark.parametrize("weights,length", [("w4", 300), ("fp16", 400)])
def test_chunks_on_the_chain_agree_with_a_whole_prompt_on_the_gemms(nets, weights, length):
    """Chunks of 100 tokens run the chain, the whole prompt the GEMMs: other sums, so not the same bits, but the same up to the
    roundings (as above)."""
    net = nets[weights]
    prompt = torch.randint(0, 2048, (length,), generator=torch.Generator().manual_seed(length))
    whole, cache = (net.new_cache(n_slots=1, s_max=448) for _ in range(2))
    _, want = net.prefill(whole, [0], [prompt])
    for at in range(0, length, 100):
        _, got = net.prefill(cache, [0], [prompt[at:at + 100]], offsets=[at])
    assert (norm(got.float() - want.float()) / norm(want.float())).item() < 2 * (40 / 3) ** 0.5 * 2 ** -11
    a, b = cache.kv[:, :, 0, :, :length].float(), whole.kv[:, :, 0, :, :length].float()
    worst = (norm(a - b, dim=(2, 4)) / norm(b, dim=(2, 4))).max().item()
    assert worst < 2 * (34 / 3) ** 0.5 * 2 ** -11, worst
