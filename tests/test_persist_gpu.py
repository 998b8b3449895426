"""The persistent decode kernel (one launch per burst of tokens, 1..4 rows here) against the CPU
oracle and against the kernel chain it replaces, through the C ABI."""

import pytest
import torch

pytestmark = pytest.mark.gpu
RTOL, ATOL = 2e-2, 5e-2


def _close(a, b):
    a, b = a.float().cpu(), b.float().cpu()
    return bool(((a - b).abs() <= ATOL + RTOL * b.abs()).all()), (a - b).abs().max().item()


def _greedy_agrees(got, ref_tokens, ref_logits, near_tie=2e-2):
    """Index of the first position where the sequences part (only allowed at a near-tie of the
    oracle's top two logits), or len(ref_tokens)."""
    for i, (g, r) in enumerate(zip(got, ref_tokens)):
        if g == r:
            continue
        top = torch.topk(ref_logits[i].float(), 2)
        gap = (top.values[0] - top.values[1]).item()
        assert gap < near_tie and g in top.indices.tolist(), (i, g, r, gap)
        return i
    return len(ref_tokens)


@pytest.fixture()
def persist_net(tiny_model):
    net = tiny_model[0]
    old = net.use_persist
    net.use_persist = True
    yield net
    net.use_persist = old


def test_single_row_logits_and_tokens_match_oracle(persist_net, tiny_model):
    """Prompt and generation token by token through forward(): every step is one launch of the
    persistent kernel with logits kept (positions 0..n, so the first launch sees an empty slot)."""
    net, ref = persist_net, tiny_model[1]
    prompt = [11, 7, 1999, 42, 0, 512, 77, 1023]
    ref_tokens, ref_logits = ref.greedy(prompt, 6)
    cache = net.new_cache(n_slots=4, s_max=256)
    cache.batch_slots = [2]
    assert net.persist_ok(1, 256)
    logits = None
    for t in prompt:
        logits = net(torch.tensor([[t]]), past_key_values=cache).logits
    got_tokens, got_logits = [], []
    for _ in range(6):
        got_logits.append(logits[0, 0].clone())
        nxt = logits[:, -1:, :].argmax(dim=-1)
        got_tokens.append(int(nxt))
        logits = net(nxt, past_key_values=cache).logits
    assert net.persist_status(cache) == 0
    n = _greedy_agrees(got_tokens, ref_tokens, ref_logits)
    ok, err = _close(torch.stack(got_logits)[: n + 1], ref_logits[: n + 1])
    assert ok, err


@pytest.mark.parametrize("rows", [1, 2, 3, 4])
def test_bursts_match_the_kernel_chain_and_the_oracle(persist_net, tiny_model, rows):
    """Ragged rows, a 40-token burst in one launch: the persistent kernel must give the oracle's
    tokens (up to a near-tie) and the logits of the kernel chain on the same fed tokens."""
    net, ref = persist_net, tiny_model[1]
    gen = torch.Generator().manual_seed(100 + rows)
    lens = [70, 9, 300, 33][:rows]
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    slots = [5, 0, 3, 6][:rows]
    steps = 40

    cache = net.new_cache(n_slots=8, s_max=512)
    first, _ = net.prefill(cache, slots, prompts)
    burst = net.decode(cache, slots, steps)
    assert net.persist_status(cache) == 0
    for i in range(rows):
        want_tokens, want_logits = ref.greedy(prompts[i].tolist(), 12)
        _greedy_agrees([int(first[i])] + burst[i][:11], want_tokens, want_logits)

    # the same burst as single steps gives the same tokens bit for bit
    cache1 = net.new_cache(n_slots=8, s_max=512)
    net.prefill(cache1, slots, prompts)
    singles = [[] for _ in range(rows)]
    for _ in range(steps):
        out = net.decode(cache1, slots, 1)
        for i in range(rows):
            singles[i] += out[i]
    assert singles == burst

    # logits of one more step, persistent kernel vs kernel chain, same cache contents
    cache.batch_slots = slots
    cache1.batch_slots = slots
    nxt = torch.tensor([[b[-1]] for b in burst])
    a = net(nxt, past_key_values=cache).logits[:, 0].clone()
    net.use_persist = False
    try:
        b = net(nxt, past_key_values=cache1).logits[:, 0].clone()
    finally:
        net.use_persist = True
    ok, err = _close(a, b)
    assert ok, err
    assert a.argmax(-1).tolist() == b.argmax(-1).tolist() or err < 2e-2


@pytest.mark.parametrize("prompt_len", [383, 384, 766, 1100, 2110, 2814, 3900])
def test_split_boundaries_and_long_contexts(persist_net, tiny_model, prompt_len):
    """One split (383, 384: the token closes or opens a half tile), the change from one split to two
    within the five steps (766: the bound goes from 768 to 896), two splits of 576 tokens (1100) and, at the bound
    of 4096, six of 704: the tokens being decoded cross from the third into the fourth (2110) and from
    the fourth into the fifth (2814), or end in the sixth (3900).  Merged by the o_proj CTAs; logits against the
    oracle's teacher-forced pass."""
    from quic_cu_b200 import kernels as K

    assert [K.lib().quic_persist_pick_splits(1, n) for n in (768, 896, 1152, 4096)] == [1, 2, 2, 6]
    from oracle.quic_ref import RefModel

    net = persist_net
    ref = RefModel(tiny_model[2], 2, max_pos=4096)
    prompt = torch.randint(0, 2048, (prompt_len,), generator=torch.Generator().manual_seed(prompt_len))
    steps = 5
    cache = net.new_cache(n_slots=2, s_max=4096)
    assert net.persist_ok(1, min(4096, prompt_len + 128))
    first, _ = net.prefill(cache, [1], [prompt])
    cache.batch_slots = [1]
    fed, kept = [int(first[0])], []
    for _ in range(steps):
        logits = net(torch.tensor([[fed[-1]]]), past_key_values=cache).logits[0, 0].clone()
        kept.append(logits)
        fed.append(int(logits.argmax()))
    assert net.persist_status(cache) == 0
    want = ref.teacher_forced(prompt.tolist(), fed)[1:]  # logits after feeding fed[0..steps-1]
    ok, err = _close(torch.stack(kept), want[:steps])
    assert ok, err


def test_host_fed_single_steps_agree_with_a_burst(persist_net):
    """The host-driven form (token in from pinned memory, id and status word out, stream
    synchronised) must reproduce the tokens of one 24-step launch."""
    net = persist_net
    prompt = torch.tensor([17, 4, 256, 1000, 31, 8, 8, 1203, 77])
    cache = net.new_cache(n_slots=2, s_max=256)
    first, _ = net.prefill(cache, [1], [prompt])
    burst = [int(first[0])] + net.decode(cache, [1], 24)[0]
    cache = net.new_cache(n_slots=2, s_max=256)
    first, _ = net.prefill(cache, [1], [prompt])
    pinned = torch.zeros(1, dtype=torch.int32).pin_memory()
    fed = [int(first[0])]
    for _ in range(24):
        pinned[0] = fed[-1]
        fed.append(net.decode(cache, [1], 1, feed=pinned)[0][0])
    assert fed == burst


def test_a_feed_is_checked_at_every_call(persist_net):
    """The same tensor object may have another size or layout at the next call, or other slots."""
    net = persist_net
    cache = net.new_cache(n_slots=2, s_max=256)
    net.prefill(cache, [0, 1], [torch.tensor([5, 6, 7]), torch.tensor([8, 9])])
    feed = torch.tensor([3, 4], dtype=torch.int32).pin_memory()
    net.decode(cache, [0, 1], 1, feed=feed)
    for spoil in (lambda: feed.resize_(1), lambda: feed.set_(torch.zeros(4, dtype=torch.int32)[::2]),
                  lambda: feed.resize_(0)):
        spoil()
        with pytest.raises(ValueError, match="feed"):
            net.decode(cache, [0, 1], 1, feed=feed)
    net.decode(cache, [1, 0], 1)
    with pytest.raises(ValueError, match="consecutive"):
        net.decode(cache, [1, 0], 1, feed=torch.tensor([3, 4], dtype=torch.int32).pin_memory())


def test_a_wait_that_runs_out_is_reported_and_the_next_launch_works(persist_net):
    """Bounded waits: with the probe limit lowered to 4096 and CTA 0 withholding its o_proj
    result of layer 0 (both through the header words of the exchange area), the polls that
    need that result give up, the kernel returns, the status word names the wait, nothing
    was generated; after clearing the hook the same area serves a normal launch whose
    tokens match an undisturbed run."""
    net = persist_net
    prompt = torch.tensor([5, 900, 13, 2000, 7])
    want_cache = net.new_cache(n_slots=2, s_max=256)
    first, _ = net.prefill(want_cache, [0], [prompt])
    want = net.decode(want_cache, [0], 6)[0]

    cache = net.new_cache(n_slots=2, s_max=256)
    net.prefill(cache, [0], [prompt])
    hdr = cache.persist_sync()[:16].view(torch.int32)
    hdr[2] = 4096
    hdr[3] = 1
    pos_before = int(cache.pos[0])
    with pytest.raises(RuntimeError, match="bounded wait"):
        net.decode(cache, [0], 1)
    torch.cuda.synchronize()
    assert int(cache.pos[0]) == pos_before      # no token was produced
    assert int(hdr[1]) == 0                     # the failing call cleared the word
    hdr[2] = 0
    hdr[3] = 0
    cache.host_steps -= 1                       # undo the host mirrors of the abandoned step
    cache.host_len[0] -= 1
    assert net.decode(cache, [0], 6)[0] == want
    assert net.persist_status(cache) == 0

    # the asynchronous form leaves the code in the status word: 0x100 | (layer * 8 + phase)
    hdr[2] = 4096
    hdr[3] = 2
    net.decode_async(cache, [0], 1)
    assert net.persist_status(cache) == (0x100 | (1 * 8 + 3))
    hdr[2] = 0
    hdr[3] = 0
    cache.host_steps -= 1
    cache.host_len[0] -= 1
    more = net.decode(cache, [0], 3)[0]
    assert more == net.decode(want_cache, [0], 3)[0]


@pytest.mark.parametrize("rows", [1, 3])
def test_layer_numbers_may_run_over(persist_net, rows):
    """Header word 0 counts layers over the life of an exchange area.  A burst that starts a few layers below the
    end of 32 bits, or of the range the numbers are kept in, gives the tokens of one that starts at zero, and so
    does a start number that was used before: the candidates of the burst that had it are still in the area."""
    net = persist_net
    gen = torch.Generator().manual_seed(rows)
    prompts = [torch.randint(0, 2048, (20 + 9 * i,), generator=gen) for i in range(rows)]
    others = [torch.randint(0, 2048, (31,), generator=gen) for _ in range(rows)]
    slots = list(range(rows))

    def burst(cache, tokens, number=None):
        net.prefill(cache, slots, tokens)
        if number is not None:
            cache.persist_sync()[:4].view(torch.int32)[0] = number - (1 << 32) if number >= 1 << 31 else number
        got = net.decode(cache, slots, 16)
        logits = torch.empty(rows, 2048, dtype=torch.float16, device="cuda")
        net.decode_async(cache, slots, 1, logits=logits)
        assert net.persist_status(cache) == 0
        return got, logits

    fresh = [burst(net.new_cache(n_slots=4, s_max=256), p) for p in (prompts, others)]
    cache = net.new_cache(n_slots=4, s_max=256)
    for number in (0, (1 << 32) - 13, (1 << 32) - 1, (3 << 28) - 13, (3 << 28) - 1, 0):
        for want, p in zip(fresh, (prompts, others)):
            got = burst(cache, p, number)
            assert got[0] == want[0] and torch.equal(got[1], want[1]), number


@pytest.mark.parametrize("lens,hint", [([1500], 900), ([1700, 40], 800), ([300, 1900, 5], 1000), ([2000] * 4, 1500), ([1100], 1)])
def test_a_context_hint_below_the_position_loses_no_token(persist_net, lens, hint):
    """The last of several attention splits takes whatever the hint left out: logits and the appended keys and
    values of a step whose hint is too small against the kernel chain with the right one."""
    import ctypes as C

    from quic_cu_b200 import kernels as K

    net, rows = persist_net, len(lens)
    gen = torch.Generator().manual_seed(sum(lens))
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    cache = net.new_cache(n_slots=4, s_max=2048)
    slots = list(range(rows))
    net.prefill(cache, slots, prompts)
    start = [t.clone() for t in (cache.kv, cache.tok, cache.pos)]
    logits = [torch.empty(rows, 2048, dtype=torch.float16, device="cuda") for _ in range(2)]

    d, row_map = net._decode_struct(cache, rows, hint, logits[0], persist=True)
    row_map.copy_(cache.rows_tensor(slots))
    K.check(K.lib().quic_decode_persist(C.byref(net._c_model), C.byref(d), K.ptr(net.persist_stream()),
                                        K.ptr(cache.persist_sync()), 1, K.stream_ptr()), "decode_persist")
    assert net.persist_status(cache) == 0
    kv = cache.kv.clone()
    for t, s in zip((cache.kv, cache.tok, cache.pos), start):
        t.copy_(s)
    net.use_persist = False
    net.decode_async(cache, slots, 1, logits=logits[1])
    ok, err = _close(logits[0], logits[1])
    assert ok, err
    assert (kv.float() - cache.kv.float()).abs().max() <= 5e-2


def test_the_weight_stream_is_complete_when_it_is_handed_out(persist_net):
    """It is packed on the stream of the first caller, behind whatever that stream still has to do; callers on other
    streams and of other threads read the same copy."""
    import threading

    net = persist_net
    want = net.persist_stream()
    kept, net._wstream = want.clone(), None
    torch.cuda.synchronize()
    got = []

    def first_use():
        with torch.cuda.stream(torch.cuda.Stream()):
            torch.cuda._sleep(20_000_000)
            t = net.persist_stream()
            got.append((t.data_ptr(), torch.cuda.current_stream().query()))

    threads = [threading.Thread(target=first_use) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    # the last caller's own sleep may still run, the packing may not
    assert len({p for p, _ in got}) == 1 and any(done for _, done in got)
    assert torch.equal(net.persist_stream(), kept)


@pytest.mark.parametrize("bits", [0x7E00, 0xFFFF], ids=hex)
def test_a_row_of_nan_ends_like_the_chain_and_leaves_the_others_alone(persist_net, bits):
    """A row whose input is NaN has no logit to choose from: token 0 in either form; no wait runs out over it
    (0xFFFF pairs are what an empty exchange word decodes to), and the row beside it is untouched."""
    net = persist_net
    gen = torch.Generator().manual_seed(5)
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in (12, 40)]
    kept, got = net.embed[77].clone(), []
    try:
        for persist in (True, False):
            net.use_persist = persist
            cache = net.new_cache(n_slots=2, s_max=128)
            net.prefill(cache, [0, 1], prompts)
            cache.tok[0] = 77
            net.embed[77].view(torch.int16).fill_(bits - 0x10000 if bits >= 0x8000 else bits)
            got.append(net.decode(cache, [0, 1], 1))
            net.embed[77] = kept
            assert not persist or net.persist_status(cache) == 0
    finally:
        net.embed[77] = kept
    assert got[0] == got[1] and got[0][0] == [0]
