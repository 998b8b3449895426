"""Stand-alone operators called from several threads on one stream, or captured into graphs: a call that is several
launches keeps its scratch memory to itself."""

from __future__ import annotations

import threading

import pytest
import torch

from quic_cu_b200 import kernels

pytestmark = pytest.mark.gpu


def _linear(seed):
    """A packed linear whose K is split: partial sums and their sum are two launches."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = kernels.W4Weight(896, 4864, torch.device("cuda"))
    w.qw.random_(-2 ** 31, 2 ** 31 - 1, generator=gen)
    w.zp.random_(0, 255, generator=gen)
    w.sc.copy_(torch.rand(w.sc.shape, device="cuda", generator=gen) * 0.02)
    x = torch.randn(100 + seed, 4864, device="cuda", generator=gen).half()
    return lambda: kernels.w4a16_linear(w, x)


def _pair_linear(seed):
    """Rows enough for the pair GEMM, which unpacks the weight into its scratch first."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = kernels.W4Weight(9728, 896, torch.device("cuda"))
    w.qw.random_(-2 ** 31, 2 ** 31 - 1, generator=gen)
    w.zp.random_(0, 255, generator=gen)
    w.sc.copy_(torch.rand(w.sc.shape, device="cuda", generator=gen) * 0.02)
    x = torch.randn(800 + seed, 896, device="cuda", generator=gen).half()
    return lambda: kernels.w4a16_linear(w, x)


def _head(seed):
    """More rows than the candidates of one launch: two launches and a clear between them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(200 + seed, 896, device="cuda", generator=gen).half()
    table = torch.randn(2048, 896, device="cuda", generator=gen).half()
    return lambda: kernels.lm_head_argmax(x, table)[0]


def _split_attention(seed):
    """Split partials merged by the CTA that arrives last at a counter."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(4, h, n, 64, device="cuda", generator=gen).half() for h, n in ((14, 1), (2, 2500), (2, 2500)))
    return lambda: kernels.flash_attn_decode().forward(q, k, v, splits=9)


@pytest.mark.parametrize("make", [_linear, _pair_linear, _head, _split_attention])
def test_two_threads_on_one_stream(make):
    calls = [make(seed) for seed in range(3)]
    want = [call() for call in calls]
    got = [[] for _ in calls]
    start = threading.Barrier(len(calls))

    def work(i):
        start.wait()
        for _ in range(300):
            got[i].append(calls[i]())

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for w, outs in zip(want, got):
        assert len(outs) == 300 and all(torch.equal(o, w) for o in outs)


def _dense_linear(seed):
    w = kernels.F16Weight(896, 896, torch.device("cuda"))
    w.w.normal_(generator=torch.Generator(device="cuda").manual_seed(seed))
    x = torch.randn(200, 896, device="cuda").half()
    return lambda: kernels.w4a16_linear(w, x)


def _attention(seed):
    q, k, v = (torch.randn(2, h, n, 64, device="cuda").half() for h, n in ((14, 1), (2, 700), (2, 700)))
    return lambda: kernels.flash_attn_decode().forward(q, k, v)


@pytest.mark.parametrize("make", [_dense_linear, _attention])
def test_a_thread_may_start_with_a_kernel_of_the_library(make):
    """The call is the thread's first use of CUDA: no context is current in it yet."""
    call = make(1)
    want, got = call(), []
    torch.cuda.synchronize()
    thread = threading.Thread(target=lambda: got.append(call()))
    thread.start()
    thread.join()
    assert len(got) == 1 and torch.equal(got[0], want)


@pytest.mark.parametrize("make", [_linear, _pair_linear, _head, _split_attention])
def test_a_captured_call_has_scratch_of_its_own(make):
    """Two graphs, the second replayed alone and then both: what one clears or leaves behind is not the other's."""
    calls = [make(seed) for seed in (1, 2)]
    want = [call() for call in calls]
    torch.cuda.synchronize()
    kept = set(kernels._scratch.blocks)
    graphs, outs = [], []
    for call in calls:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(call())
        graphs.append(g)
    assert set(kernels._scratch.blocks) == kept
    for order in ((1,), (0, 1), (1, 0, 1)):
        for o in outs:
            o.zero_()
        for i in order:
            graphs[i].replay()
        torch.cuda.synchronize()
        for i in set(order):
            assert torch.equal(outs[i], want[i])
