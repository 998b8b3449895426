"""Linears of many rows (the SM pair GEMM) against fp32 products: tile edges, every tile width, K splits
with and without room for them, bias; and a prefill that takes it against the same prompts in calls that do not."""

from __future__ import annotations

import ctypes as C

import pytest
import torch

from quic_cu_b200 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (129, 896, 896), (255, 1152, 896), (257, 192, 4864), (300, 9728, 128),
                                   (385, 896, 4864), (5000, 1152, 128)])
@pytest.mark.parametrize("bias", [False, True])
def test_dense_linear(m, n, k, bias):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    b = torch.randn(n, device="cuda", generator=gen).half() if bias else None
    w = kernels.F16Weight(n, k, torch.device("cuda"), bias=b)
    w.w.copy_(torch.randn(n, k, device="cuda", generator=gen) * 0.05)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    want = (x.float() @ w.w.float().T).half().float() + (0 if b is None else b.float())
    y = kernels.w4a16_linear(w, x)
    assert (y.float() - want).norm() <= 1e-3 * want.norm()


@pytest.mark.parametrize("m,n,k", [(689, 9728, 896), (1377, 896, 4864), (1500, 896, 4864), (5900, 1152, 896)])
def test_packed_linear_equals_the_same_rows_in_smaller_calls(m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    w = kernels.W4Weight(n, k, torch.device("cuda"))
    w.qw.random_(-2 ** 31, 2 ** 31 - 1, generator=gen)
    w.zp.random_(0, 255, generator=gen)
    w.sc.copy_(torch.rand(w.sc.shape, device="cuda", generator=gen) * 0.02)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    want = torch.cat([kernels.w4a16_linear(w, x[i:i + 500]) for i in range(0, m, 500)]).float()
    y = kernels.w4a16_linear(w, x)
    assert (y.float() - want).norm() <= 1e-3 * want.norm()


# either side of the lines where a packed linear's waves of tiles make one GEMM or the other the faster
@pytest.mark.parametrize("m,n,k", [(768, 9728, 896), (769, 9728, 896), (4864, 896, 4864), (4865, 896, 4864), (5377, 896, 4864),
                                   (6144, 1152, 896), (6145, 1152, 896)])
def test_packed_linear_around_the_lines_of_the_rule(m, n, k):
    test_packed_linear_equals_the_same_rows_in_smaller_calls(m, n, k)


@pytest.mark.parametrize("m,n,k", [(7000, 192, 4864), (3000, 448, 4864)])
def test_packed_linear_stays_inside_its_workspace(m, n, k):
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    w = kernels.W4Weight(n, k, torch.device("cuda"))
    w.qw.random_(-2 ** 31, 2 ** 31 - 1, generator=gen)
    w.zp.random_(0, 255, generator=gen)
    w.sc.copy_(torch.rand(w.sc.shape, device="cuda", generator=gen) * 0.02)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    size = kernels.lib().quic_w4a16_workspace_bytes(m, n, k)
    arena = torch.full((size + (32 << 20),), 0x5a, dtype=torch.uint8, device="cuda")
    arena[:size] = 0
    y = torch.empty(m, n, dtype=torch.float16, device="cuda")
    s = w.struct()
    kernels.check(kernels.lib().quic_w4a16_linear(x.data_ptr(), C.byref(s), y.data_ptr(), m, 1, arena.data_ptr(),
                                                  kernels.stream_ptr()), "w4a16_linear")
    want = x.float() @ w.dequant().float().T
    assert (y.float() - want).norm() <= 1e-3 * want.norm()
    assert bool((arena[size:] == 0x5a).all())


# the last row count that the pair GEMM would split six ways, and the first at four
@pytest.mark.parametrize("m", [128, 129, 768, 769])
def test_dense_linear_of_long_k_with_a_workspace(m):
    n, k = 896, 4864
    gen = torch.Generator(device="cuda").manual_seed(m)
    w = kernels.F16Weight(n, k, torch.device("cuda"))
    w.w.copy_(torch.randn(n, k, device="cuda", generator=gen) * 0.05)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    y, ws = torch.empty(m, n, device="cuda").half(), torch.empty(kernels.lib().quic_w4a16_workspace_bytes(m, n, k), dtype=torch.uint8, device="cuda")
    s = w.struct()
    kernels.check(kernels.lib().quic_w4a16_linear(x.data_ptr(), C.byref(s), y.data_ptr(), m, 1, ws.data_ptr(), kernels.stream_ptr()), "linear")
    want = x.float() @ w.w.float().T
    assert (y.float() - want).norm() <= 1e-3 * want.norm()


@pytest.mark.parametrize("n", [896, 192])
@pytest.mark.parametrize("y_off,bias_off,room", [(1, 0, False), (4, 0, True), (1, 0, True), (0, 1, False), (0, 1, True), (3, 3, True)])
def test_dense_linear_takes_any_output_and_bias_address(n, y_off, bias_off, room):
    m, k = 130, 896
    gen = torch.Generator(device="cuda").manual_seed(n + y_off)
    bias = torch.randn(n + 8, device="cuda", generator=gen).half()[bias_off:bias_off + n]
    w = kernels.F16Weight(n, k, torch.device("cuda"), bias=bias)
    w.w.copy_(torch.randn(n, k, device="cuda", generator=gen) * 0.05)
    x = torch.randn(m, k, device="cuda", generator=gen).half()
    out = torch.zeros(m * n + 8, dtype=torch.float16, device="cuda")
    ws = torch.zeros(kernels.lib().quic_w4a16_workspace_bytes(m, n, k) + 16, dtype=torch.uint8, device="cuda") if room else None
    s = w.struct()
    kernels.check(kernels.lib().quic_w4a16_linear(x.data_ptr(), C.byref(s), out.data_ptr() + 2 * y_off, m, 1, kernels.ptr(ws),
                                                  kernels.stream_ptr()), "linear")
    want = (x.float() @ w.w.float().T).half().float() + bias.float()
    y = out[y_off:y_off + m * n].view(m, n).float()
    assert (y - want).norm() <= 1e-3 * want.norm()
    assert not out[:y_off].any() and not out[y_off + m * n:].any()


@pytest.mark.parametrize("lens", [[768], [500, 266, 2], [700, 700, 650]], ids=str)
def test_prefill_equals_one_prompt_at_a_time(tiny_model, lens):
    net = tiny_model[0]
    gen = torch.Generator().manual_seed(sum(lens))
    prompts = [torch.randint(0, 2048, (n,), generator=gen) for n in lens]
    whole, parts = (net.new_cache(n_slots=4, s_max=1100) for _ in range(2))
    _, logits = net.prefill(whole, list(range(len(lens))), prompts)
    for i, p in enumerate(prompts):
        half = len(p) // 2
        if half > 1:  # in two calls of fewer rows
            net.prefill(parts, [i], [p[:half]])
        _, one = net.prefill(parts, [i], [p[half:]] if half > 1 else [p], offsets=[half] if half > 1 else None)
        assert (logits[i].float() - one[0].float()).norm() <= 1e-2 * one[0].float().norm()
    assert (whole.kv.float() - parts.kv.float()).norm() <= 5e-3 * parts.kv.float().norm()
