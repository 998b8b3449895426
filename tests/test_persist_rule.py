"""Which decode batches take the persistent kernel (no GPU needed here)."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from quic_cu_b200 import kernels, model
from quic_cu_b200.checkpoint import qwen_config_dict


@pytest.mark.parametrize("asked", [None, True])
@pytest.mark.parametrize("dense", [False, True])
def test_a_device_with_fewer_sms_keeps_the_kernel_chain(monkeypatch, asked, dense):
    real = kernels.lib()
    fits = [1]
    fake = SimpleNamespace(quic_persist_device_ok=lambda: fits[0], quic_persist_max_rows=real.quic_persist_max_rows,
                           quic_persist_stream_bytes=real.quic_persist_stream_bytes,
                           quic_persist_pick_splits=real.quic_persist_pick_splits)
    monkeypatch.setattr(kernels, "lib", lambda: fake)
    batches = [(rows, ctx) for rows in (2, 5, 16) for ctx in (128, 1024)]
    for fits[0], want in ((1, True), (0, False)):
        net = model.QUICForCausalLM(qwen_config_dict(24, 151936), device="cpu")
        net.use_persist, net.dense = asked, dense
        assert [net.persist_ok(*b) for b in batches] == [want] * len(batches)


@pytest.mark.parametrize("dense,rows,length,takes", [
    (False, 1, 700, True), (False, 1, 2100, False), (False, 2, 2100, True), (False, 2, 2600, False), (False, 2, 4200, True),
    (False, 3, 2500, True), (False, 3, 3700, False), (False, 5, 2300, True), (False, 5, 2561, False), (True, 5, 2100, True),
    (True, 5, 3700, False), (True, 8, 2100, True), (True, 8, 2400, False), (True, 2, 5000, True)])
def test_the_rule_hears_of_the_context_and_not_of_the_caches_size(monkeypatch, dense, rows, length, takes):
    """The same rows in a cache of just their size and in a large one: same kernel, and a launch that covers every row."""
    real = kernels.lib()
    fake = SimpleNamespace(quic_persist_device_ok=lambda: 1, quic_persist_max_rows=real.quic_persist_max_rows,
                           quic_persist_stream_bytes=real.quic_persist_stream_bytes,
                           quic_persist_pick_splits=real.quic_persist_pick_splits)
    monkeypatch.setattr(kernels, "lib", lambda: fake)
    net = model.QUICForCausalLM(qwen_config_dict(24, 151936), device="cpu")
    net.use_persist, net.dense = None, dense
    captured = []
    monkeypatch.setattr(net, "_graph", lambda cache, batch, ctx, steps, logits: (captured.append(ctx), cache.tok[:batch].clone()))
    for s_max in (length + 8, 8192):
        cache = model.SlotCache(1, rows, s_max, 151936, torch.device("cpu"))
        cache.host_len = [length - i for i in range(rows)]
        captured.clear()
        handle, _ = net._prepare_decode(cache, list(range(rows)), 8, None)
        assert isinstance(handle, kernels.Decode) == takes
        assert length + 8 <= (handle.ctx_hint if takes else captured[0]) <= s_max


def test_one_packed_row_takes_it_where_it_was_measured_ahead():
    """Context bounds as decode() rounds them up: the chain serves 1..512 tokens and more than 768."""
    takes = {ctx for ctx in range(128, 4097, 128) if model._persist_pays(False, 1, ctx)}
    assert takes == {640, 768}
    assert all(model._persist_pays(True, 1, ctx) for ctx in (128, 512, 4096))
    assert all(model._persist_pays(dense, rows, 512) for dense in (False, True) for rows in (2, 3, 16))
