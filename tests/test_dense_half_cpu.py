"""Products of many float32 rows as two fp16 terms: what their native call would read out of range is refused in front of it."""

import types

import pytest
import torch

from dia_tts_prune_b200 import _lib, engine
from dia_tts_prune_b200.layers import DenseGeneral

K, N, M = 64, 128, 200


@pytest.fixture
def calls(monkeypatch):
    made = []
    lib = types.SimpleNamespace(dia_b200_dense_workspace_bytes=lambda M, K: 0, dia_b200_dense_forward_half=lambda *a: made.append(a) or 0)
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(engine, "_stream", lambda device: 0)
    return made


@pytest.mark.parametrize("change", [dict(norm_weight=torch.ones(K - 4)), dict(norm_weight=torch.ones(K + 4)), dict(norm_weight=torch.ones(K).double()),
                                    dict(norm_weight=torch.ones(2 * K)[::2]), dict(norm_weight=torch.ones(K), gated=True), dict(x=torch.ones(M, K - 8)),
                                    dict(x=torch.ones(M, K).bfloat16()), dict(x=torch.ones(M, K), gated=True), dict(x=torch.ones(K, M).t()),
                                    dict(residual=torch.zeros(M, N - 4)), dict(residual=torch.zeros(M - 1, N)), dict(residual=torch.zeros(M, N).double())])
def test_what_does_not_fit_is_refused(calls, change):
    half = (torch.zeros(N, K, dtype=torch.float16), torch.ones(N))
    engine.dense_forward_half(torch.ones(M, K), half, torch.ones(K), residual=torch.zeros(M, N))
    engine.dense_forward_half(torch.ones(M, 2, K), half, gated=True)
    assert len(calls) == 2
    with pytest.raises(ValueError):
        engine.dense_forward_half(**{"x": torch.ones(M, K), "half": half, **change})
    assert len(calls) == 2


def test_a_norm_of_another_length_is_refused_by_the_layer(calls, monkeypatch):
    """As with fewer rows, whose product checks it too"""
    d = DenseGeneral((K,), (N,), weight_dtype=torch.bfloat16)
    monkeypatch.setattr(engine, "dense_half_rows", lambda M, N, K, device: True)
    monkeypatch.setattr(d, "kernel_weight_half", lambda: (torch.zeros(N, K, dtype=torch.float16), torch.ones(N)), raising=False)
    with torch.no_grad():
        assert d._forward_tcgen05(torch.ones(M, K), (1,), norm_weight=torch.ones(K)).shape == (M, N)
        with pytest.raises(ValueError):
            d._forward_tcgen05(torch.ones(M, K), (1,), norm_weight=torch.ones(K // 2))
    assert len(calls) == 1
