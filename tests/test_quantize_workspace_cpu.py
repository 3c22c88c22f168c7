"""Which workspace a call of the one-launch quantiser gets (host code only: the library is a stand-in that records its arguments)."""
import types

import pytest
import torch


@pytest.fixture
def quant(monkeypatch):
    import sm120fp4_b200._lib as L
    from sm120fp4_b200 import quant as Q
    calls = []
    fake = types.SimpleNamespace(b200moe_quantize_own_scale_workspace_bytes=lambda dt, g, r, k: 8 + 8 * g * -(-r * k // 16384),
                                 b200moe_quantize_nvfp4_own_scale=lambda *a: calls.append(types.SimpleNamespace(ws=a[9], nbytes=a[10])) or 0)
    state = types.SimpleNamespace(calls=calls, capturing=False, stream=7, Q=Q)
    monkeypatch.setattr(L, "lib", lambda: fake)
    monkeypatch.setattr(L, "stream_ptr", lambda: state.stream)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state.capturing)
    monkeypatch.setattr(Q, "_WS", {})
    return state


def call(state, rows, k=2048):
    x = torch.zeros(rows, k, dtype=torch.bfloat16)
    out = [torch.empty(n, dtype=torch.uint8) for n in (4, rows * k // 2, rows * k // 16)]
    state.Q._own_scale(x, 1, rows, k, *out, 0, "test")
    return state.calls[-1]


def test_eager_calls_of_a_stream_share_one(quant):
    a = call(quant, 128)
    assert call(quant, 100).ws == a.ws and len(quant.Q._WS) == 1
    quant.stream = 8
    assert call(quant, 128).ws != a.ws and len(quant.Q._WS) == 2
    big = call(quant, 16384)
    assert list(quant.Q._WS.values())[1].numel() >= big.nbytes and len(quant.Q._WS) == 2


def test_captured_calls_share_none(quant, monkeypatch):
    kept, zeros = [], torch.zeros
    monkeypatch.setattr(torch, "zeros", lambda *a, **k: kept.append(zeros(*a, **k)) or kept[-1])   # keeps them alive: no address is used twice
    eager = call(quant, 128)
    quant.capturing = True
    captured = [call(quant, 128) for _ in range(2)]
    assert len({eager.ws, captured[0].ws, captured[1].ws}) == 3 and len(quant.Q._WS) == 1
    quant.stream = 8           # the first call on a stream is a captured one: no eager call may find its workspace
    call(quant, 128)
    assert len(quant.Q._WS) == 1


def test_streams_that_went_do_not_pile_up(quant):
    for quant.stream in range(100):
        call(quant, 128)
    assert len(quant.Q._WS) == 64
