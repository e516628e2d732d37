"""ops.ffn_layer_decode refuses arguments that do not belong together before anything is launched: without a GPU, with the check for
CUDA tensors and the library call replaced."""
import pytest
import torch

from mlir_air_b200 import _lib, ops

H, I = 256, 384


@pytest.fixture
def launched(monkeypatch):
    calls = []
    monkeypatch.setattr(ops, "_want", lambda t, dtype, name: t)
    monkeypatch.setattr(ops, "_stream", lambda: None)
    monkeypatch.setattr(_lib, "call", lambda name, *args: calls.append(name))
    return calls


def _weight(K, N, gs=128):
    return ops.AwqWeight(torch.zeros((K, N // 8), dtype=torch.int32), torch.zeros((K // gs, N // 8), dtype=torch.int32),
                         torch.zeros((K // gs, N), dtype=torch.bfloat16), gs)


def _call(x=(9, H), gu_gs=128, down_gs=128, gamma=H, out=None):
    bf = torch.bfloat16
    return ops.ffn_layer_decode(torch.zeros(x, dtype=bf), _weight(H, 2 * I, gu_gs), _weight(I, H, down_gs),
                                ops.GemmDecodeWorkspace(2 * I, device="cpu", K=I), torch.zeros(gamma, dtype=bf),
                                out=None if out is None else torch.zeros(out, dtype=bf))


def test_accepts_what_fits(launched):
    assert _call().shape == (9, H) and _call(out=(9, H)).shape == (9, H)
    assert len(launched) == 2


@pytest.mark.parametrize("gu_gs,down_gs", [(128, 64), (128, 384), (64, 128)])
def test_refuses_weights_of_different_group_sizes(launched, gu_gs, down_gs):
    """One group size goes to the kernels: the other weight's scales and zeros would be read with the wrong row count, past
    their end where its groups are larger."""
    with pytest.raises(_lib.AwqBackendError, match="group size"):
        _call(gu_gs=gu_gs, down_gs=down_gs)
    assert not launched


@pytest.mark.parametrize("gamma", [H - 128, 2 * H, (2, H)])
def test_refuses_a_norm_weight_of_another_length(launched, gamma):
    with pytest.raises(_lib.AwqBackendError, match="gamma"):
        _call(gamma=gamma)
    assert not launched


@pytest.mark.parametrize("x,out", [((9, H), (8, H)), ((9, H), (9, I)), ((9, H), (H, 9)), ((H,), (2, H))])
def test_refuses_an_output_of_another_shape(launched, x, out):
    with pytest.raises(_lib.AwqBackendError, match="out"):
        _call(x=x, out=out)
    assert not launched


def test_one_row_may_be_a_vector(launched):
    assert _call(x=(H,)).shape == (1, H) and _call(x=(H,), out=(H,)).shape == (H,) and _call(x=(1, H), out=(1, H)).shape == (1, H)
    assert len(launched) == 3


def _stack(**attributes):
    from types import SimpleNamespace as NS
    from mlir_air_b200 import ffn
    w = lambda K, N: NS(K=K, N=N, group_size=128)
    st = object.__new__(ffn.DecodeFFNStack)  # (the constructor's buffers need a GPU; the choice of the path does not)
    layer = NS(gateup=w(H, 2 * I), down=w(I, H), gamma=torch.ones(H))
    st.__dict__.update(tp=1, plan=None, one_call=True, layers=[layer] * 3, gemm_ws=ops.GemmDecodeWorkspace(2 * I, device="cpu", K=I), **attributes)
    return st


def test_one_call_layers_are_switched_by_their_argument():
    from mlir_air_b200.ffn import DecodeFFNStack
    st = _stack()
    assert [st.uses_layer(b) for b in (8, 9, 32, 33, 64, 65)] == [False, True, True, True, True, False] and st.launches_per_step(16) == 15
    st.one_call = False
    assert not any(st.uses_layer(b) for b in range(1, 66)) and st.uses_gemm(16) and st.launches_per_step(16) == 15 and not st.uses_gemm_f8(16)
    # the class's own size bars, given to a stack again, change nothing; others choose between the separate products
    assert _stack(GEMM_F8_MIN_WEIGHTS=dict(DecodeFFNStack.GEMM_F8_MIN_WEIGHTS)).uses_layer(16)
    st = _stack(GEMM_F8_MIN_WEIGHTS={16: 0, 32: 0})
    assert not st.uses_layer(16) and st.uses_gemm_f8(16) and st.launches_per_step(16) == 21 and st.launches_per_step(33) == 15
