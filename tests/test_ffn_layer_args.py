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
