"""One decode FFN layer in one call (awq_b200_ffn_layer_decode_bf16) against the numpy oracle: every padded row count, ragged
column tiles, few and many contributors per tile."""
import numpy as np
import pytest
from ml_dtypes import bfloat16

from oracle import awq_oracle as O

pytestmark = pytest.mark.gpu

# bf16 rounding of the normed rows, of gate and up, of the SwiGLU output and of the result: about 2^-9 / sqrt(3) each
REL_L2_TOL = 4e-3


@pytest.mark.parametrize("B,H,I", [(1, 128, 128), (9, 128, 256), (16, 256, 384), (17, 512, 1408), (32, 384, 640), (33, 512, 1152),
                                   (48, 1024, 2816), (64, 2048, 5632), (64, 128, 4096), (13, 4096, 128)])
def test_layer_vs_oracle(B, H, I):
    import torch
    from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev, to_host
    from mlir_air_b200 import ops
    gate, up = synth_awq(H, I, 128, seed=H + I), synth_awq(H, I, 128, seed=H + I + 1)
    down = synth_awq(I, H, 128, seed=H + I + 2, scale_lo=0.0005, scale_hi=0.004)
    gamma = (np.random.default_rng(H).standard_normal(H) * 0.1 + 1.0).astype(bfloat16)
    wgu, wd = ops.interleave_gate_up(dev_weight(*gate), dev_weight(*up)), dev_weight(*down)
    ws = ops.GemmDecodeWorkspace(max(2 * I, H), batch=64, K=max(H, I))
    assert ws.fits_layer(B, H, I)
    ws.buf.fill_(0xFF)  # NaN in every word: nothing may be read that was not written
    x = np.asarray(randn_bf16((B, H), seed=B), dtype=np.float32)
    x[:, ::97] *= 1000.0  # groups and elements of very different size
    x[0, :64] = 0.0
    x = x.astype(bfloat16)
    y = ops.ffn_layer_decode(to_dev(x), wgu, wd, ws, to_dev(gamma))
    ops.gemm_check()
    inplace = to_dev(x)
    ops.ffn_layer_decode(inplace, wgu, wd, ws, to_dev(gamma), out=inplace)
    ops.gemm_check()
    assert torch.equal(y, inplace)
    ref = O.ffn_layer_A_ref(x, gamma, gate, up, down, 128)
    assert O.rel_l2(to_host(y), ref) <= REL_L2_TOL
    # without the residual, which is most of the result
    d, r = to_host(y).astype(np.float32) - x.astype(np.float32), ref.astype(np.float32) - x.astype(np.float32)
    small = np.ones(H, bool)
    small[::97] = False
    assert O.rel_l2(d[:, small], r[:, small]) <= 1e-2


@pytest.mark.parametrize("B", [9, 32])
def test_large_normalised_values_beside_small_ones(B):
    """A norm weight of 300 in every group, whose gate/up weights are at their zero points, so that gate and up are sums of the
    other values, which the split keeps to 2^-21 of the large one: nothing beside their bf16 rounding.  Judged column by column."""
    from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev, to_host
    from mlir_air_b200 import ops
    H, I = 512, 1408
    def at_zero(w):
        qw, qz, s = w
        nibs = O.unpack_awq_int32(qw)
        nibs[5::128] = O.unpack_awq_int32(qz)
        return O.pack_awq_int32(nibs), qz, s
    gate, up = at_zero(synth_awq(H, I, 128, seed=1)), at_zero(synth_awq(H, I, 128, seed=2))
    down = synth_awq(I, H, 128, seed=3, scale_lo=0.0005, scale_hi=0.004)
    gamma = (np.random.default_rng(4).standard_normal(H) * 0.1 + 1.0).astype(bfloat16)
    gamma[5::128] = 300.0
    x = (np.asarray(randn_bf16((B, H), seed=B), dtype=np.float32) * 2.0 ** -10).astype(bfloat16)  # (the residual does not hide the layer)
    ws = ops.GemmDecodeWorkspace(2 * I, batch=64, K=I)
    y = to_host(ops.ffn_layer_decode(to_dev(x), ops.interleave_gate_up(dev_weight(*gate), dev_weight(*up)), dev_weight(*down), ws,
                                     to_dev(gamma))).astype(np.float64)
    ops.gemm_check()
    ref = O.ffn_layer_A_ref(x, gamma, gate, up, down, 128).astype(np.float64)
    # the rounding points that REL_L2_TOL counts; a column has only B values: twice as much
    assert (np.linalg.norm(y - ref, axis=0) <= 2 * REL_L2_TOL * np.linalg.norm(ref, axis=0)).all()


def test_layer_refuses():
    import torch
    from gpu_util import dev_weight, synth_awq
    from mlir_air_b200 import ops
    from mlir_air_b200._lib import AwqBackendError
    w, d = dev_weight(*synth_awq(128, 512, 128, seed=1)), dev_weight(*synth_awq(256, 128, 128, seed=2))
    ws = ops.GemmDecodeWorkspace(512, batch=64, K=256)
    g = torch.ones(128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(AwqBackendError):
        ops.ffn_layer_decode(torch.zeros((65, 128), dtype=torch.bfloat16, device="cuda"), w, d, ws, g)
    with pytest.raises(AwqBackendError):
        ops.ffn_layer_decode(torch.zeros((8, 128), dtype=torch.bfloat16, device="cuda"), w, w, ws, g)


@pytest.mark.parametrize("B", [9, 16, 33, 64])
def test_stack_in_one_call_per_layer(B):
    """What a stack on one GPU runs by itself, in its three call forms, and the separate products that `one_call` = False asks for."""
    import torch
    from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev, to_host
    from mlir_air_b200 import ffn, ops
    H, I, L = 512, 1408, 3
    layers_np = []
    for l in range(L):
        gate, up = synth_awq(H, I, 128, seed=10 * l), synth_awq(H, I, 128, seed=10 * l + 1)
        down = synth_awq(I, H, 128, seed=10 * l + 2, scale_lo=0.0005, scale_hi=0.004)
        layers_np.append((gate, up, down, (np.random.default_rng(l).standard_normal(H) * 0.1 + 1.0).astype(bfloat16)))
    layers = [ffn.FFNLayer(ops.interleave_gate_up(dev_weight(*g), dev_weight(*u)), dev_weight(*d), to_dev(gm)) for g, u, d, gm in layers_np]
    x = randn_bf16((B, H), seed=B)
    ref = x
    for gate, up, down, gamma in layers_np:
        ref = O.ffn_layer_A_ref(ref, gamma, gate, up, down, 128)
    stack = ffn.DecodeFFNStack(layers, H)
    assert stack.uses_layer(B) and stack.launches_per_step(B) == 5 * L
    y = stack.step(to_dev(x))
    stack.load_input(to_dev(x))
    assert torch.equal(stack.replay(B), y)
    assert np.array_equal(stack.forward_host(x).view(np.uint16), to_host(y).view(np.uint16))
    assert O.rel_l2(to_host(y), ref) <= L * REL_L2_TOL
    apart = ffn.DecodeFFNStack(layers, H, one_call=False)
    assert not apart.uses_layer(B) and apart.uses_gemm(B)
    assert O.rel_l2(to_host(apart.step(to_dev(x))), ref) <= L * REL_L2_TOL
    stack.check(), apart.check()
