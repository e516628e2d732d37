"""gemv of 9 to 64 rows on the fp8-operand kernel against the oracle: every padded row count, two passes, ragged column tiles,
values of very different size, and what must keep taking the other kernels."""
import numpy as np
import pytest
from ml_dtypes import bfloat16

from oracle import awq_oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-3  # results that fall on the other side of a bf16 rounding boundary; the sums themselves agree to f32


@pytest.mark.parametrize("B,K,N", [(9, 128, 32), (16, 256, 288), (17, 512, 512), (32, 1024, 2080), (33, 384, 256), (41, 4096, 1024),
                                   (64, 2048, 5632), (64, 11008, 96)])
def test_vs_oracle(B, K, N, monkeypatch):
    import torch
    from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev, to_host
    from mlir_air_b200 import _lib, ops
    ops.set_decode_kernel("auto")
    monkeypatch.setattr(ops, "GEMV_ROWS_MIN_WEIGHTS", {16: 0, 64: 0})
    assert _lib.load().awq_b200_gemv_rows_workspace_bytes(B, K, N, 128) > 0
    qw, qz, s = synth_awq(K, N, 128, seed=K + N)
    w, ws = dev_weight(qw, qz, s), ops.Workspace(K, N)
    x = np.asarray(randn_bf16((B, K), seed=B), dtype=np.float32)
    x[:, ::61] *= 300.0
    x[1] *= 1e-6
    x[2] = 0.0
    x = x.astype(bfloat16)
    R = randn_bf16((B, N), seed=3)
    ref = O.gemv_A_ref(x, qw, qz, s, 128)
    y = to_host(ops.gemv(to_dev(x), w, ws))
    assert O.rel_l2(y, ref) <= TOL and O.rel_l2(y[1], ref[1]) <= TOL and not y[2].any()
    assert O.rel_l2(to_host(ops.gemv(to_dev(x), w, ws, residual=to_dev(R))), O.gemv_A_ref(x, qw, qz, s, 128, residual=R)) <= TOL
    f = ops.gemv(to_dev(x), w, ws, f32_out=True)
    exact = x.astype(np.float64) @ O.dequant_f32(qw, qz, s, 128).astype(np.float64)
    assert f.dtype == torch.float32 and np.array_equal(f.cpu().numpy().astype(bfloat16).view(np.uint16), y.view(np.uint16))
    assert np.linalg.norm(f.cpu().numpy() - exact) <= 1e-5 * np.linalg.norm(exact)
    ws.check()


@pytest.mark.parametrize("B,big,small", [(16, 1000.0, 0.05), (33, 1000.0, 0.05), (64, 1000.0, 1.0), (32, 40.0, 0.05)])
def test_what_the_split_keeps_of_small_values(B, big, small, monkeypatch):
    """One large value in every group, whose weights are at their zero points: each column is the sum of the small values alone,
    which are below 2^-13 of the large one in part, and there rounded to multiples of 2^-13 (with the large one in [128, 256))."""
    from gpu_util import dev_weight, synth_awq, to_dev
    from mlir_air_b200 import ops
    monkeypatch.setattr(ops, "GEMV_ROWS_MIN_WEIGHTS", {16: 0, 64: 0})
    K, N = 2048, 512
    _, qz, s = synth_awq(K, N, 128, seed=11)
    rng = np.random.default_rng(B)
    nibs = rng.integers(0, 16, size=(K, N), dtype=np.uint8)
    z = O.unpack_awq_int32(qz)
    nibs[5::128] = z
    qw = O.pack_awq_int32(nibs)
    W = (nibs.astype(np.float64) - np.repeat(z, 128, 0)) * np.repeat(s.astype(np.float64), 128, 0)
    x = rng.standard_normal((B, K)) * small
    x[:, 5::128] = big
    x = x.astype(bfloat16)
    w, ws = dev_weight(qw, qz, s), ops.Workspace(K, N)
    y = ops.gemv(to_dev(x), w, ws, f32_out=True).cpu().numpy().astype(np.float64)
    ws.check()
    err = np.linalg.norm(y - x.astype(np.float64) @ W, axis=0)
    quantum = 2.0 ** (np.floor(np.log2(big)) - 7 - 13)
    # elements off by up to half a quantum, independent and uniform: quantum / sqrt(12) each, times the weights' 2-norm; 1.5 for
    # the spread over a column's rows.  And in f32 a group's two terms of 15 times the large one, which cancel: half a unit
    # in the last place (2^-24) for each of the accumulator's four steps, the three FMAs and the sum over the groups
    split = np.sqrt(B) * np.linalg.norm(W, axis=0) * quantum / np.sqrt(12)
    f32 = np.sqrt(B) * 8 * 2.0 ** -24 * 15 * big * np.linalg.norm(s.astype(np.float64), axis=0)
    assert (err <= 1.5 * split + f32).all(), (err / (1.5 * split + f32)).max()


def test_infinity_and_nan_show(monkeypatch):
    from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev, to_host
    from mlir_air_b200 import ops
    monkeypatch.setattr(ops, "GEMV_ROWS_MIN_WEIGHTS", {16: 0, 64: 0})
    K, N = 512, 256
    w, ws = dev_weight(*synth_awq(K, N, 128, seed=5)), ops.Workspace(K, N)
    x = randn_bf16((12, K), seed=6)
    x[3, 7], x[4, 200] = bfloat16(np.inf), bfloat16(np.nan)
    y = to_host(ops.gemv(to_dev(x), w, ws)).astype(np.float32)
    assert not np.isfinite(y[3]).any() and np.isnan(y[4]).all() and np.isfinite(np.delete(y, (3, 4), 0)).all()


def test_other_kernels_stay_where_they_were(monkeypatch):
    import torch
    from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev
    from mlir_air_b200 import _lib, ops
    monkeypatch.setattr(ops, "GEMV_ROWS_MIN_WEIGHTS", {16: 0, 64: 0})
    size = _lib.load().awq_b200_gemv_rows_workspace_bytes
    assert size(8, 512, 256, 128) == 0 and size(65, 512, 256, 128) == 0 and size(16, 512, 264, 128) == 0 and size(16, 512, 256, 64) == 0
    K, N = 512, 256
    w, ws = dev_weight(*synth_awq(K, N, 128, seed=5)), ops.Workspace(K, N)
    flat = torch.zeros(12 * K + 8, dtype=torch.bfloat16, device="cuda")
    off = flat[1:1 + 12 * K].view(12, K)  # not on a 16-byte boundary
    off.copy_(to_dev(randn_bf16((12, K), seed=6)))
    a = ops.gemv(off.clone(), w, ws)
    b = ops.gemv(off, w, ws)
    assert (a.float() - b.float()).norm() <= TOL * a.float().norm()
    try:
        ops.set_decode_kernel("streamk")
        assert size(16, 512, 256, 128) == 0
    finally:
        ops.set_decode_kernel("auto")
