"""The GEMM on CTA pairs (csrc/awq_gemm_pair.cu) where its tiles, units and plans have their edges: int4 weights against the
oracle, bf16 weights against a float64 product."""

import numpy as np
import pytest
from ml_dtypes import bfloat16

from oracle import awq_oracle as O
from gpu_util import dev_weight, randn_bf16, synth_awq, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from mlir_air_b200 import ops as _ops
    return _ops


def _nan(*shape):
    """An output to be written in full: an element that no CTA writes stays NaN."""
    import torch
    return torch.full(shape, float("nan"), dtype=torch.bfloat16, device="cuda")


# unit of 32 token rows, piece of up to 256, two k-blocks of 64 at a time, 256 columns per pair (128 per CTA):
# one row; a row either side of a unit; of the two-set limit (128); of a piece; rounds and remainders over several column
# tiles, meeting at the edge of one and inside one, with cuts moved to an edge, with one accumulator set and with two; the second
# CTA's columns missing, partly missing, complete
SHAPES = [(1, 128, 32), (31, 128, 128), (33, 256, 160), (128, 384, 256), (129, 384, 288), (256, 128, 512), (257, 640, 96),
          (300, 256, 2400), (777, 256, 1056), (1030, 128, 4128), (96, 1024, 20480), (700, 256, 9600), (600, 128, 19968), (900, 384, 12992)]


@pytest.mark.parametrize("M,K,N", SHAPES)
def test_int4_edges(ops, M, K, N):
    qw, qz, s = synth_awq(K, N, 128, seed=M + 5 * N)
    A, R = randn_bf16((M, K), seed=7), randn_bf16((M, N), seed=9)
    w = dev_weight(qw, qz, s)
    acc = A.astype(np.float32) @ O.dequant_to_bf16(qw, qz, s, 128).astype(np.float32)  # the kernel's own operands
    # f32 sums in another order move a result across a bf16 rounding boundary (2^-8) now and then; a wrong product is 1e-1
    assert O.rel_l2(to_host(ops.gemm(to_dev(A), w, out=_nan(M, N))), acc.astype(bfloat16)) <= 1e-3
    assert O.rel_l2(to_host(ops.gemm(to_dev(A), w, residual=to_dev(R), out=_nan(M, N))), (acc + R.astype(np.float32)).astype(bfloat16)) <= 1e-3
    gate, up = (acc[:, i::2].astype(bfloat16).astype(np.float32) for i in (0, 1))
    swiglu = (gate * 0.5 * (np.tanh(gate * 0.5) + 1.0) * up).astype(bfloat16)
    assert O.rel_l2(to_host(ops.gemm(to_dev(A), w, swiglu=True, out=_nan(M, N // 2))), swiglu) <= 2e-3  # two rounded factors
    ops.gemm_check()


@pytest.mark.parametrize("M,K,N", [(16, 8, 8), (17, 72, 136), (64, 136, 250), (129, 2048, 257), (256, 200, 1000), (300, 64, 4104),
                                   (1025, 192, 520)])
def test_bf16_edges(ops, M, K, N):
    """K and N that fill no k-block, no tile and (N % 8 != 0) no 16-byte store."""
    x, W = randn_bf16((M, K), seed=1), randn_bf16((N, K), seed=2)
    y = to_host(ops.linear_bf16(to_dev(x), to_dev(W), out=_nan(M, N)))
    ops.gemm_check()
    ref = (x.astype(np.float64) @ W.astype(np.float64).T).astype(np.float32).astype(bfloat16)
    assert O.rel_l2(y, ref) <= 1e-3


# sizes at which a plan of one round of whole tiles and a rest that begins inside a column tile, two units before its edge, would be
# the cheapest if those two units were nobody's; and one whose rounds and rest do meet inside a column tile
@pytest.mark.parametrize("M,K,N", [(160, 2048, 6400), (300, 4096, 3840), (129, 1024, 6145), (192, 512, 6272), (288, 512, 3840), (320, 512, 3600), (2000, 512, 9000)])
@pytest.mark.parametrize("scratch", [True, False])
def test_bf16_round_and_rest(ops, M, K, N, scratch):
    import torch
    from mlir_air_b200 import _lib
    x, W = to_dev(randn_bf16((M, K), seed=1)), to_dev(randn_bf16((N, K), seed=2))
    y = _nan(M, N)
    if scratch:
        ops.linear_bf16(x, W, out=y)
    else:
        _lib.call("awq_b200_linear_bf16", x.data_ptr(), W.data_ptr(), y.data_ptr(), M, K, N, torch.cuda.current_stream().cuda_stream)
    ops.gemm_check()
    ref = (x.double() @ W.double().T).to(torch.bfloat16).double()
    # f32 sums in another order: now and then across a bf16 rounding boundary.  Rows and column tiles by themselves: what is left
    # out is a small part of the whole
    for d, r in ((y.double() - ref, ref), (y.double().T - ref.T, ref.T)):
        assert bool((d.norm(dim=1) <= 2e-3 * r.norm(dim=1)).all())


def test_bf16_output_at_any_even_address(ops):
    import torch
    x, W = to_dev(randn_bf16((40, 64), seed=1)), to_dev(randn_bf16((136, 64), seed=2))
    flat = torch.zeros(40 * 136 + 8, dtype=torch.bfloat16, device="cuda")
    out = flat[1:1 + 40 * 136].view(40, 136)
    ops.linear_bf16(x, W, out=out)
    assert torch.equal(out, ops.linear_bf16(x, W)) and not flat[0] and not flat[1 + 40 * 136:].any()


def test_runs_back_to_back_are_independent(ops):
    """Launches overlap by programmatic dependent launch: a chain whose every product reads the one before."""
    import torch
    x = to_dev(randn_bf16((200, 512), seed=3))
    W = to_dev((np.random.default_rng(4).standard_normal((512, 512)) / (1.7 * 512 ** 0.5)).astype(bfloat16))
    ws = [dev_weight(*synth_awq(512, 512, 128, seed=i)) for i in range(2)]
    chained, synced = x, x
    for i in range(6):
        chained = ops.linear_bf16(ops.gemm(chained, ws[i % 2]), W)
    for i in range(6):
        synced = ops.gemm(synced, ws[i % 2])
        torch.cuda.synchronize()
        synced = ops.linear_bf16(synced, W)
        torch.cuda.synchronize()
    assert torch.equal(chained, synced)


@pytest.mark.parametrize("M,K,N", [(3000, 4096, 2048), (4096, 8192, 1056), (2048, 2048, 4096)])
def test_int4_deep_products_repeat(ops, M, K, N):
    """Pieces of 256 token rows, whose ring has seven stages, and token rows that come from HBM: k-blocks land out of order and the
    dequant groups look for them at very different times.  Each run gives the same bits."""
    import torch
    w, A = dev_weight(*synth_awq(K, N, 128, seed=5)), torch.randn((M, K), device="cuda").to(torch.bfloat16)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")  # twice the L2
    first = ops.gemm(A, w)
    ref = A.double() @ ops.dequant(w).double()
    assert ((first.double() - ref).norm() <= 3e-3 * ref.norm()).item()  # one bf16 rounding; a k-block of K / 64 that is wrong is 0.1 in its piece
    for i in range(60):
        if i % 2:
            flush.fill_(i)
        assert torch.equal(ops.gemm(A, w, out=_nan(M, N)), first), i
    ops.gemm_check()


# K cut into parts: one piece per part, ragged last tiles and rows, parts of unequal length, N that takes scalar stores
@pytest.mark.parametrize("M,K,N", [(65, 4096, 4096), (16, 8192, 256), (100, 2048, 544), (300, 8192, 2048), (257, 14336, 1056), (40, 1152, 32)])
def test_int4_k_parts(ops, M, K, N):
    qw, qz, s = synth_awq(K, N, 128, seed=M + N)
    A, R = randn_bf16((M, K), seed=7), randn_bf16((M, N), seed=9)
    w = dev_weight(qw, qz, s)
    acc = A.astype(np.float64) @ O.dequant_to_bf16(qw, qz, s, 128).astype(np.float64)
    assert O.rel_l2(to_host(ops.gemm(to_dev(A), w)), acc.astype(np.float32).astype(bfloat16)) <= 1e-3
    assert O.rel_l2(to_host(ops.gemm(to_dev(A), w, residual=to_dev(R))), (acc + R.astype(np.float64)).astype(np.float32).astype(bfloat16)) <= 1e-3
    gate, up = (acc[:, i::2].astype(np.float32).astype(bfloat16).astype(np.float32) for i in (0, 1))
    swiglu = (gate * 0.5 * (np.tanh(gate * 0.5) + 1.0) * up).astype(bfloat16)
    assert O.rel_l2(to_host(ops.gemm(to_dev(A), w, swiglu=True)), swiglu) <= 2e-3
    ops.gemm_check()


@pytest.mark.parametrize("M,K,N", [(512, 8192, 2048), (64, 4096, 250), (17, 8200, 257), (300, 1100 * 8, 520)])
def test_bf16_k_parts(ops, M, K, N):
    x, W = randn_bf16((M, K), seed=1), randn_bf16((N, K), seed=2)
    y = to_host(ops.linear_bf16(to_dev(x), to_dev(W)))
    ops.gemm_check()
    assert O.rel_l2(y, (x.astype(np.float64) @ W.astype(np.float64).T).astype(np.float32).astype(bfloat16)) <= 1e-3


def test_k_parts_without_a_workspace(ops):
    """The entry point without scratch, and one that is given too little, run the product uncut."""
    import torch
    from mlir_air_b200 import _lib
    M, K, N = 128, 14336, 4096
    w, A = dev_weight(*synth_awq(K, N, 128, seed=3)), to_dev(randn_bf16((M, K), seed=4))
    need = _lib.load().awq_b200_gemm_workspace_bytes(M, K, N, 128)
    assert need > 0
    cut, whole, small = ops.gemm(A, w), torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    args = (A.data_ptr(), w.qweight.data_ptr(), w.qzeros.data_ptr(), w.scales.data_ptr())
    stream = torch.cuda.current_stream().cuda_stream
    _lib.call("awq_b200_gemm_bf16", *args, whole.data_ptr(), M, K, N, 128, stream)
    ws = torch.empty(need - 16, dtype=torch.uint8, device="cuda")
    _lib.call("awq_b200_gemm_ws_bf16", *args, None, small.data_ptr(), 0, M, K, N, 128, ws.data_ptr(), ws.numel(), stream)
    ops.gemm_check()
    assert torch.equal(whole, small)
    assert (cut.double() - whole.double()).norm() <= 1e-3 * whole.double().norm()
