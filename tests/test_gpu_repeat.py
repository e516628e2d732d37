"""Decode products whose code and operands are not in the caches: loads come late and out of step, and a warp that released a stage
of its ring before it had read all of it would take another unit's values now and then.  The sums are added as integers, so every run
gives the same bits."""
import pytest
from ml_dtypes import bfloat16

from oracle import awq_oracle as O

pytestmark = pytest.mark.gpu


# one and two rows (the hand-over of the rows that exist), eight, more than eight (the multi-row kernel, the fp8-operand kernel)
@pytest.mark.parametrize("B", [1, 2, 8, 12, 33])
@pytest.mark.parametrize("K,N", [(8192, 28672), (28672, 8192)])
def test_cold_launches_give_the_same_bits(B, K, N):
    import torch
    from mlir_air_b200 import ops
    gen = torch.Generator(device="cuda")
    gen.manual_seed(B)
    words = lambda *shape: torch.randint(-2 ** 31, 2 ** 31 - 1, shape, dtype=torch.int32, device="cuda", generator=gen)
    w = ops.AwqWeight(words(K, N // 8), words(K // 128, N // 8),
                      (torch.rand((K // 128, N), device="cuda", generator=gen) * 0.019 + 0.001).to(torch.bfloat16))
    x = torch.randn((B, K), device="cuda", generator=gen).to(torch.bfloat16)
    ws = ops.Workspace(K, N)
    flush = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")  # twice the L2
    first = ops.gemv(x, w, ws).clone()
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for i in range(500):
        flush.fill_(i & 255)
        differ += (ops.gemv(x, w, ws).view(torch.int16) != first.view(torch.int16)).any()
    assert int(differ) == 0
    ws.check()
    cols = slice(0, 64)  # and they are the right ones, on the columns of one warp
    part = ops.AwqWeight(w.qweight[:, :8].contiguous(), w.qzeros[:, :8].contiguous(), w.scales[:, cols].contiguous())
    ref = O.gemv_A_ref(x.cpu().view(torch.int16).numpy().view(bfloat16), part.qweight.cpu().numpy(), part.qzeros.cpu().numpy(),
                       part.scales.cpu().view(torch.int16).numpy().view(bfloat16), 128)
    got = first[:, cols].contiguous().cpu().view(torch.int16).numpy().view(bfloat16)
    assert O.rel_l2(got, ref) <= 1e-3
