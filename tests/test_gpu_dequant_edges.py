"""dequant where the numbering of its threads over (block of k, word column) has its edges: bit for bit what the oracle gives."""
import numpy as np
import pytest

from oracle import awq_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N,gs", [(4, 8, 4), (12, 24, 4), (128, 8, 128), (136, 1032, 8), (256, 264, 32), (128, 1024, 128), (9, 40, 3)])
def test_dequant_edges(K, N, gs):
    import torch
    from gpu_util import dev_weight, synth_awq, to_host
    from mlir_air_b200 import ops
    qw, qz, s = synth_awq(K, N, gs, seed=K + N)
    flat = torch.zeros(K * N + 16, dtype=torch.bfloat16, device="cuda")
    w = dev_weight(qw, qz, s, gs)
    ops.dequant(w, out=flat[8:8 + K * N].view(K, N))
    assert np.array_equal(to_host(flat[8:8 + K * N].view(K, N)).view(np.uint16), O.dequant_to_bf16(qw, qz, s, gs).view(np.uint16))
    assert not flat[:8].any() and not flat[8 + K * N:].any()
