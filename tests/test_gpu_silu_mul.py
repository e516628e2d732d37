"""silu_mul on whole 16-byte pieces, remainders and buffers off the 16-byte boundary."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,off", [(1, 0), (7, 0), (8, 0), (2051, 0), (4096, 1), (33, 4)])
def test_silu_mul(n, off):
    """Whole eights, a remainder, and buffers off the 16-byte boundary: bit for bit what one value at a time gives."""
    import torch
    from mlir_air_b200 import ops
    g, u = (torch.randn(n + 8, device="cuda").mul(4).bfloat16()[off:off + n] for _ in range(2))
    flat = torch.zeros(n + 16, dtype=torch.bfloat16, device="cuda")
    ops.silu_mul(g, u, out=flat[off:off + n])
    gd, ud = g.double(), u.double()
    ref = (gd / (1 + torch.exp(-gd)) * ud)
    # one bf16 rounding (8 significant bits: at most 2^-8 of the value) and f32 arithmetic
    assert ((flat[off:off + n].double() - ref).abs() <= ref.abs() * (2 ** -8 + 1e-5) + 1e-38).all()
    assert not flat[:off].any() and not flat[off + n:].any()
    one = torch.stack([ops.silu_mul(g[i:i + 1].clone(), u[i:i + 1].clone())[0] for i in range(min(n, 40))])
    assert torch.equal(one, flat[off:off + min(n, 40)])
