"""The per-head norm with a gate where heads are read in pieces of four, and the general kernel where they cannot be."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# one piece; heads that do not fill their group of lanes; the borders of one, two and four pieces a lane; too long, and not of whole pieces
@pytest.mark.parametrize("head_dim", [4, 12, 64, 100, 128, 132, 256, 260, 512, 516, 30])
@pytest.mark.parametrize("n,heads", [(1, 1), (3, 5), (70, 8)])
@pytest.mark.parametrize("dtype,left", [(torch.float32, 0), (torch.bfloat16, 4), (torch.bfloat16, 1)])
def test_head_norm_gate(n, heads, head_dim, dtype, left):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(n + heads + head_dim)
    width = heads * head_dim
    pitch = (left + width + 7) // 4 * 4
    x = torch.randn(n, width, generator=g).to(DEV)
    gate = torch.randn(n, pitch, generator=g).to(dtype).to(DEV)[:, left:left + width]
    w = torch.randn(head_dim, generator=g).to(DEV)
    whole = torch.full((n, pitch), 7.0, dtype=dtype, device=DEV)
    for act in ("silu", "sigmoid"):
        ops.head_norm_gate(x, w, 1e-5, gate, whole[:, left:left + width], heads, head_dim, act)
        y, z = x.double().reshape(n, heads, head_dim), gate.double().reshape(n, heads, head_dim)
        want = y * torch.rsqrt((y * y).mean(-1, keepdim=True) + 1e-5) * w.double() * torch.sigmoid(z) * (z if act == "silu" else 1)
        got = whole[:, left:left + width].double().reshape(want.shape)
        assert (got - want).norm() <= (1e-6 if dtype == torch.float32 else 4e-3) * want.norm()       # a rounding to the output's type
        assert bool((whole[:, :left] == 7.0).all()) and bool((whole[:, left + width:] == 7.0).all())
