"""The scaled sum and the norm behind it, in pieces of four numbers and one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# one piece up to the four a thread holds, one number past each limit, and widths that are no whole pieces
@pytest.mark.parametrize("n,width", [(1, 4), (3, 1024), (2, 1028), (5, 2048), (1, 2052), (2, 4096), (2, 4100), (3, 30)])
@pytest.mark.parametrize("dtype,rel", [(torch.float32, 1e-5), (torch.bfloat16, 4e-3)])       # float32 sums; rounded to bfloat16
def test_scaled_add_norm(n, width, dtype, rel):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(width)
    y, r = (torch.randn(n, width, generator=g).to(DEV) for _ in range(2))
    w = (1 + 0.1 * torch.randn(width, generator=g)).to(DEV)
    want = r.double() + 0.37 * y.double()
    out = torch.full((n + 1, width), 7.0, dtype=dtype, device=DEV)
    ops.scaled_add_norm(y, 0.37, r, w, 1e-5, out[:n])
    normed = want * torch.rsqrt((want * want).mean(1, keepdim=True) + 1e-5) * w.double()
    assert (r.double() - want).norm() <= 1e-6 * want.norm()
    assert (out[:n].double() - normed).norm() <= rel * normed.norm() and bool((out[n] == 7.0).all())
    ops.scaled_add(y, -0.37, r)
    back = want - 0.37 * y.double()
    assert (r.double() - back).norm() <= 1e-6 * want.norm()
