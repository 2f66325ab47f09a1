"""RMS norm of many rows: one warp a row and four, widths around the changes, rows that do not fill a block, chosen rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [256, 257, 301])
@pytest.mark.parametrize("width", [4, 1024, 1028, 2048, 2052, 3072, 4092, 4096, 4100])
@pytest.mark.parametrize("chosen,add_unit", [(False, False), (True, True)])
def test_rows(n, width, chosen, add_unit):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(n + width)
    x = torch.randn(n + 9, width, generator=g).to(DEV)
    w = torch.randn(width, generator=g).to(DEV)
    rows = torch.randperm(n + 9, generator=g)[:n].to(torch.int32).to(DEV) if chosen else None
    out = torch.full((n + 1, width), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.rmsnorm(x if chosen else x[:n], w, out[:n], 1e-5, rows, add_unit)
    y = (x[rows.long()] if chosen else x[:n]).double()
    want = y * torch.rsqrt((y * y).mean(1, keepdim=True) + 1e-5) * (w.double() + (1 if add_unit else 0))
    assert (out[:n].double() - want).norm() <= 4e-3 * want.norm()        # rounded to bfloat16
    assert bool((out[n] == 7.0).all())
