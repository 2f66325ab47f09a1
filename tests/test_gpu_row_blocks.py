"""Residual streams of few tokens (sixteen warps a row) against the same tokens among many (eight; the same bits) and float64; the gate
per head in whole pieces and single elements."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# widths around one piece a thread of eight and of sixteen warps; groups that split the warps evenly, unevenly and one each
@pytest.mark.parametrize("width,groups", [(1024, 2), (1032, 1), (2048, 2), (2048, 16), (2080, 5), (3072, 3), (3072, 4), (3072, 8), (4104, 9)])
@pytest.mark.parametrize("streams", [1, 4])
@pytest.mark.parametrize("shifted", [False, True])
def test_streams_of_few_tokens(width, groups, streams, shifted):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(width + groups)
    rand = lambda *s: torch.randn(*s, generator=g).to(DEV)
    many, few = 400, 5
    x, y = rand(many, streams, width), rand(many, width)
    a, b, mix, w, mu = rand(streams), rand(streams), rand(streams, streams), rand(width), rand(width)
    states = rand(many, width)
    results = []
    for n in (many, few):
        out, new, state = torch.empty(n, width, device=DEV), torch.empty(n, streams, width, device=DEV), states.clone()
        i32 = lambda t: t.to(torch.int32).to(DEV)
        step = types.SimpleNamespace(cu_tokens=i32(torch.arange(n + 1)), slot_of_token=i32(torch.arange(n)), r=n, n=n)
        ops.stream_step(x[:n], w, 1e-5, groups, out, a, (y[:n], mix, b), new, shift=(mu, state, True) if shifted else None,
                        step=step if shifted else None)
        results.append((out[:few], new[:few], state[:few]))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    X, Y = x[:few].double(), y[:few].double()
    new = torch.einsum("nsw,st->ntw", X, mix.double()) + b.double()[None, :, None] * Y[:, None]
    u = (new * a.double()[None, :, None]).sum(1).reshape(few, groups, -1)
    h = (u * torch.rsqrt((u * u).mean(-1, keepdim=True) + 1e-5)).reshape(few, width) * w.double()
    out = h + (states[:few].double() - h) * mu.double() if shifted else h
    close = lambda got, want: bool((got.double() - want).norm() <= 2e-6 * want.norm())         # sums of a few float32 products
    for got in results:
        assert close(got[0], out) and close(got[1], new) and close(got[2], h if shifted else states[:few].double())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,heads,dim,left", [(1, 1, 8, 0), (5, 3, 64, 0), (300, 4, 24, 8), (7, 2, 20, 0), (3, 2, 30, 0), (4, 2, 64, 1)])
def test_gate_per_head(dtype, n, heads, dim, left):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(n + dim)
    width = heads * dim
    whole = torch.randn(n, left + width + 8, generator=g).to(dtype).to(DEV)
    gate = torch.randn(n, heads + 3, generator=g).to(dtype).to(DEV)[:, 1:1 + heads]
    before = whole.clone()
    ops.head_gate(whole[:, left:left + width], gate, heads, dim)
    x = before[:, left:left + width].double().reshape(n, heads, dim)
    want = (x * torch.sigmoid(gate.double())[:, :, None]).reshape(n, width)
    assert (whole[:, left:left + width].double() - want).norm() <= (1e-6 if dtype == torch.float32 else 4e-3) * want.norm()
    whole[:, left:left + width] = before[:, left:left + width]
    assert torch.equal(whole, before)
