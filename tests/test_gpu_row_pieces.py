"""Rows on their way from a projection to the score kernels, in 16-byte pieces: rotation, unit norm per head, cache pages."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(shape, seed):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).to(DEV)


def _rotated(x, cs, off, dim):
    """x [n, heads, len] float64; cs [n, dim / 2, 2]."""
    out = x.clone()
    if dim:
        a, b = x[..., off:off + dim // 2], x[..., off + dim // 2:off + dim]
        c, s = cs[:, None, :, 0].double(), cs[:, None, :, 1].double()
        out[..., off:off + dim // 2], out[..., off + dim // 2:off + dim] = a * c - b * s, b * c + a * s
    return out


# a row of one head up to more than a block's threads, norms on both, one or none; values of their own columns or the keys as they came
@pytest.mark.parametrize("n,heads,kv,dim,rope", [(1, 32, 8, 64, 64), (3, 4, 2, 128, 64), (2, 3, 1, 16, 16), (5, 6, 3, 20, 8), (2, 96, 24, 128, 128)])
@pytest.mark.parametrize("norms", [(True, True), (False, True), (False, False)])
@pytest.mark.parametrize("own_values", [False, True])
def test_qk_norm_rope_cache(n, heads, kv, dim, rope, norms, own_values):
    from hfee_b200.kernels import ops
    page, eps = 16, 1e-5
    src = _rand((n, (heads + 2 * kv) * dim), 3)
    weights = [(1 + 0.1 * torch.randn(c * dim, generator=torch.Generator().manual_seed(4 + c))).to(DEV) if on else None
               for c, on in zip((heads, kv), norms)]
    cs = torch.randn(n, rope // 2, 2, generator=torch.Generator().manual_seed(9)).to(DEV)
    positions = torch.arange(n, dtype=torch.int32, device=DEV)
    slots = torch.zeros(n, dtype=torch.int32, device=DEV)
    table = torch.tensor([[1]], dtype=torch.int32, device=DEV)
    q = torch.empty(n, heads * dim, dtype=torch.bfloat16, device=DEV)
    k, v = (torch.zeros(2, kv, page, dim, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    ops.qk_norm_rope_cache(src, weights[0], weights[1], eps, cs, rope, positions, slots, q, k, v, table, page, heads, kv, dim,
                           (heads + kv) * dim if own_values else -1)
    x = src.double()
    for cols, count, weight, got in ((x[:, :heads * dim], heads, weights[0], q.double().reshape(n, heads, dim)),
                                     (x[:, heads * dim:(heads + kv) * dim], kv, weights[1], k[1].double().transpose(0, 1)[:n])):
        y = cols if weight is None else cols * torch.rsqrt((cols * cols).mean(-1, keepdim=True) + eps) * weight.double()
        want = _rotated(y.reshape(n, count, dim), cs, 0, rope)
        assert (got - want).norm() <= 4e-3 * want.norm()                        # rounded to bfloat16: 2^-9 an element
    raw = x[:, (heads + kv) * dim:] if own_values else x[:, heads * dim:(heads + kv) * dim]
    assert bool((v[1].double().transpose(0, 1)[:n] == raw.reshape(n, kv, dim)).all()) and bool((k[0] == 0).all())
