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


# heads of one piece up to 32, lengths that are no power of two, a rotated part inside the head, values of another length; and sizes that
# are no whole pieces, which the other kernel takes
@pytest.mark.parametrize("n,heads,kv,length,vlen,rope,rope_off", [
    (1, 32, 8, 64, 64, 64, 0), (3, 4, 2, 96, 32, 32, 64), (130, 3, 1, 8, 256, 0, 0), (5, 2, 2, 256, 8, 16, 8), (2, 6, 3, 24, 40, 16, 8),
    (4, 2, 1, 20, 12, 8, 4), (3, 2, 1, 64, 64, 24, 0), (2, 1, 1, 320, 64, 64, 0)])
@pytest.mark.parametrize("eps", [None, 1e-5])
def test_rope_norm_cache(n, heads, kv, length, vlen, rope, rope_off, eps):
    from hfee_b200.kernels import ops
    page, pages = 16, 12
    cols = heads * length + kv * (length + vlen)
    src = _rand((n, cols + 8), 1)[:, :cols]
    cs = torch.randn(n, max(rope, 2) // 2, 2, generator=torch.Generator().manual_seed(2)).to(DEV) if rope else None
    positions = torch.arange(n, dtype=torch.int32, device=DEV) % page
    slots = torch.arange(n, dtype=torch.int32, device=DEV) // page
    table = torch.arange(pages, dtype=torch.int32, device=DEV).flip(0).reshape(pages, 1).contiguous()
    q = torch.full((n, heads * (length + 8)), 7.0, dtype=torch.bfloat16, device=DEV)
    k = torch.full((pages, kv, page, length + 8), 7.0, dtype=torch.bfloat16, device=DEV)
    v = torch.full((pages, kv, page, vlen), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.rope_norm_cache(src, cs, rope, eps, positions, slots, table, page,
                        q=(heads, 0, length, length, rope_off, q, 8, length + 8),
                        k=(kv, heads * length, length, length, rope_off, k, 8), v=(heads * length + kv * length, vlen, vlen, v))
    x = src.double()

    def want(block):
        y = _rotated(block, cs, rope_off, rope)
        return y if eps is None else y * torch.rsqrt((y * y).mean(-1, keepdim=True) + eps)
    want_q = want(x[:, :heads * length].reshape(n, heads, length))
    want_k = want(x[:, heads * length:heads * length + kv * length].reshape(n, kv, length))
    want_v = x[:, heads * length + kv * length:].reshape(n, kv, vlen)
    at = table[slots.long(), 0].long()
    got_q = q.double().reshape(n, heads, length + 8)
    got_k, got_v = (t.double()[at, :, positions.long()] for t in (k, v))
    assert (got_q[..., 8:] - want_q).norm() <= 4e-3 * want_q.norm() and bool((got_q[..., :8] == 7.0).all())      # rounded to bfloat16
    assert (got_k[..., 8:] - want_k).norm() <= 4e-3 * want_k.norm() and bool((got_k[..., :8] == 7.0).all())
    assert bool((got_v == want_v).all())
    assert int((v[..., 0] != 7.0).sum()) <= n * kv                               # nothing beside the tokens' places


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
