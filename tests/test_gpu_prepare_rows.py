"""Attention preparation with biases and norms in whole 16-byte pieces: against float64, and against the general kernel on the same rows off
a 16-byte boundary."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 16


def _step(n, before):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(positions=i32([before + i for i in range(n)]), slot_of_token=i32([0] * n), n=n)


def _rotated(t, cs, rope, interleaved):
    """t [n, heads, dim], cs [n, rope / 2, 2], float64."""
    if not rope:
        return t
    a, b = ((t[..., 0:rope:2], t[..., 1:rope:2]) if interleaved else (t[..., :rope // 2], t[..., rope // 2:rope]))
    c, s = cs[:, None, :, 0], cs[:, None, :, 1]
    u, v = a * c - b * s, b * c + a * s
    turned = torch.stack([u, v], -1).flatten(-2) if interleaved else torch.cat([u, v], -1)
    return torch.cat([turned, t[..., rope:]], -1)


# one token, several, and so many that a block takes every fourth group of pieces; fewer pieces than a block has threads, and several
# blocks a token; a block that holds the last queries and the first keys
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [1, 13, 600])
@pytest.mark.parametrize("heads,kv,dim,vdim,rope,interleaved", [(4, 2, 16, 24, 16, True), (36, 4, 64, 64, 32, False), (40, 8, 64, 32, 64, False),
                                                              (3, 1, 8, 8, 0, False)])
@pytest.mark.parametrize("normed,biased,mix", [(True, True, True), (True, False, False), (False, True, False)])
def test_biases_and_norms(dtype, n, heads, kv, dim, vdim, rope, interleaved, normed, biased, mix):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(heads + n)
    rand = lambda *s: torch.randn(*s, generator=g)
    qc, kc, vc, before, eps = heads * dim, kv * dim, kv * vdim, 5, 1e-4
    x, first = rand(n, qc + kc + vc).to(dtype).to(DEV), rand(n, vc).to(dtype).to(DEV)
    biases = tuple(rand(c).to(DEV) if biased else None for c in (qc, kc, vc))
    weights = tuple((rand(c) + 1).to(DEV) if normed else None for c in (qc, kc))
    cs = rand(n, rope // 2, 2).to(DEV) if rope else None
    pages = -(-(before + n) // PAGE)
    order = torch.randperm(pages, generator=g)
    table = order.to(torch.int32).reshape(1, -1).to(DEV)
    step = _step(n, before)

    def run(src, q_out, write=True):
        pools = [torch.zeros(pages, kv, PAGE, d, dtype=dtype, device=DEV) for d in (dim, vdim)] if write else [None, None]
        mixing = mix and write
        ops.attention_prepare(src, 0, qc, qc + kc, heads, kv, dim, vdim, step, q_out, *pools, table, PAGE, cs, rope, interleaved,
                              biases, weights, eps, first if mixing else None, ops.VALUES_MIX if mixing else ops.VALUES_AS_THEY_ARE,
                              0.25 if mixing else 0.0)
        return q_out, pools
    q, pools = run(x, torch.empty(n, qc, dtype=dtype, device=DEV))
    d = lambda t: t.double()
    wq, wk, wv = (d(x[:, a:b]) + (d(t) if biased else 0) for a, b, t in zip((0, qc, qc + kc), (qc, qc + kc, qc + kc + vc), biases))
    if normed:
        wq, wk = (t / (t.pow(2).mean(1, keepdim=True) + eps).sqrt() * d(w) for t, w in zip((wq, wk), weights))
    wq, wk = (_rotated(t.reshape(n, -1, dim), None if cs is None else d(cs), rope, interleaved) for t in (wq, wk))
    if mix:
        wv = 0.25 * d(first) + 0.75 * wv
    at = torch.arange(before, before + n)
    page, inside = order[at // PAGE].to(DEV), (at % PAGE).to(DEV)
    tol = 2e-6 if dtype == torch.float32 else 4e-3             # float32 arithmetic; bfloat16 rounds the result
    close = lambda got, want: bool((d(got) - want).norm() <= tol * want.norm())
    assert close(q, wq.reshape(n, qc))
    assert close(pools[0][page, :, inside], wk) and close(pools[1][page, :, inside], wv.reshape(n, kv, vdim))
    # the general kernel: the same sums in another order
    wide = torch.zeros(n, qc + kc + vc + 1, dtype=dtype, device=DEV)
    wide[:, 1:] = x
    q2, pools2 = run(wide[:, 1:], torch.empty(n, qc, dtype=dtype, device=DEV))
    for got, want in zip((q, *pools), (q2, *pools2)):
        assert (d(got) - d(want)).norm() <= (1e-6 if dtype == torch.float32 else 2e-3) * d(want).norm()
    assert torch.equal(run(x, torch.empty(n, qc, dtype=dtype, device=DEV), write=False)[0], q)
    # queries that overwrite the projection they come from
    over = x.clone()
    q3, pools3 = run(over, over[:, :qc])
    for got, want in zip((q3, *pools3), (q2, *pools2)):
        assert (d(got) - d(want)).norm() <= (1e-6 if dtype == torch.float32 else 2e-3) * d(want).norm()
