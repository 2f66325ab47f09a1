"""CUDA-core attention whose keys go to eight parts in blocks of 32: scores of minus infinity, the parts' borders, and the two launch
forms (eight warps for few (token, head) pairs, two for many), which give the same bits."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 16


def _cache(keys, values, dtype):
    """Pools with one request's keys [n, kv, dim] on pages in another order than the positions'."""
    n, pages = len(keys), -(-len(keys) // PAGE)
    table = torch.stack([torch.full((pages,), -1), torch.randperm(pages, generator=torch.Generator().manual_seed(pages))]).to(torch.int32)
    pools = []
    for rows in (keys, values):
        pool = torch.zeros(pages, rows.shape[1], PAGE, rows.shape[2])
        for i in range(n):
            pool[table[1, i // PAGE].item(), :, i % PAGE] = rows[i]
        pools.append(pool.to(dtype).to(DEV))
    return pools[0], pools[1], table.to(DEV)


def _step(positions):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(positions=i32(positions), slot_of_token=i32([1] * len(positions)), n=len(positions), r=1,
                                 max_new=len(positions))


def _exact(q, k, v, positions, scale, window, keep, sink):
    """float64 [tokens, heads, value size]; a score of minus infinity weighs nothing."""
    group = q.shape[1] // k.shape[1]
    k, v = (t.double().repeat_interleave(group, 1) for t in (k, v))
    out = []
    for i, pos in enumerate(positions):
        seen = [j for j in range(pos + 1) if not window or j > pos - window or j < keep]
        s = torch.einsum("hd,jhd->hj", q[i].double(), k[seen]) * scale
        if sink is not None:
            s = torch.cat([s, sink.double()[:, None]], 1)
        p = torch.softmax(s, 1)[:, :len(seen)]
        out.append(torch.einsum("hj,jhd->hd", p, v[seen]))
    return torch.stack(out)


# one block and a key more, all eight parts and a block more; a window whose blocks start inside a page, with and without first
# positions; `hidden`: positions whose key scores minus infinity for every query, a whole part's block among them
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("length,window,keep,hidden", [
    (65, 0, 0, [64]), (96, 0, 0, list(range(32, 64))), (33, 0, 0, list(range(32))), (257, 0, 0, list(range(0, 32)) + [256]),
    (289, 0, 0, list(range(64, 96)) + list(range(256, 288))), (32, 0, 0, []), (33, 0, 0, []), (256, 0, 0, []), (257, 0, 0, []),
    (300, 70, 0, list(range(230, 262))), (300, 70, 5, [0, 1, 2, 3, 4]), (300, 45, 40, list(range(32)))])
@pytest.mark.parametrize("sunk", [False, True])
def test_scores_of_minus_infinity_weigh_nothing(dtype, length, window, keep, hidden, sunk):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(length + window + keep)
    heads, kv, dim, vdim = 4, 2, 20, 12                        # sizes that bfloat16 runs here too
    rand = lambda *s: torch.randn(*s, generator=g).to(dtype).float()
    q, k, v = rand(1, heads, dim), rand(length, kv, dim), rand(length, kv, vdim)
    q[..., 0] = (q[..., 0].abs() + 0.25).to(dtype).float()
    k[hidden, :, 0] = float("-inf")
    sink = torch.randn(heads, generator=g) if sunk else None
    kp, vp, table = _cache(k, v, dtype)
    out = torch.full((1, heads * vdim), float("nan"), dtype=dtype, device=DEV)
    ops.softmax_attention(q.reshape(1, -1).to(dtype).to(DEV), kp, vp, table, PAGE, _step([length - 1]), out, heads, kv, dim, vdim, dim ** -0.5,
                          window, None if sink is None else sink.to(DEV), 1.0, None, keep)
    want = _exact(q, k, v, [length - 1], dim ** -0.5, window, keep, sink).reshape(1, -1)
    # float32 sums of at most 300 terms; bfloat16 rounds the result
    assert (out.double().cpu() - want).norm() <= (1e-5 if dtype == torch.float32 else 4e-3) * want.norm()


# value sizes on both sides of the registers' 64, 128 and 256; more pairs than eight an SM, contexts past eight blocks of 32
@pytest.mark.parametrize("dim,vdim", [(32, 64), (20, 65), (64, 128), (8, 132), (64, 256), (64, 300)])
@pytest.mark.parametrize("window,keep,sunk,sigmoid", [(0, 0, False, False), (90, 40, True, False), (0, 0, False, True)])
def test_many_tokens_give_the_bits_of_one(dim, vdim, window, keep, sunk, sigmoid):
    from hfee_b200.kernels import ops
    if sigmoid:
        vdim = dim
    g = torch.Generator().manual_seed(dim + vdim + window)
    heads, kv, before = 8, 2, 310
    n = 8 * ops.sm_count() // heads + 37
    rand = lambda *s: torch.randn(*s, generator=g)
    q, k, v = rand(n, heads, dim), rand(before + n, kv, dim), rand(before + n, kv, vdim)
    sink = rand(heads) if sunk else None
    kp, vp, table = _cache(k, v, torch.float32)
    qd = q.reshape(n, -1).to(DEV)

    def run(rows):
        step, out = _step([before + i for i in rows]), torch.full((len(rows), heads * vdim), float("nan"), device=DEV)
        if sigmoid:
            ops.sigmoid_attention(qd[rows], kp, vp, table, PAGE, step, out, heads, kv, dim, dim ** -0.5)
        else:
            ops.softmax_attention(qd[rows], kp, vp, table, PAGE, step, out, heads, kv, dim, vdim, dim ** -0.5, window,
                                  None if sink is None else sink.to(DEV), 1.0, None, keep)
        return out
    whole = run(list(range(n)))
    picked = [0, 1, 9, 10, 41, 42, n // 2, n - 1]
    for i in picked:
        assert torch.equal(run([i])[0], whole[i]), i
    if not sigmoid:
        want = _exact(q[picked], k, v, [before + i for i in picked], dim ** -0.5, window, keep, sink).reshape(len(picked), -1)
        assert (whole[picked].double().cpu() - want).norm() <= 1e-5 * want.norm()
