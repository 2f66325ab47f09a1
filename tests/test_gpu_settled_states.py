"""States read in front of the wait for the kernel before (a step whose states are settled): the same numbers, bit for bit, as behind it."""
import pytest
import torch

from test_gpu_dobelix_ops import make_step

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rule", ["linear", "channel", "gates", "step"])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (24, 40), (128, 96)])
@pytest.mark.parametrize("counts", [[1], [1, 1, 1, 1], [2, 1, 3]])
def test_same_numbers(rule, dim, vdim, counts):
    from hfee_b200.kernels import ops
    heads, n = 3, sum(counts)
    gen = torch.Generator(device=DEV).manual_seed(7)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV)
    buf = rand(n, heads * (2 * dim + vdim)).bfloat16()
    q, k, v = buf[:, :heads * dim], buf[:, heads * dim:2 * heads * dim], buf[:, 2 * heads * dim:]
    state, norm, top = rand(8, heads, dim, vdim), rand(8, heads, dim), rand(8, heads)
    decay, pre, bias = rand(heads).sigmoid(), rand(n, 2 * heads if rule == "gates" else heads * dim), rand(heads)
    size = rand(n, heads).bfloat16()
    results = []
    for settled in (False, True):
        step = make_step(counts, slots=[5, 0, 7, 2][:len(counts)])
        step.states_settled = settled
        S, N, M = state.clone(), norm.clone(), top.clone()
        out = torch.full((n, heads * vdim), float("nan"), device=DEV)
        if rule == "linear":
            ops.linear_attention(q, k, v, decay, S, step, out, heads, dim, vdim, "silu")
        elif rule == "step":
            ops.head_scan(v, k, q, size, bias, -decay, bias, S, step, out, heads, heads, dim, vdim)
        elif rule == "gates":
            ops.gated_recurrence(1, q, k, v, pre, None, 15.0, 0.1, S, step, out, heads, dim, vdim, True, N, M)
        else:
            ops.gated_recurrence(0, q, k, v, pre, None, 0.5, 0.1, S, step, out, heads, dim, vdim)
        results.append((out, S, N, M))
    assert torch.isfinite(results[0][0]).all() and not torch.equal(results[0][1], state)
    for a, b in zip(*results):
        assert torch.equal(a, b)
