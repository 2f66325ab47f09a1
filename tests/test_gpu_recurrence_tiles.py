"""The gated recurrences in runs of 64 tokens, where values of more than 64 columns take 16 rows of four columns a thread, against the
walk token by token: outputs and states, both gates, both types."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# key sizes around groups of 16 rows, the smallest and the largest; values around 64, 128 and 256 columns; portions around a run and a
# stage of eight tokens, a single token beside them
@pytest.mark.parametrize("dim,vdim", [(5, 65), (16, 128), (33, 130), (128, 256), (256, 72), (64, 64)])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_runs_match_the_walk(dim, vdim, mode, dtype):
    from hfee_b200.kernels import ops
    heads, portions = 2, [129, 1, 70, 64]
    g = torch.Generator().manual_seed(dim * 3 + vdim + mode)
    rand = lambda *s: torch.randn(*s, generator=g)
    n, slots = sum(portions), [4, 0, 1, 3]
    cu = torch.tensor([0] + torch.tensor(portions).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    step = types.SimpleNamespace(cu_tokens=cu, slots=torch.tensor(slots, dtype=torch.int32, device=DEV), r=len(portions), n=n,
                                 max_new=max(portions))
    qk = heads * dim
    x = (rand(n, 2 * qk + heads * vdim + 3) * 0.7).to(dtype).to(DEV)
    cols = qk if mode == 0 else 2 * heads
    pre, bias = (rand(n, cols) * 2).to(DEV), (rand(cols) + (2 if mode == 0 else 0)).to(DEV)
    state, norm, top = (rand(5, heads, dim, vdim) * 0.3).to(DEV), (rand(5, heads, dim) * 0.3).to(DEV), rand(5, heads).to(DEV)
    results = []
    for ws in (None, torch.full((ops.gated_recurrence_workspace(len(portions), n, heads, dim, vdim),), float("nan"), device=DEV)):
        s, nn, m, out = state.clone(), norm.clone(), top.clone(), torch.full((n, heads * vdim), float("nan"), device=DEV)
        ops.gated_recurrence(mode, x[:, :qk], x[:, qk:2 * qk], x[:, 2 * qk:2 * qk + heads * vdim], pre.clone(), bias, 0.5 if mode == 0 else 6.0,
                             dim ** -0.5, s, step, out, heads, dim, vdim, True, nn if mode else None, m if mode else None, ws)
        results.append((out, s, nn, m))
    for got, want in zip(results[1], results[0]):          # the same float32 sums in another association
        assert (got.double() - want.double()).norm() <= 2e-5 * want.double().norm()
    assert torch.equal(results[1][1][2], state[2])         # a slot that is not in the batch
