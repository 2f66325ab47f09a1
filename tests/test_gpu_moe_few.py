"""Routed experts of a step of few (token, choice) pairs, and the weighted sum in whole and single columns."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rand(shape, seed, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype).to(DEV)


# one pair and the most there may be; depths and widths that end inside a piece of 32 and a tile of 16 rows; one expert for all (four
# times eight pairs), every token with every expert, more experts than pairs
@pytest.mark.parametrize("n,top,experts,width,inner", [(1, 1, 1, 8, 8), (1, 2, 16, 2048, 2048), (3, 2, 16, 72, 24), (32, 1, 1, 40, 8),
                                                       (5, 5, 5, 264, 56), (16, 2, 64, 520, 1032), (9, 3, 4, 1032, 96)])
@pytest.mark.parametrize("limit,alpha,shift", [(7.0, 1.702, 1.0), (float("inf"), 1.0, 0.0)])
def test_few_pairs(n, top, experts, width, inner, limit, alpha, shift):
    from hfee_b200.kernels import ops
    wide = _rand((n, width + 8), 1)
    x = wide[:, :width]                                        # rows with a pitch of their own
    gate, up = _rand((experts, inner, width), 2, 0.1), _rand((experts, inner, width), 3, 0.1)
    down = _rand((experts, width, inner), 4, 0.1)
    g = torch.Generator().manual_seed(n + experts)
    choice = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(n)]).to(torch.int32).to(DEV)
    hidden = torch.full((n * top, inner), float("nan"), dtype=torch.bfloat16, device=DEV)
    out = torch.full((n * top + 1, width), 7.0, dtype=torch.float32, device=DEV)
    ops.moe_experts_few(x, top, choice, ops.interleave_gate_up(gate, up), down, limit, hidden, out[:-1], alpha, shift)
    for t in range(n):
        for k in range(top):
            e = int(choice[t, k])
            a, b = gate[e].double() @ x[t].double(), up[e].double() @ x[t].double()
            a, b = a.clamp(max=limit), b.clamp(-limit, limit)
            want = a * torch.sigmoid(alpha * a) * (b + shift)
            got = hidden[t * top + k].double()
            assert (got - want).norm() <= 4e-3 * want.norm()                              # rounded to bfloat16: 2^-9 an element
            y = down[e].double() @ got
            assert (out[t * top + k].double() - y).norm() <= 1e-5 * y.norm() + 1e-6       # float32 sums
    assert bool((out[-1] == 7.0).all())


@pytest.mark.parametrize("n,top,width", [(1, 1, 4), (3, 2, 2048), (2, 6, 1030), (5, 9, 12), (300, 2, 1028), (70000, 1, 8), (66000, 2, 5)])
@pytest.mark.parametrize("accumulate,extra,placed", [(False, False, False), (True, True, True), (True, False, True), (False, True, False)])
def test_weighted_sum(n, top, width, accumulate, extra, placed):
    from hfee_b200.kernels import ops
    pairs = n * top
    rows = pairs + 5 if placed else pairs
    pair_out, weight = _rand((rows, width), 5, dtype=torch.float32), _rand((n, top), 6, dtype=torch.float32)
    place = torch.randperm(rows, generator=torch.Generator().manual_seed(7))[:pairs].to(torch.int32).to(DEV) if placed else None
    more = _rand((n, width), 8, dtype=torch.float32) if extra else None
    share = _rand((n, 24), 9, dtype=torch.float32)[:, 16:17] if extra else None
    y = _rand((n, width), 10, dtype=torch.float32)
    want = y.double() if accumulate else torch.zeros(n, width, dtype=torch.float64, device=DEV)
    if extra:
        want = want + torch.sigmoid(share.double()) * more.double()
    at = place.long() if placed else torch.arange(pairs, device=DEV)
    want = want + (pair_out[at].double().reshape(n, top, width) * weight.double()[:, :, None]).sum(1)
    ops.moe_combine(pair_out, weight, y, accumulate, place, more, share)
    assert (y.double() - want).norm() <= 1e-6 * want.norm()
