"""Tokens whose router scores are not numbers, and expert numbers out of range: every pair still goes to an expert that exists, and the
other tokens get what they get beside healthy ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAN = float("nan")


def _route(router, logits, experts, top):
    from hfee_b200.kernels import ops
    n = len(logits)
    choice, weight = torch.full((n, top), -7, dtype=torch.int32, device=DEV), torch.zeros((n, top), device=DEV)
    if router == "softmax":
        ops.moe_route(logits, top, 1.5, choice, weight)
    elif router == "groups":
        ops.moe_route_grouped(logits, experts, top, 4, 2, 1.5, choice, weight)
    else:
        ops.moe_route_chosen(logits, experts, top, 1.5, choice, weight)
    return choice, weight


# the last of four warps of a block and a block's only one; the last token's row ends the shared scores
@pytest.mark.parametrize("router", ["softmax", "groups", "chosen"])
@pytest.mark.parametrize("n", [5, 8])
def test_routers_choose_experts_that_exist(router, n):
    experts, top = 16, 3
    clean = torch.randn(n, experts, generator=torch.Generator().manual_seed(n)).to(DEV)
    logits = clean.clone()
    sick = [1, n - 1]
    logits[1] = NAN
    logits[n - 1, 2:] = NAN
    choice, weight = _route(router, logits, experts, top)
    assert bool(((choice >= 0) & (choice < experts)).all())
    healthy = [i for i in range(n) if i not in sick]
    want = _route(router, clean, experts, top)
    assert torch.equal(choice[healthy], want[0][healthy]) and torch.equal(weight[healthy], want[1][healthy])
    if router != "chosen":
        assert bool(weight[1].isnan().all())


def _experts(form, x, top, choice, gate, up, down):
    from hfee_b200.kernels import ops
    (n, width), (experts, inner, _), pairs = x.shape, gate.shape, x.shape[0] * top
    i32 = lambda size: torch.zeros(size, dtype=torch.int32, device=DEV)
    if form == "few":
        hidden, out = torch.zeros((pairs, inner), dtype=x.dtype, device=DEV), torch.full((pairs, width), 7.0, device=DEV)
        ops.moe_experts_few(x, top, choice, ops.interleave_gate_up(gate, up), down, 7.0, hidden, out)
        return out
    if form == "grouped":
        tiles = ops.moe_tiles_grouped(pairs, experts)
        rows = tiles * ops.GROUPED_TILE_ROWS
        place, out = i32(pairs), torch.full((rows, width), 7.0, device=DEV)
        ops.moe_experts_grouped(x, top, choice, ops.interleave_gate_up(gate, up), down, 7.0, place, i32(rows), i32(tiles),
                                torch.zeros((rows, width), dtype=x.dtype, device=DEV), None,
                                torch.zeros((rows, inner), dtype=x.dtype, device=DEV), out)
        ops.check_status()
        return out[place.long()]
    tiles = ops.moe_max_tiles(pairs, experts)
    offsets, order, tile_expert, tile_row = i32(experts + 1), i32(pairs), i32(tiles), i32(tiles)
    ops.moe_plan(choice, experts, offsets, order, tile_expert, tile_row)
    hidden, out = torch.zeros((pairs, inner), dtype=x.dtype, device=DEV), torch.full((pairs, width), 7.0, device=DEV)
    ops.moe_experts(x, top, gate, up, down, 7.0, offsets, order, tile_expert, tile_row, hidden, out)
    return out


@pytest.mark.parametrize("form", ["few", "grouped", "tiles"])
@pytest.mark.parametrize("n", [1, 7, 16])
def test_a_token_of_nan_and_numbers_out_of_range(form, n):
    experts, top, width, inner = 5, 2, 72, 24
    g = torch.Generator().manual_seed(n)
    rand = lambda *s: (torch.randn(*s, generator=g) * 0.3).bfloat16().to(DEV)
    x, gate, up, down = rand(n, width), rand(experts, inner, width), rand(experts, inner, width), rand(experts, width, inner)
    choice = torch.randint(0, experts, (n, top), generator=g, dtype=torch.int32).to(DEV)
    want = _experts(form, x, top, choice, gate, up, down)
    sick = x.clone()
    sick[n // 2] = NAN
    got = _experts(form, sick, top, choice, gate, up, down)
    rows = torch.arange(n * top, device=DEV) // top == n // 2
    assert torch.equal(got[~rows], want[~rows])
    wild = choice.clone()
    wild[0, 0], wild[n - 1, 1] = experts, -3
    tame = choice.clone()
    tame[0, 0], tame[n - 1, 1] = experts - 1, 0
    assert torch.equal(_experts(form, x, top, wild, gate, up, down), _experts(form, x, top, tame, gate, up, down))
