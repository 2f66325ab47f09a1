"""The delta rule with one decay per head over portions of several tokens: tiles solved at once against the kernel that takes them one by
one (no workspace) and against float64."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _step(portions):
    cu = torch.tensor([0] + torch.tensor(portions).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    slots = torch.tensor([2 * i + 1 for i in range(len(portions))], dtype=torch.int32, device=DEV)
    return types.SimpleNamespace(cu_tokens=cu, slots=slots, r=len(portions), n=sum(portions), max_new=max(portions))


def _exact(q, k, v, b, a, a_log, dt_bias, s):
    unit = lambda x: x / (x.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k = unit(q) * q.shape[-1] ** -0.5, unit(k)
    beta, g = torch.sigmoid(b), torch.exp(-torch.exp(a_log) * torch.nn.functional.softplus(a + dt_bias))
    out = []
    for t in range(len(q)):
        s = s * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", s, k[t]))
        s = s + k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hdv,hd->hv", s, q[t]))
    return torch.stack(out), s


# portions around a tile of 16, single tokens beside longer ones; key sizes around 32 and 64 and not of whole 16 bytes; values
# around a group of 16 columns and too long for a tile's solution; a before b and after it; offsets off 16 bytes
@pytest.mark.parametrize("heads,groups,dim,vdim,portions", [(4, 2, 64, 64, [17, 1, 40]), (3, 1, 20, 17, [16, 15, 33]), (2, 2, 33, 8, [50]),
                                                            (2, 1, 128, 40, [31, 2]), (1, 1, 8, 3000, [18]), (1, 1, 8, 3200, [18])])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("a_first,shift,write", [(False, 0, True), (True, 3, False)])
def test_tiles_match_one_by_one(heads, groups, dim, vdim, portions, dtype, a_first, shift, write):
    from hfee_b200.kernels import ops
    g = torch.Generator().manual_seed(dim + vdim)
    rand = lambda *s: torch.randn(*s, generator=g)
    step = _step(portions)
    cols = 2 * groups * dim + heads * vdim
    qkv = rand(step.n, shift + cols + 5).to(dtype).to(DEV)
    ba = rand(step.n, 2 * heads + 3).to(dtype).to(DEV)
    b_off, a_off = (heads + 2, 1) if a_first else (0, heads)
    a_log, dt_bias = (rand(heads) - 1).to(DEV), rand(heads).to(DEV)
    state = rand(2 * len(portions) + 1, heads, dim, vdim).to(DEV) * 0.3
    ws = torch.empty(ops.channel_delta_workspace(step.r, step.n, heads, dim, vdim), device=DEV)
    offs = (shift, shift + groups * dim, shift + 2 * groups * dim)
    results = []
    for workspace in (ws, None):
        s, out = state.clone(), torch.full((step.n, heads * vdim), float("nan"), device=DEV)
        ops.delta_rule(qkv, *offs, ba, b_off, a_off, a_log, dt_bias, s, step, out, heads, groups, dim, vdim, write, workspace)
        ops.check_status()
        results.append((out, s))
    d = lambda t: t.double()
    q, k = (d(qkv[:, o:o + groups * dim]).reshape(-1, groups, dim).repeat_interleave(heads // groups, 1) for o in offs[:2])
    v = d(qkv[:, offs[2]:offs[2] + heads * vdim]).reshape(-1, heads, vdim)
    b, a = d(ba[:, b_off:b_off + heads]), d(ba[:, a_off:a_off + heads])
    for i, count in enumerate(portions):
        at = slice(int(step.cu_tokens[i]), int(step.cu_tokens[i]) + count)
        want, last = _exact(q[at], k[at], v[at], b[at], a[at], d(a_log), d(dt_bias), d(state[2 * i + 1]))
        for out, s in results:                  # float32 sums of up to 128 products, carried over up to 50 tokens
            assert (d(out[at]).reshape(want.shape) - want).norm() <= 1e-5 * want.norm()
            assert (d(s[2 * i + 1]) - (last if write else d(state[2 * i + 1]))).norm() <= 1e-5 * last.norm()
    for out, s in results:
        assert torch.equal(s[::2], state[::2])


def test_workspaces_of_every_size(monkeypatch):
    """A workspace of the size asked for takes the tiles; one for values of the keys' length runs longer values as one kernel; values
    too long for the tiles want none; less is refused."""
    from hfee_b200.kernels import ops
    heads, groups, dim, portions = 2, 1, 32, [20, 3]
    step = _step(portions)
    launches = []
    real = ops.count_launches
    monkeypatch.setattr(ops, "count_launches", lambda k: (launches.append(k), real(k)))

    def run(vdim, floats):
        g = torch.Generator().manual_seed(vdim)
        rand = lambda *s: torch.randn(*s, generator=g).to(DEV)
        qkv, ba, state = rand(step.n, 2 * groups * dim + heads * vdim), rand(step.n, 2 * heads), rand(4, heads, dim, vdim)
        out = torch.empty(step.n, heads * vdim, device=DEV)
        ws = torch.empty(floats, device=DEV) if floats else None
        launches.clear()
        ops.delta_rule(qkv, 0, groups * dim, 2 * groups * dim, ba, 0, heads, rand(heads), rand(heads), state, step, out, heads, groups, dim,
                       vdim, True, ws)
        ops.check_status()
        return out, state, sum(launches)
    size = lambda *v: ops.delta_rule_workspace(step.r, step.n, heads, groups, dim, *v)
    assert size() == size(dim) < size(100) and size(5000) == 0
    for vdim, floats, kernels in ((dim, size(), 2), (8, size(8), 2), (8, size(), 2), (100, size(100), 2), (100, size(), 1), (5000, size(), 1)):
        got, want = run(vdim, floats), run(vdim, 0)
        assert got[2] - want[2] == kernels - 1
        for a, b in zip(got[:2], want[:2]):
            assert torch.equal(a, b) if kernels == 1 else (a - b).norm() <= 2e-5 * b.norm()
    for vdim, floats in ((dim, size() - 1), (8, size(8) - 1), (100, size() - 1)):
        with pytest.raises(ops.KernelLibraryError):
            run(vdim, floats)


# many tiles, small and large keys, sizes that do not fill their rows
@pytest.mark.parametrize("dim,vdim,tokens", [(64, 64, 256), (256, 64, 200), (20, 17, 300)])
def test_decays_are_as_exact_as_one_by_one(dim, vdim, tokens):
    """Against 64 bits the tiles are no further off than the token-by-token kernel (whose error is 2 to 3e-7 here)."""
    from hfee_b200.kernels import ops
    heads, groups = 4, 2
    g = torch.Generator().manual_seed(dim)
    rand = lambda *s: torch.randn(*s, generator=g).to(DEV)
    step = _step([tokens])
    qkv, ba, state = rand(tokens, 2 * groups * dim + heads * vdim), rand(tokens, 2 * heads), rand(2, heads, dim, vdim) * 0.1
    a_log, dt_bias = torch.linspace(-4, 1, heads, device=DEV), torch.linspace(-3, 1, heads, device=DEV)
    d = lambda t: t.double()
    q, k = (d(qkv[:, o:o + groups * dim]).reshape(-1, groups, dim).repeat_interleave(heads // groups, 1) for o in (0, groups * dim))
    want = _exact(q, k, d(qkv[:, 2 * groups * dim:]).reshape(-1, heads, vdim), d(ba[:, :heads]), d(ba[:, heads:]), d(a_log), d(dt_bias),
                  d(state[1]))
    errors = []
    for workspace in (torch.empty(ops.delta_rule_workspace(1, tokens, heads, groups, dim, vdim), device=DEV), None):
        s, out = state.clone(), torch.empty(tokens, heads * vdim, device=DEV)
        ops.delta_rule(qkv, 0, groups * dim, 2 * groups * dim, ba, 0, heads, a_log, dt_bias, s, step, out, heads, groups, dim, vdim, True, workspace)
        ops.check_status()
        errors.append([float((d(got) - ref).norm() / ref.norm()) for got, ref in ((out.reshape(want[0].shape), want[0]), (s[1], want[1]))])
    assert max(errors[0]) <= 4e-7 and all(a <= 1.2 * b for a, b in zip(*errors)), errors


def test_decays_to_nothing():
    from hfee_b200.kernels import ops
    heads, dim, tokens = 2, 32, 40
    g = torch.Generator().manual_seed(1)
    rand = lambda *s: torch.randn(*s, generator=g).to(DEV)
    step = _step([tokens])
    qkv, ba, state = rand(tokens, 4 * dim + heads * dim), rand(tokens, 2 * heads), rand(2, heads, dim, dim)
    ba[3::7, heads:] = 80.0                                    # exp(-exp(88) * 80): the logarithm itself is minus infinity in 32 bits
    a_log, dt_bias = torch.tensor([0.5, 88.0], device=DEV), torch.zeros(heads, device=DEV)
    s, out = state.clone(), torch.empty(tokens, heads * dim, device=DEV)
    ops.delta_rule(qkv, 0, 2 * dim, 4 * dim, ba, 0, heads, a_log, dt_bias, s, step, out, heads, 2, dim, dim, True,
                   torch.empty(ops.delta_rule_workspace(1, tokens, heads, 2, dim), device=DEV))
    ops.check_status()
    d = lambda t: t.double()
    q, k, v = (d(qkv[:, o:o + 2 * dim]).reshape(tokens, 2, dim) for o in (0, 2 * dim, 4 * dim))
    want, last = _exact(q, k, v, d(ba[:, :heads]), d(ba[:, heads:]), d(a_log), d(dt_bias), d(state[1]))
    for got, ref in ((out.reshape(want.shape), want), (s[1], last)):
        assert (d(got) - ref).norm() <= 1e-6 * ref.norm()
