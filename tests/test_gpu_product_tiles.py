"""Products of prompt portions: which kind of tile a shape takes, tiles of 192 columns by pairs of CTAs, and stores that leave by bulk
copies (whole and ragged edges, and outputs that no tensor map can describe)."""
import pytest
import torch

from hfee_b200.kernels import ops

DEV = "cuda:0"


def test_tile_choice_takes_the_kind_whose_rounds_take_least():
    choose = lambda m, n, pairs=True, store=False: ops.tile_choice(m, n, 148, pairs, store)
    assert choose(2048, 2048) == (True, 256)                       # 64 pair tiles, one round
    assert choose(564, 4096) == (True, 256)                        # 160 narrow tiles would be two rounds
    assert choose(1100, 4096) == (False, 256)                      # 80 pair tiles would be two rounds of 74
    assert choose(300, 2048) == (False, 128)                       # few tiles: the narrow ones take least
    assert choose(64, 16384) == (False, 128) and choose(128, 4096 * 8) == (False, 256)     # a pair would be half empty
    assert choose(2048, 3072, store=True) == (True, 192)
    assert choose(2048, 3072, pairs=False) == (False, 192)
    for m in (65, 129, 700, 2048):
        for n in (8, 192, 2048, 6656, 128256):
            pair, block = choose(m, n, store=True)
            assert block in (128, 192, 256) and (not pair or (m > 128 and block >= 192)) and (block != 192 or n % 192 == 0)


def test_tile_choice_weighs_the_split_by_k():
    choose = lambda m, n, k, **more: ops.tile_choice(m, n, 148, True, True, k, True, **more)
    assert choose(256, 768, 8192) == (False, 128)                  # 12 tiles in four pieces each; 4 pair tiles would run all of K
    assert choose(256, 3072, 4096) == (False, 128)                 # 48 tiles in three pieces each against 16 pair tiles
    assert choose(256, 3072, 2048) == (True, 192)                  # too short to be split
    assert choose(2048, 3072, 4096, narrow=False)[1] != 192
    assert ops.split_pieces(12, 8192, 148) == 4 and ops.split_pieces(74, 8192, 148) == 2 and ops.split_pieces(75, 8192, 148) == 1
    assert ops.split_pieces(12, 4032, 148) == 1 and ops.split_pieces(1, 4096, 148) == 4


def _case(m, n, k):
    g = torch.Generator().manual_seed(m + 3 * n + k)
    a = torch.randn(m, k, generator=g).to(torch.bfloat16).to(DEV)
    w = torch.randn(n, k, generator=g).to(torch.bfloat16).to(DEV)
    return a, w, a.double().cpu() @ w.double().cpu().t()


def _close(out, ref, rel):
    assert float((out.double().cpu() - ref).norm() / ref.norm()) < rel


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(256, 192, 64), (129, 384, 200), (300, 200, 72), (2048 + 7, 3072, 512)])
def test_pairs_on_tiles_of_192_columns(m, n, k):
    a, w, ref = _case(m, n, k)
    for dtype, rel in ((torch.float32, 1e-5), (torch.bfloat16, 4e-3)):       # sums of bfloat16 products in float32; their rounding
        out = torch.full((m, n), float("nan"), dtype=dtype, device=DEV)
        ops.gemm_tcgen05_pair(a, w, out, ops.EPI_STORE, 192)
        ops.check_status()
        _close(out, ref, rel)


@pytest.mark.gpu
@pytest.mark.parametrize("run", [lambda *x: ops.gemm_tcgen05(*x, block_n=128), lambda *x: ops.gemm_tcgen05(*x, block_n=256),
                                 ops.gemm_tcgen05_pair])
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (131, 40, 136), (333, 1000, 520), (64, 4, 8)])
@pytest.mark.parametrize("relu2", [False, True])
def test_stores_leave_nothing_beyond_the_matrix_and_take_any_pitch(run, m, n, k, relu2):
    a, w, ref = _case(m, n, k)
    ref = torch.relu(ref) ** 2 if relu2 else ref
    kinds = ((torch.bfloat16, 8e-3),) if relu2 else ((torch.float32, 1e-5), (torch.bfloat16, 4e-3))
    for dtype, rel in kinds:
        for left, pitch in ((0, n + 16), (8, n + 24), (1, n + 5)):     # the last: base and pitch that a bulk copy cannot take
            whole = torch.full((m + 3, (pitch + 7) // 8 * 8 if left != 1 else pitch), 7.0, dtype=dtype, device=DEV)
            run(a, w, whole[:m, left:left + n], ops.EPI_RELU2 if relu2 else ops.EPI_STORE)
            ops.check_status()
            _close(whole[:m, left:left + n], ref, rel)
            whole[:m, left:left + n] = 7.0
            assert bool((whole == 7.0).all())


@pytest.mark.gpu
def test_the_launch_splits_as_the_choice_expects():
    lib = ops.library()
    for m, n, k in ((128, 128, 4096), (256, 768, 8192), (65, 4736, 4104), (129, 4736, 4096), (512, 2048, 8192), (300, 5000, 4090), (100, 40, 64)):
        for bn in (128, 192, 256):
            tiles = -(-m // 128) * -(-n // bn)
            pieces = ops.split_pieces(tiles, k, ops.sm_count())
            assert lib.hfee_gemm_tcgen05_stream_k(m, n, k, bn, 1 << 40) == (tiles * pieces if pieces > 1 else 0)


@pytest.mark.gpu
def test_a_split_that_is_asked_for_is_made(monkeypatch):
    a, w, ref = _case(256, 384, 4096)
    assert ops.tile_choice(256, 384, ops.sm_count(), True, True, 2048) == (True, 192)
    monkeypatch.setattr(ops, "gemm_tcgen05_pair", None)
    for k in (2048, 4096):                                         # short and long enough for the split
        out = torch.empty(256, 384, device=DEV)
        ops.gemm_tcgen05(a[:, :k].contiguous(), w[:, :k].contiguous(), out, stream_k=True)
        ops.check_status()
        _close(out, ref if k == 4096 else a[:, :k].double().cpu() @ w[:, :k].double().cpu().t(), 1e-5)


@pytest.mark.gpu
def test_tiles_that_do_not_hold_whole_heads_are_refused():
    n, heads, dim, k = 300, 3, 128, 64
    a, w = (torch.zeros(r, k, dtype=torch.bfloat16, device=DEV) for r in (n, heads * dim))
    q, ints = torch.empty(n, heads * dim, dtype=torch.bfloat16, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    lib = ops.library()
    for block, pairs in ((192, 0), (192, 1), (128, 1), (64, 0)):
        assert lib.hfee_gemm_tcgen05_rope(a.data_ptr(), k, w.data_ptr(), k, n, heads * dim, k, None, ints.data_ptr(), ints.data_ptr(), q.data_ptr(),
                                          heads * dim, None, None, ints.data_ptr(), 1, 16, heads, 1, dim, 0, block, pairs, None,
                                          torch.cuda.current_stream().cuda_stream) != 0
