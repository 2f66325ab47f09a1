"""The float32 product's kernels (16 rows of the weights a block, tiles, the general kernel) add in one order, segment by segment of 512:
every output element is the same bits whichever of them runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from hfee_b200.kernels import ops as o
    o.library()
    return o


def _shifted(t):
    """The same rows one float off a 16-byte boundary: only the general kernel takes them."""
    wide = torch.zeros(t.shape[0], t.shape[1] + 1, device=t.device)
    wide[:, 1:] = t
    return wide[:, 1:]


# token counts around every change of kernel (2, 4, 8, 16) and tile (32), widths around a warp's 16 rows and a
# tile's 64, depths below, at and past a piece, a segment (512) and a round of segments (2,048, 4,096)
@pytest.mark.parametrize("n,k", [(1, 4), (16, 60), (17, 64), (130, 100), (2500, 36), (300, 2052), (20000, 8), (40, 512), (40, 516),
                                 (48, 8200)])
def test_every_kernel_gives_the_same_bits(ops, n, k):
    g = torch.Generator().manual_seed(n + k)
    w = torch.randn(n, k, generator=g).cuda()
    for m in (1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 65, 129, 700):
        a = torch.randn(m, k, generator=g).cuda()
        plain = torch.empty(m, n, device="cuda")
        ops.gemm_simt(_shifted(a), _shifted(w), plain)
        # k additions of rounded products: at most (k + 1) 2^-24 of the sum of magnitudes
        ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
        assert ((plain.double() - ref).abs() <= (k + 1) * 2.0 ** -24 * size).all()
        out = torch.full((m, n + 3), 7.0, device="cuda")
        ops.gemm_simt(a, w, out[:, :n])
        assert torch.equal(out[:, :n], plain) and (out[:, n:] == 7.0).all(), m
        acc = torch.ones(m, n, device="cuda")
        ops.gemm_simt(a, w, acc, accumulate=True)
        assert torch.equal(acc, 1.0 + plain), m
        narrow = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        ops.gemm_simt(a, w, narrow)
        assert torch.equal(narrow, plain.bfloat16()), m


# depths on both sides of every change between the general kernel and the others, remainders of a piece and of a segment; token counts and
# widths whose tiles fit the chip once, twice and more, and whose 64 x 64 blocks do and do not
@pytest.mark.parametrize("k", [8, 64, 68, 252, 256, 512, 516, 764, 768, 1020, 1028, 1536])
@pytest.mark.parametrize("m,n", [(3, 70), (16, 1000), (17, 8200), (33, 8192), (285, 2048), (64, 130), (300, 5000)])
def test_short_sums_give_the_same_bits(ops, m, n, k):
    g = torch.Generator().manual_seed(m + n + k)
    a, w = torch.randn(m, k, generator=g).cuda(), torch.randn(n, k, generator=g).cuda()
    plain, out = torch.empty(m, n, device="cuda"), torch.full((m, n + 2), 7.0, device="cuda")
    ops.gemm_simt(_shifted(a), _shifted(w), plain)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert ((plain.double() - ref).abs() <= (k + 1) * 2.0 ** -24 * size).all()
    ops.gemm_simt(a, w, out[:, :n])
    assert torch.equal(out[:, :n], plain) and (out[:, n:] == 7.0).all()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_every_device_gives_the_kernels_their_shared_memory(ops):
    """The consent to more than 48 KB of shared memory is each device's own."""
    for m, k in ((2, 2048), (40, 2048)):
        a, w = torch.randn(m, k), torch.randn(64, k)
        got = []
        for device in ("cuda:0", "cuda:1"):
            with torch.cuda.device(device):
                out = torch.empty(m, 64, device=device)
                ops.gemm_simt(a.to(device), w.to(device), out)
                got.append(out.cpu())
        assert torch.equal(*got)
