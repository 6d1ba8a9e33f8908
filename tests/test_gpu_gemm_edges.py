"""The tcgen05 GEMM tile where its dispatch changes and where its column blocks end (bar of test_gemm_matches_fp32:
1e-5 of the largest entry against an FP32 product of the same BF16 operands; the sums differ in order only)."""
import pytest

pytestmark = pytest.mark.gpu


def _operands(M, N, K, seed):
    import torch
    gen = torch.Generator().manual_seed(seed)
    return (torch.randn(M, K, generator=gen).to(torch.bfloat16).cuda(),
            torch.randn(N, K, generator=gen).to(torch.bfloat16).cuda())


def _close(c, a, b):
    ref = a.float() @ b.float().T
    return ((c - ref).abs().max() / ref.abs().max()).item() <= 1e-5


@pytest.mark.parametrize("N", [16, 128, 240])
@pytest.mark.parametrize("kps", [448, 496, 512, 528, 544, 576, 1024])
def test_split_reduction_lengths(so, kps, N):
    """Reductions around 512 a split, multiples of 64, 32 and 16: every split's plane by itself, for one and three
    splits (64-wide slices in a ring of three from 512 on, for multiples of 64 and up to 128 columns)."""
    for splits in (1, 3):
        a, b = _operands(256, N, kps * splits, kps + splits)
        c = so.sur_gemm(a, b, splits=splits, layout=1)
        t = so.sur_gemm(a, b, splits=splits, layout=2)
        for z in range(splits):
            part = slice(z * kps, (z + 1) * kps)
            assert _close(c[z], a[:, part], b[:, part]) and _close(t[z].T, a[:, part], b[:, part])


@pytest.mark.parametrize("N", [48, 80, 112, 208])
def test_odd_multiples_of_16_columns(so, N):
    """A tile whose last column block is 16 wide: the product, and nothing written past it."""
    import torch
    a, b = _operands(256, N, 320, N)
    for layout in range(3):
        c = torch.full((256 * N + 256,), 7.0, device="cuda")
        torch.cuda.synchronize()
        assert so.lib().so_sur_gemm(a.data_ptr(), b.data_ptr(), None, c.data_ptr(), 256, N, 320, 1, layout) == 0
        p = c[:256 * N].view(N, 256).T if layout == 2 else c[:256 * N].view(256, N)
        assert _close(p, a, b) and bool((c[256 * N:] == 7.0).all())
