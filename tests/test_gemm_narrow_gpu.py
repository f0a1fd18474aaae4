"""Products with few columns on CUDA cores, on both sides of every line between the narrow and the tiled kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = {
    "nn": [(m, n, k) for m in (1, 4736, 4737, 16_384, 16_385) for n in (1, 3, 8, 9, 16) for k in (15, 16, 127, 128, 1537)],
    "nt": [(m, n, k) for m in (5, 4736, 4737) for n in (7, 8, 9, 16) for k in (15, 16, 127, 128, 1537)],
    "tn": [(m, n, k) for m in (1, 31, 32, 33, 64, 65, 8192, 8193, 16_385) for n in (1, 8, 9, 16)
           for k in (15, 16, 63, 64, 128, 129, 1536, 1537, 2816, 2817)] +
          [(m, n, k) for m in (16, 64, 65, 128, 130) for n in (3, 8, 16) for k in (8192, 8193, 65_537)],
}


@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
def test_lines_between_the_kernels(cuda, layout):
    """Against float64 products; the error of an fp32 sum of K products in any order is at most (K + 1) / 2^24 of the sum
    of their magnitudes."""
    import graphcuda_b200 as gc
    g = torch.Generator(device=cuda).manual_seed(ord(layout[0]))
    for M, N, K in SIZES[layout]:
        A = torch.randn(K, M, generator=g, device=cuda).t() if layout[0] == "t" else torch.randn(M, K, generator=g, device=cuda)
        B = torch.randn(N, K, generator=g, device=cuda).t() if layout[1] == "t" else torch.randn(K, N, generator=g, device=cuda)
        bias = torch.randn(N, generator=g, device=cuda)
        got, mask = gc.gemm(A, B, bias=bias, relu=True, want_mask=True, precision="fp32_simt")
        pre = A.double() @ B.double() + bias.double()
        bound = (K + 2) / 2 ** 24 * (A.abs().double() @ B.abs().double() + bias.abs().double())
        clear = pre.abs() > bound
        assert bool((mask[clear] == (pre[clear] > 0).float()).all()), (M, N, K)
        assert bool(((got.double() - pre.clamp_min(0)).abs() <= bound).all()), (M, N, K)
