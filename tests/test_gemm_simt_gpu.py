"""fp32 CUDA-core products at the edges of their tiles, splits and dispatch rules, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K): each tile shape with a remainder, one cluster split, long sums with partial tiles; the narrow kernels at
# the ends of their ranges (8 / 9 / 16 / 17 columns, k just below and above a chunk of 1536, few and many rows)
SHAPES = [(65, 9, 70), (63, 33, 129), (129, 130, 35), (200, 65, 1000), (40, 40, 9001), (16, 17, 20_000),
          (5, 8, 127), (5, 8, 128), (701, 16, 1537), (2500, 7, 200), (1300, 13, 333), (3, 1, 4000), (33, 5, 64),
          (32, 16, 65), (600, 10, 900), (8193, 3, 70), (16_385, 16, 130), (1, 1, 1)]


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("shape", SHAPES)
def test_edges(cuda, shape, layout):
    from graphcuda_b200 import gemm
    M, N, K = shape
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    A = torch.rand((K, M) if layout[0] == "t" else (M, K), generator=g, device=cuda) * 2 - 1
    B = torch.rand((N, K) if layout[1] == "t" else (K, N), generator=g, device=cuda) * 2 - 1
    A = A.t() if layout[0] == "t" else A
    B = B.t() if layout[1] == "t" else B
    ref = A.double() @ B.double()
    scale = (A.double().abs() @ B.double().abs()).clamp_min(1e-30)
    out = gemm(A, B, precision="fp32_simt")
    assert ((out - ref).abs() / scale).max() < 2e-6
    assert torch.equal(out, gemm(A, B, precision="fp32_simt"))
    # the fused epilogue, written transposed
    bias = torch.rand(N, generator=g, device=cuda) - 0.5
    gate = torch.rand(N, M, generator=g, device=cuda) - 0.5
    pre = ref + bias.double()
    Y, mask = gemm(A, B, bias=bias, relu=True, want_mask=True, transposed_out=True, gate=gate, precision="fp32_simt")
    sure = (pre.abs() > 1e-5 * (scale + 1)).t()
    assert torch.equal(mask[sure], (pre > 0).float().t()[sure])
    expect = (pre * (pre > 0)).t() * (gate > 0)
    assert ((Y - expect).abs() / (scale.t() + 1)).max() < 1e-5


def test_views_with_gaps(cuda):
    """Row pitches larger than the rows, aligned and not."""
    from graphcuda_b200 import gemm
    g = torch.Generator(device=cuda).manual_seed(1)
    for pa, pb, n in ((64, 24, 20), (61, 23, 16), (64, 16, 16), (200, 100, 90)):
        A = torch.rand(300, pa + 3, generator=g, device=cuda)[:, 1:pa]
        B = torch.rand(pa - 1, pb, generator=g, device=cuda)[:, :min(n, pb)]
        ref = A.double() @ B.double()
        assert (gemm(A, B, precision="fp32_simt") - ref).norm() / ref.norm() < 1e-6
