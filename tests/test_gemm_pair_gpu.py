"""Tensor-core products on CTA pairs (256-row tiles): ragged rows, columns and k, every operand layout and epilogue,
against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (M, N, K, layout): last pair half or wholly empty, N over one and several tiles, k not a multiple of a stage;
# nn / nt with small and large B, tn split along k and not
SHAPES = [(19_000, 256, 100, "nn"), (18_945, 256, 256, "nn"), (38_000, 128, 36, "nn"), (19_001, 244, 64, "nt"),
          (9_600, 512, 48, "nt"), (4_096, 4_096, 520, "nn"), (5_000, 3_000, 1_100, "nt"), (300, 256, 60_000, "tn"),
          (2_560, 2_048, 1_000, "tn"), (257, 260, 40_000, "tn")]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("prec,tol", [("tf32x3", 1e-5), ("tf32", 2e-3), ("bf16", 1e-2)])
def test_pairs(cuda, shape, prec, tol):
    from graphcuda_b200 import gemm, ops
    M, N, K, layout = shape
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    A = torch.rand((K, M) if layout[0] == "t" else (M, K), generator=g, device=cuda) * 2 - 1
    B = torch.rand((N, K) if layout[1] == "t" else (K, N), generator=g, device=cuda) * 2 - 1
    A = A.t() if layout[0] == "t" else A
    B = B.t() if layout[1] == "t" else B
    if M % 4 and layout[0] == "t":
        A = torch.nn.functional.pad(A.t(), (0, 4 - M % 4))[:, :M].t()  # a pitch TMA can read
    ref = A.double() @ B.double()
    out = gemm(A, B, precision=prec)
    ops.check_gemm_flag(cuda)
    assert (out - ref).norm() / ref.norm() < tol * max(1.0, K / 2048 if K < 4000 else 1.5)
    assert torch.equal(out, gemm(A, B, precision=prec))
    rows = torch.cat([torch.arange(0, min(300, M)), torch.arange(max(0, M - 300), M)]).to(cuda)
    assert (out[rows] - ref[rows]).norm() / ref[rows].norm() < 3 * tol
    if prec == "tf32x3":
        bias, gate = torch.rand(N, generator=g, device=cuda) - 0.5, torch.rand(M, N, generator=g, device=cuda) - 0.5
        Y = gemm(A, B, bias=bias, relu=True, gate=gate, precision=prec)
        pre = ref + bias.double()
        assert (Y - pre * (pre > 0) * (gate > 0)).norm() / pre.norm() < 1e-4
        ops.check_gemm_flag(cuda)
