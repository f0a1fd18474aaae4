"""Tensor-core products whose last block of 32 columns is not full: vector stores where rows of C are aligned, whole rows
of scalars where they are not; nothing behind the last row is touched.  Against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [20, 35, 36, 47, 48, 60, 100, 129, 131, 252])
@pytest.mark.parametrize("M", [4_096, 20_001])
def test_ragged_columns(cuda, M, N):
    from graphcuda_b200 import gemm, ops
    g = torch.Generator(device=cuda).manual_seed(M + N)
    A, B = (torch.rand(*s, generator=g, device=cuda) * 2 - 1 for s in ((M, 132), (132, (N + 3) // 4 * 4)))
    B = B[:, :N]  # an odd N still has a pitch that TMA can read
    bias, gate = torch.rand(N, generator=g, device=cuda) - 0.5, torch.rand(M, N, generator=g, device=cuda) - 0.5
    ref = A.double() @ B.double()
    for prec, tol in (("tf32x3", 1e-5), ("tf32", 2e-3)):
        buf = torch.full((M * N + 64,), -7.0, device=cuda)
        C = buf[:M * N].view(M, N)
        gemm(A, B, out=C, precision=prec)
        ops.check_gemm_flag(cuda)
        assert (C - ref).norm() / ref.norm() < tol and bool((buf[M * N:] == -7).all())
    Y = gemm(A, B, bias=bias, relu=True, gate=gate, precision="tf32x3")
    pre = ref + bias.double()
    assert (Y - pre * (pre > 0) * (gate > 0)).norm() / pre.norm() < 1e-4
