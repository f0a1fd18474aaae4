"""Aggregation of 65 to 256 columns on graphs with few rows: both sides of the sizes where the mapping changes."""
import pytest
import torch

from oracle import gcn_oracle as O
from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [65, 68, 128, 131, 252, 256, 260])
@pytest.mark.parametrize("n,deg", [(40, 3.0), (1_500, 40.0), (9_000, 4.0), (20_000, 9.0), (45_000, 5.0)])
def test_wide_rows_of_small_graphs(cuda, F, n, deg):
    A = random_csr(n, n, deg, seed=F + n, long_rows=((7, min(n, 1200)), (20, min(n, 300))), empty_rows=(0, 13, n - 1))
    g = torch.Generator().manual_seed(F)
    H, b, gate = torch.randn(n, F, generator=g), torch.randn(F, generator=g), torch.randn(n, F, generator=g)
    ref = O.spmm(A, H)
    adj = to_gpu_csr(A, cuda)
    Hg = H.to(cuda)
    out = adj.matmul(Hg)
    assert O.rel_fro(out, ref) < 1e-5 and torch.equal(out, adj.matmul(Hg))
    pre = ref + b
    Y, mask = adj.matmul(Hg, bias=b.to(cuda), relu=True, want_mask=True, gate=gate.to(cuda))
    assert O.rel_fro(Y, pre * (pre > 0) * (gate > 0)) < 1e-5
    assert (mask.cpu() != (pre > 0).float()).float().mean() < 1e-4


@pytest.mark.parametrize("F", [52, 64, 65, 96, 130, 192, 200, 224, 256, 300, 384, 387, 512, 600, 1028])
def test_widths_of_larger_graphs(cuda, F):
    n = 90_000
    A = random_csr(n, n, 5.0, seed=F, long_rows=((7, 2500), (100, 300)), empty_rows=(0, 13, n - 1))
    g = torch.Generator().manual_seed(F)
    H, b, gate = torch.randn(n, F, generator=g), torch.randn(F, generator=g), torch.randn(n, F, generator=g)
    pre = O.spmm(A, H) + b
    Y = to_gpu_csr(A, cuda).matmul(H.to(cuda), bias=b.to(cuda), relu=True, gate=gate.to(cuda))
    assert O.rel_fro(Y, pre * (pre > 0) * (gate > 0)) < 1e-5


def test_many_pieces_of_48_columns(cuda):
    n = 240_000
    A = random_csr(n, n, 3.0, seed=1, long_rows=((7, 2500), (100, 300)), empty_rows=(0, 13, n - 1))
    H = torch.randn(n, 48, generator=torch.Generator().manual_seed(1))
    assert O.rel_fro(to_gpu_csr(A, cuda).matmul(H.to(cuda)), O.spmm(A, H)) < 1e-5


@pytest.mark.parametrize("F", [64, 96, 128, 184, 192, 256, 384, 512, 640, 1024])
def test_bf16_operand_widths(cuda, F):
    n = 20_000
    A = random_csr(n, n, 20.0, seed=F, long_rows=((7, 2500), (100, 300)), empty_rows=(0, 13, n - 1))
    H = torch.randn(n, F, generator=torch.Generator().manual_seed(F)).bfloat16()
    assert O.rel_fro(to_gpu_csr(A, cuda).matmul(H.to(cuda)), O.spmm(A, H.float())) < 1e-5
