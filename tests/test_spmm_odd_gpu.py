"""Aggregation of matrices whose rows are not 16-byte aligned: odd widths, gaps between rows, few and many pieces."""
import pytest
import torch

from oracle import gcn_oracle as O
from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [5, 9, 11, 13, 17, 30, 33, 47, 50, 66, 101, 130, 259])
@pytest.mark.parametrize("n,deg", [(3000, 30.0), (90_000, 5.0)])
def test_odd_widths_are_padded(cuda, F, n, deg):
    import graphcuda_b200 as gc
    A = random_csr(n, n, deg, seed=F, long_rows=((7, 2500), (100, 300)), empty_rows=(0, 13, n - 1))
    g = torch.Generator().manual_seed(F)
    H, b = torch.randn(n, F, generator=g), torch.randn(F, generator=g)
    gate = torch.randn(n, F, generator=g)
    ref = O.spmm(A, H)
    adj = to_gpu_csr(A, cuda)
    Hg = H.to(cuda)
    assert O.rel_fro(adj.matmul(Hg), ref) < 1e-5
    pre = ref + b
    Y, mask = adj.matmul(Hg, bias=b.to(cuda), relu=True, want_mask=True, gate=gate.to(cuda))
    assert O.rel_fro(Y, pre * (pre > 0) * (gate > 0)) < 1e-5
    assert (mask.cpu() != (pre > 0).float()).float().mean() < 1e-4
    # a view of wider rows (used in place) whose pad holds NaN, and rows that start off a 16-byte boundary
    wide = torch.full((n, (F + 3) // 4 * 4), float("nan"), device=cuda)
    wide[:, :F] = Hg
    assert O.rel_fro(adj.matmul(wide[:, :F]), ref) < 1e-5
    off = torch.zeros(n, F + 6, device=cuda)
    off[:, 1:F + 1] = Hg
    assert O.rel_fro(adj.matmul(off[:, 1:F + 1]), ref) < 1e-5
    out = torch.full((n, F + 3), -1.0, device=cuda)
    adj.matmul(Hg, out=out[:, 1:F + 1])
    assert O.rel_fro(out[:, 1:F + 1], ref) < 1e-5 and bool((out[:, 0] == -1).all()) and bool((out[:, F + 1:] == -1).all())
