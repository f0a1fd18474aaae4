"""Which operand the aggregation of the bf16 tier gathers, on both sides of every line of the rule."""
import pytest
import torch

from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,per_row,bf16_widths", [
    (3000, 20, (392, 512)), (20_000, 25, (136, 256, 392, 512)), (45_000, 24, (136, 256, 264, 384, 392, 512)),
    (60_000, 20, (128, 136, 256, 264, 384, 392, 512)), (60_000, 14, ())])
def test_either_side_of_the_lines(cuda, rows, per_row, bf16_widths):
    from graphcuda_b200 import _lib, ops
    adj = to_gpu_csr(random_csr(rows, rows, per_row, seed=rows, long_rows=((3, 1500),), empty_rows=(0,)), cuda)
    g = torch.Generator(device=cuda).manual_seed(per_row)
    for F in (120, 128, 132, 136, 256, 260, 264, 384, 392, 512):
        H = torch.randn(rows, F, generator=g, device=cuda)
        got = _lib.host.adj_matmul(adj._h, H, _lib.PREC_BF16)
        if F in bf16_widths:
            assert torch.equal(got, adj.matmul(ops.to_bf16(H)))
        else:
            assert torch.equal(got, adj.matmul(H))
