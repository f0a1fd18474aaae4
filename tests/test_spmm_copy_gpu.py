"""The aligned copy that odd widths are gathered from: bounded, and done without where memory is short."""
import pytest
import torch

from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("F", [1433, 2042])
def test_wide_matrices_are_copied_in_slabs(cuda, F):
    """300 K rows: the copy of the whole matrix would take 1.7 and 2.4 GB; at most 1 GiB is taken at a time, and the
    slabs, their remainders included, give what an aligned H gives, with every epilogue."""
    n = 300_000
    adj = to_gpu_csr(random_csr(n, n, 13.0, seed=F, long_rows=((7, 3000), (n - 1, 400)), empty_rows=(0, 9)), cuda)
    g = torch.Generator(device=cuda).manual_seed(F)
    wide = torch.randn(n, (F + 3) // 4 * 4, generator=g, device=cuda)
    H, bias = wide[:, :F].contiguous(), torch.randn(F, generator=g, device=cuda)
    pre = adj.matmul(wide)[:, :F] + bias
    adj.plan_for(F)
    Y = adj.matmul(H, bias=bias, relu=True)  # the scratch grows here
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    adj.matmul(H, bias=bias, relu=True, out=Y)
    assert torch.cuda.max_memory_allocated() - before <= (1 << 30)
    # sums of a row in another order: at most some 3000 terms, 1e-5 of the norm as elsewhere in these tests
    ref = pre * (pre > 0)
    assert ((Y - ref).norm() / ref.norm()).item() < 1e-5
    del Y
    Y = torch.ones(n, F, device=cuda)
    adj.matmul(H, accumulate_into=Y, gate=H)
    ref = (pre - bias + 1.0) * (H > 0)
    assert ((Y - ref).norm() / ref.norm()).item() < 1e-5


def test_without_room_for_the_copy_the_product_still_runs(cuda):
    n, F = 40_000, 4097
    adj = to_gpu_csr(random_csr(n, n, 14.0, seed=3), cuda)
    H, Y = torch.randn(n, F, device=cuda), torch.empty(n, F, device=cuda)
    expect = adj.matmul(H)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda).total_memory
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(n, F + 3, device=cuda)
        adj.matmul(H, out=Y)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert ((Y - expect).norm() / expect.norm()).item() < 1e-5
