"""Plans with a chosen segment length: what the no-allocation aggregation can still take."""
import pytest
import torch

from oracle import gcn_oracle as O
from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


def test_long_segments_fit_the_built_in_scratch(cuda):
    """2.5 M non-zeros in long rows, F = 256: the plan that products use needs more than the 8 MiB of built-in scratch
    and is refused; the plan of the default segment fits, beside the first one, and gives the product."""
    from graphcuda_b200 import _lib
    L = _lib.lib()
    A = random_csr(700, 9000, 4.0, seed=2, long_rows=tuple((2 * r, 8000) for r in range(320)))
    adj = to_gpu_csr(A, cuda)
    H = torch.randn(9000, 256, generator=torch.Generator().manual_seed(1)).to(cuda)
    expect = adj.matmul(H)
    Y = torch.full_like(expect, float("nan"))

    def noalloc(plan):
        return L.gc_spmm_csr_f32_noalloc(
            adj.rowptr.data_ptr(), adj.col.data_ptr(), adj.val.data_ptr(), 700, 9000, 256, H.data_ptr(), 256, None, 0,
            Y.data_ptr(), 256, None, None, plan.buf.data_ptr(), plan.n_pieces, plan.n_slots, plan.n_cut,
            torch.cuda.current_stream().cuda_stream)

    fast = adj.plan_for(256)
    assert L.gc_spmm_scratch_bytes(fast.n_slots, 256) > _lib.SPMM_STATIC_SCRATCH_BYTES
    assert noalloc(fast) == -4
    long = adj.plan_for(256, segment=L.gc_spmm_default_segment(adj.nnz))
    assert adj.plan_for(256).n_slots == fast.n_slots  # products keep theirs
    assert noalloc(long) == 0, L.gc_last_error()
    assert O.rel_fro(Y, O.spmm(A, H.cpu())) < 1e-5 and O.rel_fro(Y, expect) < 1e-5
