"""Edge list -> CSR at the vertex counts where the sort key changes width, with duplicates, without self-loops, relabelled:
bit for bit what the oracle builds."""
import pytest
import torch

from oracle import gcn_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 1000, 65_536, 65_537, 200_000])
@pytest.mark.parametrize("loops", [True, False])
@pytest.mark.parametrize("reorder", [None, "degree"])
def test_edges_to_csr(cuda, n, loops, reorder):
    import graphcuda_b200 as gc
    g = torch.Generator().manual_seed(n)
    E = 4 * n + 3
    ei = torch.randint(0, n, (2, E), generator=g)
    ei[:, :E // 8] = ei[:, E // 8:E // 8 * 2]  # duplicates
    ei[1, -1] = n - 1
    adj = gc.normalized_adjacency(ei.to(cuda), n, add_self_loops=loops, reorder=reorder)
    ref_ei = ei
    if reorder:
        deg = torch.bincount(ei[1], minlength=n)
        perm = torch.argsort(deg, descending=True, stable=True)
        assert torch.equal(adj.perm.cpu(), perm)
        inv = torch.empty_like(perm)
        inv[perm] = torch.arange(n)
        assert torch.equal(adj.inv_perm.cpu(), inv)
        ref_ei = inv[ei]
        assert all(torch.equal(a.cpu(), b) for a, b in zip(gc.degree_order(ei.to(cuda), n), (perm, inv)))
    if loops:
        A = O.normalized_adjacency_coo(ref_ei, n)
    else:
        A = torch.sparse_coo_tensor(ref_ei, O.gcn_norm(ref_ei, n), (n, n)).coalesce()
    row, col = A.indices()
    assert torch.equal(adj.col.cpu().long(), col)
    assert torch.equal(adj.val.cpu().view(torch.int32), A.values().view(torch.int32))
    rowptr = torch.zeros(n + 1, dtype=torch.int64)
    rowptr[1:] = torch.bincount(row, minlength=n).cumsum(0)
    assert torch.equal(adj.rowptr.cpu().long(), rowptr)
