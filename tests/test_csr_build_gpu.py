"""gc_csr_count_unique / gc_csr_fill: a CSR from a sorted edge list, duplicates summed in input order."""
import pytest
import torch

from oracle import gcn_oracle as O

pytestmark = pytest.mark.gpu


def _build(cuda, row, col, w, M):
    from graphcuda_b200 import _lib
    L, E = _lib.lib(), row.numel()
    s = torch.cuda.current_stream().cuda_stream
    r, c, v = row.to(cuda), col.to(cuda), w.to(cuda)
    head = torch.empty(max(E, 1), dtype=torch.int32, device=cuda)
    nnz = torch.empty(1, dtype=torch.int64, device=cuda)
    wsb = L.gc_csr_build_workspace_bytes(E)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda)
    p = lambda t: t.data_ptr() if t.numel() else None  # noqa: E731
    assert L.gc_csr_count_unique(p(r), p(c), E, p(head), nnz.data_ptr(), ws.data_ptr(), wsb, s) == 0, L.gc_last_error()
    n = int(nnz.item())
    rowptr = torch.full((M + 1,), -1, dtype=torch.int32, device=cuda)
    ccol, val = torch.empty(max(n, 1), dtype=torch.int32, device=cuda), torch.empty(max(n, 1), device=cuda)
    assert L.gc_csr_fill(p(r), p(c), p(v), E, M, head.data_ptr(), rowptr.data_ptr(), ccol.data_ptr(), val.data_ptr(), s) == 0
    if E > 0:
        assert L.gc_csr_count_unique(p(r), p(c), E, p(head), nnz.data_ptr(), ws.data_ptr(), 0, s) == -4
    return rowptr.cpu(), ccol[:n].cpu(), val[:n].cpu()


@pytest.mark.parametrize("M,E,share", [(1, 1, 0.0), (7, 0, 0.0), (300, 255, 0.5), (300, 256, 0.9), (300, 257, 0.1), (5000, 70_001, 0.3)])
def test_sorted_edge_list_becomes_csr(cuda, M, E, share):
    """Structure exact; a duplicated entry is the sum of its weights in the order given, bit for bit."""
    g = torch.Generator().manual_seed(E)
    row, col = torch.randint(0, M, (E,), generator=g), torch.randint(0, M, (E,), generator=g)
    dup = int(E * share)
    if dup:
        at = torch.randint(0, E, (dup,), generator=g)
        row[:dup], col[:dup] = row[at], col[at]
    order = torch.argsort(row * M + col, stable=True)
    row, col = row[order], col[order]
    w = torch.randn(E, generator=g)
    expect_col, expect_val, counts = [], [], torch.zeros(M, dtype=torch.int64)
    last = None
    for r, c, v in zip(row.tolist(), col.tolist(), w):
        if last == (r, c):
            expect_val[-1] = expect_val[-1] + v
        else:
            expect_col.append(c)
            expect_val.append(v)
            counts[r] += 1
            last = (r, c)
    rowptr, ccol, val = _build(cuda, row, col, w, M)
    assert torch.equal(rowptr.long(), torch.cat([torch.zeros(1, dtype=torch.int64), counts.cumsum(0)]))
    assert ccol.tolist() == expect_col
    if expect_val:
        assert torch.equal(val.view(torch.int32), torch.stack(expect_val).view(torch.int32))


def test_the_scripts_preprocessing_from_these_steps(cuda):
    """Normalised weights, then this CSR: the bits of normalized_adjacency, which builds from keys instead."""
    from graphcuda_b200 import gcn_norm, normalized_adjacency, synth
    n = 5000
    ei = synth.symmetrize(synth.rmat_edges(13, n, 30_000, 3))
    loops = O.add_self_loops(ei, n)
    w = gcn_norm(loops.to(cuda), n).cpu()
    order = torch.argsort(loops[0] * n + loops[1], stable=True)
    rowptr, col, val = _build(cuda, loops[0][order], loops[1][order], w[order], n)
    adj = normalized_adjacency(ei.to(cuda), n)
    assert torch.equal(rowptr, adj.rowptr.cpu()) and torch.equal(col, adj.col.cpu())
    assert torch.equal(val.view(torch.int32), adj.val.cpu().view(torch.int32))
