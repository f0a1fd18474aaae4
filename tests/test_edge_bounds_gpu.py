"""Edge lists that name vertices outside the graph: an error, never an access outside the arrays."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [-1, 5000, 70_000, 1 << 40, -(1 << 40)])
@pytest.mark.parametrize("end", [0, 1])
@pytest.mark.parametrize("n", [5000, 70_000])
def test_vertices_outside_the_graph_are_refused(cuda, bad, end, n):
    import graphcuda_b200 as gc
    if 0 <= bad < n:
        return
    ei = torch.randint(0, n, (2, 20_000), generator=torch.Generator().manual_seed(1))
    good = gc.normalized_adjacency(ei.to(cuda), n)
    broken = ei.clone()
    broken[end, 777] = bad
    for reorder in (None, "degree"):
        with pytest.raises(RuntimeError, match="outside the graph"):
            gc.normalized_adjacency(broken.to(cuda), n, reorder=reorder)
    w = gc.gcn_norm(broken.to(cuda), n)
    assert bool(w[777].isnan()) and not bool(w[:777].isnan().any()) and not bool(w[778:].isnan().any())
    again = gc.normalized_adjacency(ei.to(cuda), n)  # the word is cleared for every list
    assert torch.equal(again.val, good.val) and torch.equal(again.col, good.col)
