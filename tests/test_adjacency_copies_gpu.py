"""Adjacencies as objects: copies, pickles, and new values in place of the old ones."""
import copy
import io
import pickle

import pytest
import torch

from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


def _saved(x):
    b = io.BytesIO()
    torch.save(x, b)
    b.seek(0)
    return torch.load(b, weights_only=False)


@pytest.mark.parametrize("way", [copy.copy, copy.deepcopy, lambda x: pickle.loads(pickle.dumps(x)), _saved])
@pytest.mark.parametrize("kind", ["csr", "dense", "model"])
def test_copies_and_pickles(cuda, way, kind):
    import graphcuda_b200 as gc
    from graphcuda_b200.models import GCN
    A = random_csr(300, 300, 4.0, seed=1, long_rows=((3, 250),))
    A = (A + A.t()).coalesce()
    X = torch.randn(300, 24, device=cuda)
    adj = gc.DenseAdjacency(A.to_dense().to(cuda)) if kind == "dense" else to_gpu_csr(A, cuda)
    if kind == "csr":
        adj.segment, adj.perm = 256, torch.arange(300)
    model = GCN([24, 16, 7]).to(cuda)
    expect = model(X, adj)
    if kind == "model":
        model.adj = adj
        other_model = way(model)
        assert torch.equal(other_model(X, other_model.adj), expect)
        return
    other = way(adj)
    assert torch.equal(model(X, other), expect)
    assert other.symmetric and other.shape == adj.shape and other.device == adj.device
    if kind == "csr":
        assert other.nnz == adj.nnz and other.segment == 256 and torch.equal(other.perm, adj.perm)


def test_new_arrays_take_effect(cuda):
    import graphcuda_b200 as gc
    A = random_csr(300, 300, 4.0, seed=1, long_rows=((3, 250),))
    S = (A + A.t()).coalesce()
    H = torch.randn(300, 16, device=cuda)
    conv = gc.GCNConv(16, 24, apply_relu=False).to(cuda)
    adj, other = to_gpu_csr(S, cuda), to_gpu_csr(A, cuda)
    expect = adj.matmul(H)
    adj.val = adj.val * 2
    assert torch.equal(adj.matmul(H), 2 * expect) and adj.symmetric
    assert torch.allclose(conv(H, adj), adj.matmul(H) @ conv.weights, rtol=1e-4, atol=1e-4)
    adj.val = torch.arange(adj.nnz, device=cuda, dtype=torch.float32)
    assert not adj.symmetric
    for bad in (adj.val[:-1], adj.val.double(), adj.val.cpu()):
        with pytest.raises(RuntimeError):
            adj.val = bad
    shifted = (other.col + 1) % 300
    order = torch.argsort(torch.repeat_interleave(torch.arange(300, device=cuda), other.rowptr.diff()) * 300 + shifted)
    other.matmul(H)
    other.col = shifted[order].int()
    dense = torch.zeros(300, 300, device=cuda)
    rows = torch.repeat_interleave(torch.arange(300, device=cuda), other.rowptr.diff())
    dense[rows, other.col.long()] = other.val
    assert torch.allclose(other.matmul(H), dense @ H, rtol=1e-4, atol=1e-4)
    d = gc.DenseAdjacency(S.to_dense().to(cuda))
    y = conv(H, d)
    d.A = d.A * 2
    assert torch.allclose(conv(H, d), 2 * y, rtol=1e-4, atol=1e-5) and torch.allclose(d.matmul(H), 2 * expect, rtol=1e-4, atol=1e-5)
