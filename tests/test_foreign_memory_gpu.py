"""Host tensors, and tensors of another size or type, where a kernel would be given their pointer: refused."""
import pytest
import torch

from tests.helpers import random_csr, to_gpu_csr

pytestmark = pytest.mark.gpu


def test_products_refuse_host_memory(cuda):
    import graphcuda_b200 as gc
    from graphcuda_b200 import ops
    A, B = torch.randn(40, 32, device=cuda), torch.randn(32, 16, device=cuda)
    host = torch.zeros(40, 16)
    adj = to_gpu_csr(random_csr(40, 40, 3.0, seed=1), cuda)
    H = torch.randn(40, 16, device=cuda)
    A16, B16 = ops.to_bf16(A), ops.to_bf16(B, transpose=True)
    for call in (gc.gemm, lambda a, b, **k: ops.gemm_bf16_operands(A16, B16, **k), lambda a, b, **k: adj.matmul(H, **k)):
        for bad in (dict(out=host), dict(gate=host), dict(bias=torch.zeros(16)), dict(out=torch.zeros(40, 16, device=cuda).double())):
            with pytest.raises(RuntimeError):
                call(A, B, **bad)
    with pytest.raises(RuntimeError):
        adj.matmul(H, accumulate_into=host)
    with pytest.raises(RuntimeError):
        ops.gemm_bf16_operands(A16, B16.cpu())
    for fn in (ops.relu_backward, ops.mask_mul):
        for bad in (host, host.to(cuda).double(), host.to(cuda)[0]):
            with pytest.raises(RuntimeError):
                fn(H, bad)
    with pytest.raises(RuntimeError):
        gc.CSRAdjacency(adj.rowptr, adj.col, adj.val.cpu(), adj.shape)


def test_loss_layer_and_optimizers_refuse_host_memory(cuda):
    import graphcuda_b200 as gc
    Z, y = torch.randn(40, 7, device=cuda), torch.zeros(40, dtype=torch.int64, device=cuda)
    for labels, mask in ((y.cpu(), None), (y, torch.ones(40, dtype=torch.bool))):
        with pytest.raises(RuntimeError):
            gc.log_softmax_nll_loss(Z, labels, mask, scale=1.0)
    adj = to_gpu_csr(random_csr(40, 40, 3.0, seed=1), cuda)
    with pytest.raises(RuntimeError):
        gc.GCNConvFunction.apply(Z, adj, torch.randn(7, 5, device=cuda), True, torch.zeros(5))
    p = torch.nn.Parameter(torch.zeros(4, 6, device=cuda))
    p.grad = torch.ones(4, 6, device=cuda)
    for bad in (torch.zeros(4, 6), torch.zeros(4, 5, device=cuda), torch.zeros(6, 4, device=cuda).t(),
                torch.zeros(4, 6, device=cuda).double()):
        opt = gc.FusedAdam([p], lr=0.1)
        opt.state[p]["exp_avg"], opt.state[p]["exp_avg_sq"] = torch.zeros_like(p), bad
        with pytest.raises(RuntimeError):
            opt.step()
    assert bool((p == 0).all())
