"""The row selection of a loss belongs to the forward call: changing it afterwards does not touch the gradient."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [7, 47, 130])
@pytest.mark.parametrize("dtype", [torch.bool, torch.uint8, torch.int64])
def test_selection_may_change_before_the_backward_pass(cuda, C, dtype):
    import graphcuda_b200 as gc
    M = 1001
    g = torch.Generator(device=cuda).manual_seed(C)
    Z = torch.randn(M, C, generator=g, device=cuda)
    y = torch.randint(0, C, (M,), generator=g, device=cuda)
    keep = torch.rand(M, generator=g, device=cuda) < 0.4
    mask = (keep * 3).to(dtype)  # any non-zero value selects
    ref = Z.detach().double().requires_grad_()
    torch.nn.functional.nll_loss(torch.log_softmax(ref, 1)[keep], y[keep]).backward()
    z = Z.clone().requires_grad_()
    loss = gc.log_softmax_nll_loss(z, y, mask, scale=1.0 / int(keep.sum()))
    mask.copy_(~keep)
    loss.backward()
    assert torch.allclose(z.grad.double(), ref.grad, rtol=1e-5, atol=1e-8)
    assert bool((z.grad[~keep] == 0).all())
