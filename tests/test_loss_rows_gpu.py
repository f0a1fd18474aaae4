"""The loss and evaluation kernels at the class counts where their lane mapping changes, rows aligned and not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C", [1, 2, 4, 15, 16, 17, 32, 33, 47, 64, 65, 128, 129, 300])
@pytest.mark.parametrize("gap", [0, 1, 4])
@pytest.mark.parametrize("M", [1, 37, 20_011])
def test_rows(cuda, C, gap, M):
    import graphcuda_b200 as gc
    g = torch.Generator(device=cuda).manual_seed(C * 10 + gap)
    ld = (C + 3) // 4 * 4 if gap == 4 else C + gap
    base = torch.full((M, ld), float("nan"), device=cuda)
    base[:, :C] = torch.randn(M, C, generator=g, device=cuda) * 4
    Z = base[:, :C].detach()
    y = torch.randint(0, C, (M,), generator=g, device=cuda)
    mask = torch.rand(M, generator=g, device=cuda) < 0.5
    mask[0] = True
    Zg = Z.clone() if gap == 0 else Z
    Zg = Zg.requires_grad_()
    loss = gc.log_softmax_nll_loss(Zg, y, mask)
    (grad,) = torch.autograd.grad(loss, Zg)
    Zr = Z.double().contiguous().requires_grad_()
    ref = torch.nn.functional.nll_loss(torch.log_softmax(Zr, 1)[mask], y[mask])
    (gref,) = torch.autograd.grad(ref, Zr)
    assert abs(float(loss) - float(ref)) < 1e-5 * max(1.0, float(ref))
    assert (grad - gref).norm() <= 1e-5 * gref.norm() + 1e-12
    if grad.stride(0) > C and M > 1:  # the padded gradient: zeros beyond the classes
        assert bool((grad.as_strided((M, grad.stride(0)), (grad.stride(0), 1))[:, C:] == 0).all())
    masks = [mask, ~mask, torch.ones(M, dtype=torch.uint8, device=cuda), mask.float()]
    pred, counts = gc.argmax_accuracy(Z, y, masks)
    assert torch.equal(pred, Z.contiguous().argmax(1))
    hit = pred == y
    for k, m in enumerate(masks):
        assert counts[k].tolist() == [int((hit & m.bool()).sum()), int(m.bool().sum())]
    assert gc.argmax_accuracy(Z, y)[1].tolist() == [[int(hit.sum()), M]]
