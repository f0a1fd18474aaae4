"""The layer under torch's other modes: forward-mode differentiation is refused."""
import pytest
import torch
import torch.autograd.forward_ad as fw

pytestmark = pytest.mark.gpu


def _layer(cuda, n=200, fin=24, fout=8):
    import graphcuda_b200 as gc
    from tests.helpers import random_csr, to_gpu_csr
    A = random_csr(n, n, 4.0, seed=1)
    torch.manual_seed(0)
    return gc, A, to_gpu_csr(A, cuda), gc.GCNConv(fin, fout, apply_relu=True, bias=True).to(cuda)


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("which", ["input", "weights", "bias"])
def test_forward_mode_is_refused_not_dropped(cuda, which, grad):
    """There is no forward-mode rule: a tangent must raise, also where nothing requires a gradient."""
    gc, _, adj, conv = _layer(cuda)
    t = dict(input=torch.randn(200, 24, device=cuda), weights=conv.weights.detach(), bias=conv.bias.detach())
    with fw.dual_level():
        t = {k: (fw.make_dual(v, torch.ones_like(v)) if k == which else v).requires_grad_(grad) for k, v in t.items()}
        with pytest.raises(RuntimeError, match="jvp"):
            gc.GCNConvFunction.apply(t["input"], adj, t["weights"], True, t["bias"])
