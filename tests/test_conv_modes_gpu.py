"""The layer and the loss under torch's other modes: forward-mode differentiation is refused, tracing records a call."""
import pytest
import torch
import torch.autograd.forward_ad as fw

from oracle import gcn_oracle as O

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


class _Model(torch.nn.Module):
    def __init__(self, conv, adj):
        super().__init__()
        self.conv, self.adj = conv, adj

    def forward(self, x):
        return self.conv(x, self.adj)


@pytest.mark.parametrize("grad", [True, False])
def test_traced_layer_runs_on_new_inputs(cuda, grad):
    gc, A, adj, conv = _layer(cuda)
    X = [torch.randn(200, 24, generator=torch.Generator().manual_seed(i)).to(cuda) for i in range(3)]
    y = torch.randint(0, 8, (200,), device=cuda)
    with torch.set_grad_enabled(grad):
        layer = torch.jit.trace(_Model(conv, adj), (X[0],), check_trace=False)
        loss = torch.jit.trace(lambda z: gc.log_softmax_nll_loss(z, y, scale=1.0 / 200), (conv(X[0], adj).detach(),),
                               check_trace=False)
        for x in X:
            for leaf in (x, conv.weights, conv.bias):
                leaf.grad = None
            x.requires_grad_(grad)
            Y = conv(x, adj)
            expect = gc.log_softmax_nll_loss(Y, y, scale=1.0 / 200)
            junk = [torch.full_like(Y, float("nan")) for _ in range(4)]  # what fresh memory would hold
            del junk
            got_Y = layer(x)
            got = loss(got_Y)
            assert torch.equal(got_Y, Y) and torch.equal(got, expect)
            if grad:
                expect.backward()
                ref = [t.grad.clone() for t in (x, conv.weights, conv.bias)]
                for leaf in (x, conv.weights, conv.bias):
                    leaf.grad = None
                got.backward()
                assert all(torch.equal(a.grad, b) for a, b in zip((x, conv.weights, conv.bias), ref))
            pre = O.spmm(A, x.detach().cpu()) @ conv.weights.detach().cpu() + conv.bias.detach().cpu()
            assert O.rel_fro(got_Y, pre.clamp_min(0)) < 1e-5
