"""The ReLU mask and the bias gradient from one pass, at vector and scalar widths and few and many rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 7, 130, 5000, 170_001])
@pytest.mark.parametrize("N", [1, 3, 4, 16, 47, 100, 256, 1030, 1433])
@pytest.mark.parametrize("relu", [True, False])
def test_bias_gradient(cuda, M, N, relu):
    from graphcuda_b200 import _lib
    if M * N > 60_000_000:
        pytest.skip("covered by the narrower widths")
    L = _lib.lib()
    g = torch.Generator(device=cuda).manual_seed(M + N)
    dY = torch.randn(M, N + 1, generator=g, device=cuda)[:, :N]  # rows with a gap
    dY = dY.contiguous() if N % 4 == 0 else dY
    Y = torch.randn(M, N, generator=g, device=cuda)
    G, db = torch.empty(M, N, device=cuda), torch.empty(N, device=cuda)
    wsb = L.gc_relu_bias_backward_workspace_bytes(M, N)
    ws = torch.empty(wsb, dtype=torch.uint8, device=cuda)
    args = (dY.data_ptr(), dY.stride(0), Y.data_ptr() if relu else None, N, G.data_ptr() if relu else None, N, M, N,
            db.data_ptr(), ws.data_ptr())
    s = torch.cuda.current_stream().cuda_stream
    assert L.gc_relu_bias_backward_f32(*args, wsb, s) == 0, L.gc_last_error()
    ref = dY * (Y > 0) if relu else dY
    if relu:
        assert torch.equal(G, ref)
    scale = ref.double().abs().sum(0) + 1e-30
    assert ((db.double() - ref.double().sum(0)).abs() / scale).max() < 1e-6
    assert L.gc_relu_bias_backward_f32(*args, 16, s) == -4 or wsb <= 256
