"""The native host side (csrc/host): scratch buffers under capture."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_recorded_steps_own_their_scratch(cuda):
    """Graphs recorded one after the other, the later ones needing more scratch: a recorded launch must not use (or
    copy from) a buffer that the next recording outgrows.  Replays equal the eager products."""
    import graphcuda_b200 as gc
    g = torch.Generator(device=cuda).manual_seed(0)
    graphs = []
    for k in (600, 2500, 9000):  # split-K products: scratch grows with the number of splits
        A, B = (torch.randn(s, generator=g, device=cuda) for s in ((64, k), (k, 48)))
        expect = gc.gemm(A, B)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            gc.gemm(A, B)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = gc.gemm(A, B)
        graphs.append((graph, out, expect, A, B))
    for _ in range(2):
        for graph, out, expect, _, _ in graphs:
            out.zero_()
            graph.replay()
            assert torch.equal(out, expect)


def test_errors_reach_python_as_runtime_errors(cuda):
    import graphcuda_b200 as gc
    with pytest.raises(RuntimeError, match="A.cols must match B.rows"):
        gc.gemm(torch.zeros(3, 4, device=cuda), torch.zeros(5, 2, device=cuda))
    with pytest.raises(RuntimeError, match="status"):
        gc.gemm(torch.zeros(8, 7, device=cuda), torch.zeros(7, 8, device=cuda), precision="tf32")
