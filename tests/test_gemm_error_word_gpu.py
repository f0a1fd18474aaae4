"""The device's word for tensor-core waits that ran out: what check_gemm_flag reads, whoever owns the workspace."""
import ctypes

import pytest
import torch


def test_null_pointer_is_refused():
    from graphcuda_b200 import _lib
    assert _lib.lib().gc_gemm_error_word(None) == -1


def _set_word(value):
    """Writes the word as a launch that gives up would (no wait is made to run out)."""
    from graphcuda_b200 import _lib
    word, src = ctypes.c_void_p(), torch.full((1,), value, dtype=torch.int64, device="cuda")
    assert _lib.lib().gc_gemm_error_word(ctypes.byref(word)) == 0
    assert _lib.lib().gc_narrow_i64_i32(src.data_ptr(), word, 1, torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.gpu
def test_recorded_steps_report_on_the_devices_word(cuda):
    """A recorded GEMM has a workspace of its own, in the graph's memory; its report must still reach the check that
    follows a replay, on whatever stream either runs, and survive the growth of the eager launches' scratch."""
    import graphcuda_b200 as gc
    from graphcuda_b200 import ops
    A, B = torch.randn(2048, 512, device=cuda), torch.randn(512, 1024, device=cuda)
    gc.gemm(A, B, precision="tf32x3")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = gc.gemm(A, B, precision="tf32x3")
    graph.replay()
    ops.check_gemm_flag(cuda)
    try:
        _set_word(1)
        graph.replay()
        with pytest.raises(RuntimeError, match="bounded wait"):
            ops.check_gemm_flag(cuda)
        gc.gemm(torch.randn(4096, 4096, device=cuda), torch.randn(4096, 512, device=cuda), precision="tf32x3")
        with torch.cuda.stream(torch.cuda.Stream()):
            with pytest.raises(RuntimeError, match="bounded wait"):
                ops.check_gemm_flag(cuda)
    finally:
        _set_word(0)
    graph.replay()
    ops.check_gemm_flag(cuda)
    ref = (A.double() @ B.double()).float()
    assert (out - ref).norm() / ref.norm() < 1e-4
