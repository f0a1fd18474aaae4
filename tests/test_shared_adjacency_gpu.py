"""One adjacency, or one stream, used by several threads at once."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _together(n, fn):
    """fn(i) in n threads that start at the same moment; their results."""
    barrier, out, errors = threading.Barrier(n), [None] * n, []

    def work(i):
        try:
            barrier.wait()
            out[i] = fn(i)
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    return out


def test_symmetry_is_found_once(cuda):
    from graphcuda_b200 import CSRAdjacency, _lib, normalized_adjacency, synth
    e = synth.symmetrize(synth.rmat_edges(14, 12_000, 60_000, 5)).to(cuda)
    base = normalized_adjacency(e, 12_000)
    L = _lib.lib()
    for _ in range(20):
        fresh = [CSRAdjacency(base.rowptr, base.col, base.val, base.shape) for _ in range(2)]
        before = L.gc_launch_count()
        assert fresh[0].symmetric
        once = L.gc_launch_count() - before
        before = L.gc_launch_count()
        assert all(_together(8, lambda i: fresh[1].symmetric))
        assert L.gc_launch_count() - before == once


def test_threads_on_one_stream_keep_their_scratch_apart(cuda):
    """Products of several launches that pass data through the stream's scratch (operand splits, partial sums of split
    sums and of cut rows), issued by several threads on the same stream: every result is the one issued alone."""
    import graphcuda_b200 as gc
    from tests.helpers import random_csr, to_gpu_csr
    g = torch.Generator(device=cuda).manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=g, device=cuda)  # noqa: E731
    adj = to_gpu_csr(random_csr(3000, 3000, 4.0, seed=1, long_rows=((5, 2500), (9, 2000))), cuda)
    work = []
    for i in range(6):
        A, B, C, H = rnd(256, 700 + 64 * i), rnd(700 + 64 * i, 33), rnd(1024, 640 + 128 * i), rnd(3000, 16 + 4 * i)
        D = rnd(640 + 128 * i, 512)
        work.append(lambda A=A, B=B, C=C, D=D, H=H: (gc.gemm(A, B, precision="fp32_simt"),
                                                     gc.gemm(C, D, precision="tf32x3"), adj.matmul(H)))
    alone = [w() for w in work]
    for i, got in enumerate(_together(len(work), lambda i: [work[i]() for _ in range(150)])):
        for r in got:
            assert all(torch.equal(x, y) for x, y in zip(r, alone[i]))
