"""One adjacency used by several threads at once."""
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
