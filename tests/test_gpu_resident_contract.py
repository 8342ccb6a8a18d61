"""What callers may rely on around the on-chip solvers: host threads with a context each,
ill-conditioned systems, routes that do not depend on earlier calls."""
import threading

import numpy as np
import pytest

from helpers import cgauss, hot_links, rel, to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "mixed"])
def test_host_threads_with_contexts_of_different_sizes(prec):
    """One context per host thread (qed2d.h): launches of the same kernel with different
    amounts of shared memory do not disturb one another.  Each call makes 61 solves from
    native code, so the threads' launches interleave; results are those of a single
    thread, bit for bit.  (All of these lattices are solved by one thread-block cluster.)"""
    import torch
    import qed2d
    qed2d.set_precision(prec)
    sizes, ns, calls = [(80, 80), (16, 16), (32, 32), (64, 64)], 60, 12

    def inputs(L1, L2):
        F = to_dev(cgauss(L1, L2, 5, 2))
        return (qed2d.rfield(L1, L2), to_dev(hot_links(L1, L2, 7)), qed2d.cfield(L1, L2), F, qed2d.cfield(L1, L2))

    def run(L1, L2):
        prm = qed2d.LattParm((L1, L2), 4.0)
        out = None
        for _ in range(calls):
            mom, U, X, F, g5DX = inputs(L1, L2)
            qed2d.leapfrog_(mom, U, X, F, g5DX, 2.0, 1e-3, ns, 1000, 1e-6, prm, None)
            assert out is None or np.array_equal(to_host(U), out)
            out = to_host(U)
        return out

    def thread(i, L1, L2):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got[i] = run(L1, L2)
                torch.cuda.current_stream().synchronize()
        except Exception as e:   # noqa: BLE001
            got[i] = e

    try:
        want = [run(*s) for s in sizes]
        got = [None] * len(sizes)
        threads = [threading.Thread(target=thread, args=(i, *s)) for i, s in enumerate(sizes)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        qed2d.set_precision("f64")
    for g, w in zip(got, want):
        assert isinstance(g, np.ndarray), repr(g)
        assert np.array_equal(g, w)
