"""Gram-Schmidt columns and whole Lanczos runs of two bases on two streams, from two threads at once.

Both kinds of launch wait for all their CTAs at barriers inside the kernel, so they rely on every CTA of a launch
being resident however launches of the two streams overlap.  The results are those of each basis by itself, bit
for bit (fixed orders of all sums).  A run column by column, a run of one CTA per SM and a run of one cluster, each
against each.
"""
import threading

import numpy as np
import pytest

from slepc_b200 import problems as P

pytestmark = pytest.mark.gpu


class Run:
    """Lanczos columns 0..m of a grid Laplacian."""

    def __init__(self, b200, n, m, stream):
        csr = P.laplacian_2d(n // 50, 50)
        self.A = b200.Mat().createAIJ(csr, stream=stream)
        self.m, self.v0 = m, P.start_vector(len(csr[0]) - 1, 2)
        self.bv = b200.BV().create(len(csr[0]) - 1, m + 1, stream=stream)

    def run(self, times):
        self.bv.setColumn(0, self.v0)
        self.bv.orthonormalizeColumn(0)
        for _ in range(times):  # each gives the same columns
            self.bv.matLanczos(self.A, 0, self.m)
        return self.bv.getColumns()


# rows and last column: 24 cooperative launches, one launch on all SMs, one cluster
KINDS = {"columns": (400_000, 24), "chip": (40_000, 30), "cluster": (10_000, 20)}


@pytest.mark.parametrize("first,second", [("columns", "columns"), ("columns", "chip"), ("columns", "cluster"),
                                          ("chip", "chip"), ("chip", "cluster"), ("cluster", "cluster")])
def test_two_streams_at_once(b200, first, second):
    import torch

    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    work = []
    for kind, s in zip((first, second), streams):
        work.append(Run(b200, *KINDS[kind], s.cuda_stream))
    alone = [w.run(1) for w in work]
    got, errors = [[], []], []
    start = threading.Barrier(2)

    def body(i):
        try:
            start.wait(timeout=60)
            for _ in range(3):
                got[i].append(work[i].run(40))
        except Exception as e:  # a bounded wait that ran out, or any other status
            errors.append(e)

    threads = [threading.Thread(target=body, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for i in range(2):
        for g in got[i]:
            np.testing.assert_array_equal(g, alone[i])
