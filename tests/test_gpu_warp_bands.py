"""The forest phases' lowest levels as warp tasks or as CTA bands, on trees of any chunk count.

The parameter warp_bands chooses per phase; the deepest level of a tree whose chunk count is no power
of two is partly filled, and a task then holds leaves of two levels (src/tree_approach.cpp:123-257,
379-503).  Byte for byte against the oracle, baselines and increments, single handles and batches.
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import CheckpointBatch, TreeDeduplicator, synth

pytestmark = pytest.mark.gpu
CS = 64
COUNTS = [129, 511, 513, 1025, 4095, 12345, 32769, 100001]


def series(n):
    return synth.ByteSeries(n * CS - 7, CS, lambda r, m: synth.plan_varied(r, m, 32), 17, buf_id=n)


@pytest.mark.parametrize("mask", [0, 1, 2, 3])
@pytest.mark.parametrize("n", COUNTS)
def test_single_handles(cuda, mask, n):
    import torch

    s, g, o = series(n), TreeDeduplicator(CS), O.OracleTreeDeduplicator(CS)
    g.set_param("warp_bands", mask)
    for k in range(4):
        x = s.next()
        assert g.checkpoint(torch.from_numpy(np.ascontiguousarray(x)).cuda(), k == 0) == o.checkpoint(x, k == 0), k
    g.close()
    o.close()


@pytest.mark.parametrize("mask", [0, 1, 2, 3])
def test_batches(cuda, mask):
    import torch

    ss = [series(n) for n in COUNTS]
    hs, os_ = [TreeDeduplicator(CS) for _ in COUNTS], [O.OracleTreeDeduplicator(CS) for _ in COUNTS]
    with CheckpointBatch() as b:
        b.set_param("warp_bands", mask)
        for k in range(4):
            xs = [s.next() for s in ss]
            b.checkpoint(hs, [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in xs], [k == 0] * len(hs))
            for n, h, o, x in zip(COUNTS, hs, os_, xs):
                assert bytes(h.copy_diff()) == o.checkpoint(x, k == 0), (k, n)
    for h, o in zip(hs, os_):
        h.close()
        o.close()
