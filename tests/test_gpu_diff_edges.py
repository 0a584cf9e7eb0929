"""Diff assembly at the edges of its groups and units.

The data section is copied in 16-byte units whatever the chunk size and the buffer's alignment, and
region roots are collected 64 positions at a time, level by level: chunk sizes that no unit divides,
views at every alignment, group boundaries, and series long after their first checkpoint (source
buckets are relative to the last baseline) against the oracle, byte for byte
(src/tree_approach.cpp:511-710, src/list_approach.cpp:79-257).
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import ListDeduplicator, TreeDeduplicator, synth

pytestmark = pytest.mark.gpu


def compare(approach, cs, nbytes, offset, baselines, buf_id):
    import torch

    tree = approach == "tree"
    g = (TreeDeduplicator if tree else ListDeduplicator)(cs)
    o = (O.OracleTreeDeduplicator if tree else O.OracleListDeduplicator)(cs)
    s = synth.ByteSeries(nbytes, cs, lambda r, n: synth.plan_varied(r, n, 16), 21, buf_id=buf_id)
    mem = torch.zeros(nbytes + 64, dtype=torch.uint8, device="cuda")
    view = mem[offset:offset + nbytes]
    for k, base in enumerate(baselines):
        x = s.next()
        view.copy_(torch.from_numpy(np.ascontiguousarray(x)))
        assert g.checkpoint(view, bool(base)) == o.checkpoint(x, bool(base)), (approach, cs, nbytes, offset, k)
    g.close()
    o.close()


@pytest.mark.parametrize("approach", ["tree", "list"])
@pytest.mark.parametrize("offset", [0, 1, 4, 8, 15])
@pytest.mark.parametrize("cs", [1, 5, 16, 48, 100, 1000])
def test_units_and_alignments(cuda, approach, cs, offset):
    for n in (130, 1024):
        compare(approach, cs, n * cs - cs // 3, offset, [1, 0, 0], cs + offset)


@pytest.mark.parametrize("approach", ["tree", "list"])
@pytest.mark.parametrize("n", [31, 32, 33, 63, 64, 65, 16383, 16384, 16385, 40000])
def test_group_boundaries(cuda, approach, n):
    compare(approach, 64, n * 64, 0, [1, 0, 0, 0], n)


@pytest.mark.parametrize("approach", ["tree", "list"])
def test_many_checkpoints_after_a_late_baseline(cuda, approach):
    compare(approach, 128, 64 << 10, 0, [1] + [0] * 5 + [1] + [0] * 70, 7)
