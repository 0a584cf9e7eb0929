"""Which baselines are built in bulk, and chunk sizes under 64 bytes among them.

A bulk baseline makes more launches than the increment after it, whose launches are those of a baseline
that inserts its digests one by one.  Trees of more than 256 table ranges take two passes, whose entries
fit the diff buffer from 64-byte chunks on.
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import ListDeduplicator, TreeDeduplicator
from reproducibility_icpp23_scalable_gpu_deduplication_b200.tree import HASH_MD5, HASH_MURMUR3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approach,n,cs,bulk", [
    ("tree", (1 << 15) - 1, 64, False), ("tree", 1 << 15, 64, True), ("tree", 1 << 15, 20, False),
    ("tree", 1 << 15, 24, True), ("tree", 1 << 19, 32, True), ("tree", (1 << 19) - 999, 48, True),
    ("tree", (1 << 19) + 12345, 48, False), ("tree", (1 << 19) + 12345, 64, True),
    ("list", (1 << 19) - 1, 64, False), ("list", 1 << 19, 64, True), ("list", (1 << 19) + 12345, 32, True),
])
@pytest.mark.parametrize("hash_kind", [HASH_MURMUR3, HASH_MD5])
def test_reach(cuda, approach, n, cs, bulk, hash_kind):
    import torch

    rng = np.random.default_rng(n + cs)
    x = rng.integers(0, 256, (n, cs), dtype=np.uint8)
    x[rng.integers(0, n, n // 10)] = 0
    y = x.copy()
    y[1000:1100] = x[5000:5100]
    y[2000:2050] = rng.integers(0, 256, (50, cs), dtype=np.uint8)
    tree = approach == "tree"
    g = (TreeDeduplicator if tree else ListDeduplicator)(cs, hash_kind)
    o = (O.OracleTreeDeduplicator if tree else O.OracleListDeduplicator)(cs, hash_kind, threads=8)
    launches = []
    for k, b in enumerate((x, y)):
        b = b.reshape(-1)
        assert g.checkpoint(torch.from_numpy(b).cuda(), k == 0) == o.checkpoint(b, k == 0), k
        launches.append(g.last_launch_count())
    assert (launches[0] > launches[1]) == bulk, launches
    g.close()
    o.close()
