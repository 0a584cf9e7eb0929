"""Baselines whose tree digests and digest map are built in bulk (trees of 2^15 chunks and more, lists of
2^19).

The build partitions all digests by table range instead of inserting them one by one; labels, map
owners and everything that later checkpoints find in the map have to be those of the sequential
inserts (src/tree_approach.cpp:54-224, src/list_approach.cpp:23-77).  Byte for byte against the
oracle: the baseline and increments after it that refer to its chunks and subtrees, for one and two
scatter passes, chunk counts that are and are not powers of two, both hashes, both approaches, and
contents from all-distinct to all-equal.
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import ListDeduplicator, TreeDeduplicator
from reproducibility_icpp23_scalable_gpu_deduplication_b200.tree import HASH_MD5, HASH_MURMUR3

pytestmark = pytest.mark.gpu
TREE, LIST = 1 << 15, 1 << 19


def content(kind, n, cs, rng):
    if kind == "random":
        return rng.integers(0, 256, (n, cs), dtype=np.uint8)
    if kind == "sparse":   # a tenth of the chunks zero, repeated blocks of 64 chunks
        x = rng.integers(0, 256, (n, cs), dtype=np.uint8)
        x[rng.integers(0, n, n // 10)] = 0
        for at in rng.integers(0, n - 64, 200):
            x[at:at + 64] = x[64:128]
        return x
    if kind == "few":   # four chunk values: equal subtrees at every height
        return np.repeat(rng.integers(0, 4, (n, 1), dtype=np.uint8), cs, axis=1)
    if kind == "half":   # the second half repeats the first: one large equal subtree
        x = rng.integers(0, 256, (n, cs), dtype=np.uint8)
        x[n // 2:n // 2 * 2] = x[:n // 2]
        return x
    return np.full((n, cs), 7, np.uint8)   # equal


def series(kind, n, cs, seed):
    rng = np.random.default_rng(seed)
    x = content(kind, n, cs, rng)
    out = [x.copy()]
    for _ in range(2):
        x = x.copy()
        for at in rng.integers(0, n - 40, 60):   # fresh runs
            x[at:at + 40] = rng.integers(0, 256, (40, cs), dtype=np.uint8)
        for at, src in rng.integers(0, n - 256, (60, 2)) // 32 * 32:   # moved subtrees
            x[at:at + 32] = out[0][src:src + 32]
        out.append(x)
    return out


def compare(approach, kind, n, cs, hash_kind=HASH_MURMUR3, short=0, baselines=(1, 0, 0)):
    import torch

    tree = approach == "tree"
    bufs = [b.reshape(-1)[:n * cs - short] for b in series(kind, n, cs, n + cs)]
    g = (TreeDeduplicator if tree else ListDeduplicator)(cs, hash_kind)
    o = (O.OracleTreeDeduplicator if tree else O.OracleListDeduplicator)(cs, hash_kind, threads=8)
    for k, base in enumerate(baselines):
        b = np.ascontiguousarray(bufs[k])
        got = g.checkpoint(torch.from_numpy(b).cuda(), bool(base))
        assert got == o.checkpoint(b, bool(base)), (approach, kind, n, cs, k)
    g.close()
    o.close()


@pytest.mark.parametrize("kind", ["random", "sparse", "few", "half", "equal"])
@pytest.mark.parametrize("n", [TREE - 1, TREE, TREE + 1, 300001, 600000, 1 << 20])
def test_tree_contents_and_counts(cuda, kind, n):
    compare("tree", kind, n, 64)


@pytest.mark.parametrize("kind", ["random", "sparse", "few", "equal"])
@pytest.mark.parametrize("n", [LIST - 1, LIST, 1100000])
def test_list_contents_and_counts(cuda, kind, n):
    compare("list", kind, n, 64)


@pytest.mark.parametrize("approach", ["tree", "list"])
@pytest.mark.parametrize("hash_kind", [HASH_MURMUR3, HASH_MD5])
@pytest.mark.parametrize("cs,short", [(32, 0), (48, 5), (100, 99), (128, 0)])
def test_hashes_and_chunk_sizes(cuda, approach, hash_kind, cs, short):
    compare(approach, "sparse", LIST + 12345, cs, hash_kind, short)


@pytest.mark.parametrize("approach", ["tree", "list"])
def test_second_baseline(cuda, approach):
    compare(approach, "sparse", LIST + 12345, 64, baselines=(1, 0, 1))

