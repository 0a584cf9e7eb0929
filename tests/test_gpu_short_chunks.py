"""Chunks that are hashed where they lie and chunks that are staged, on both sides of the line.

Short chunks on buffers or sizes the tensor-map kernel does not take are read directly, longer ones
through shared memory; where the line lies depends on the hash and on whether chunks and buffer are
4-byte aligned.  Whole series against the oracle, byte for byte: chunk counts around a warp's and around
those of a bulk build, short last chunks, views at odd offsets, both hashes, both approaches, and batches.
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import CheckpointBatch, ListDeduplicator, TreeDeduplicator
from reproducibility_icpp23_scalable_gpu_deduplication_b200.tree import HASH_MD5, HASH_MURMUR3

pytestmark = pytest.mark.gpu


def series(cs, nbytes, seed):
    """three states: random bytes, then fresh, moved and zeroed chunks"""
    rng = np.random.default_rng(seed)
    x = rng.integers(0, 256, nbytes, dtype=np.uint8)
    out = [x]
    m = nbytes // cs
    for _ in range(2):
        x = x.copy()
        rows, was = x[:m * cs].reshape(m, cs), out[-1][:m * cs].reshape(m, cs)
        if m:
            at = rng.integers(0, m, 1 + m // 20)
            rows[at] = rng.integers(0, 256, (at.size, cs), dtype=np.uint8)
            at = rng.integers(0, m, 1 + m // 50)
            rows[at] = was[rng.integers(0, m, at.size)]
            rows[rng.integers(0, m, 1 + m // 100)] = 0
        x[-1] ^= 1
        out.append(x)
    return out


def place(x, offset):
    import torch

    mem = torch.zeros(x.size + 64, dtype=torch.uint8, device="cuda")
    view = mem[offset:offset + x.size]
    view.copy_(torch.from_numpy(np.ascontiguousarray(x)))
    return view


@pytest.mark.parametrize("hash_kind,cs", [
    (HASH_MURMUR3, 3), (HASH_MURMUR3, 44), (HASH_MURMUR3, 47), (HASH_MURMUR3, 48), (HASH_MURMUR3, 49),
    (HASH_MURMUR3, 108), (HASH_MURMUR3, 111), (HASH_MURMUR3, 112), (HASH_MD5, 3), (HASH_MD5, 32), (HASH_MD5, 63),
    (HASH_MD5, 64), (HASH_MD5, 65)])
@pytest.mark.parametrize("offset", [0, 1, 4, 8])
@pytest.mark.parametrize("n", [1, 31, 33, 5000])
def test_lines(cuda, hash_kind, cs, offset, n):
    for D, R in ((TreeDeduplicator, O.OracleTreeDeduplicator), (ListDeduplicator, O.OracleListDeduplicator)):
        nbytes = n * cs - cs // 2
        g, o = D(cs, hash_kind), R(cs, hash_kind)
        for k, x in enumerate(series(cs, nbytes, n + cs)):
            assert g.checkpoint(place(x, offset), k == 0) == o.checkpoint(x, k == 0), (D.__name__, k)
        if offset or cs % (64 if hash_kind == HASH_MD5 else 16):
            assert g.phase_times()[1] == 0
        g.close()
        o.close()


@pytest.mark.parametrize("D,R,n", [(TreeDeduplicator, O.OracleTreeDeduplicator, 40001),
                                   (ListDeduplicator, O.OracleListDeduplicator, (1 << 19) + 77)])
@pytest.mark.parametrize("cs,hash_kind", [(44, HASH_MURMUR3), (36, HASH_MD5)])
def test_bulk_baselines(cuda, D, R, n, cs, hash_kind):
    """with runs of equal chunks, which the hashing labels, and scattered ones"""
    rng = np.random.default_rng(n)
    x = rng.integers(0, 256, (n, cs), dtype=np.uint8)
    x[100:300] = x[99]
    x[rng.integers(0, n, n // 20)] = 0
    g, o = D(cs, hash_kind), R(cs, hash_kind)
    launches = []
    for k in range(2):
        x[5000 + k] = x[7]
        b = x.reshape(-1)[:n * cs - 5]
        assert g.checkpoint(place(b, 4), k == 0) == o.checkpoint(b, k == 0), k
        launches.append(g.last_launch_count())
    assert launches[0] > launches[1]   # the baseline was built in bulk
    g.close()
    o.close()


def test_batch(cuda):
    specs = [(44, 3000 * 44 - 7, 4), (63, 2000 * 63, 1), (100, 999 * 100, 8), (5, 40000, 3)]
    ss = [series(cs, nb, i) for i, (cs, nb, _) in enumerate(specs)]
    hs, os_ = [TreeDeduplicator(cs) for cs, _, _ in specs], [O.OracleTreeDeduplicator(cs) for cs, _, _ in specs]
    with CheckpointBatch() as b:
        for k in range(3):
            xs = [s[k] for s in ss]
            b.checkpoint(hs, [place(x, off) for x, (_, _, off) in zip(xs, specs)], [k == 0] * len(hs))
            for h, o, x in zip(hs, os_, xs):
                assert bytes(h.copy_diff()) == o.checkpoint(x, k == 0), k
    for h, o in zip(hs, os_):
        h.close()
        o.close()
