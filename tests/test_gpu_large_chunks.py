"""Chunk sizes far above the buffer's length, up to the largest that fits 32 bits.

The whole buffer is one short chunk then, whose digest is that of the bytes there are, whatever the
chunk size.  Trees against the oracle, byte for byte (a tree of one chunk has no region, so its diff
is a header); a list's diff, whose data section is a whole chunk, by its digest and its first bytes.
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import ListDeduplicator, TreeDeduplicator
from reproducibility_icpp23_scalable_gpu_deduplication_b200.tree import HASH_MD5, HASH_MURMUR3

pytestmark = pytest.mark.gpu

SIZES = [0xffffffff, 0xfffffff1, 0xfffffff0, (1 << 30) + 7]
LENGTHS = [1, 63, 64, 127, 128, 129, 1000]


def buffers(cs):
    rng = np.random.default_rng(cs)
    return [rng.integers(1, 256, n, dtype=np.uint8) for n in LENGTHS]


@pytest.mark.parametrize("hash_kind", [HASH_MURMUR3, HASH_MD5])
@pytest.mark.parametrize("cs", SIZES)
def test_tree_of_one_short_chunk(cuda, cs, hash_kind):
    import torch

    g, o = TreeDeduplicator(cs, hash_kind), O.OracleTreeDeduplicator(cs, hash_kind)
    for x in buffers(cs):
        t = torch.from_numpy(x).cuda()
        for base in (True, False):
            assert g.checkpoint(t, base) == o.checkpoint(x, base), (x.size, base)
            assert g.debug_tree(1)[0].tobytes() == O.hash_bytes(x, hash_kind), (x.size, base)
            # the work follows the bytes there are: following the chunk size, it took 15 s
            assert g.phase_times()[0][0] < 0.1
    g.close()
    o.close()


@pytest.mark.parametrize("cs", SIZES)
def test_list_of_one_short_chunk(cuda, cs):
    import torch

    class Device:
        pass

    g = ListDeduplicator(cs)
    for x in buffers(cs)[::3]:
        t = torch.from_numpy(x).cuda()
        assert g.checkpoint_device(t, make_baseline=True) == 32 + 4 + cs
        assert g.debug_tree(1)[0].tobytes() == O.hash_bytes(x)
        d = Device()
        d.__cuda_array_interface__ = {"shape": (36 + cs,), "typestr": "|u1", "data": (g.diff_device()[0], False),
                                      "version": 3}
        diff = torch.as_tensor(d, device="cuda")
        assert torch.equal(diff[36:36 + x.size], t) and int(diff[36 + x.size:].max()) == 0
        assert g.checkpoint_device(t) == 32   # unchanged
    g.close()
