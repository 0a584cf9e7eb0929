"""Restarts from lists of device diffs: what is read of the list, and when.

A restart follows the chain from the selected diff down to its baseline (src/tree_approach.cpp:966-1128)
and reads the headers of the diffs on it, after the work that made them.
"""
import ctypes

import numpy as np
import pytest

from reproducibility_icpp23_scalable_gpu_deduplication_b200 import TreeDeduplicator
from reproducibility_icpp23_scalable_gpu_deduplication_b200._lib import lib

pytestmark = pytest.mark.gpu

CS, N = 128, 4096
B2D_ERR_CUDA, B2D_ERR_FORMAT = -2, -4


def to_dev(a):
    import torch

    return torch.from_numpy(np.frombuffer(a, np.uint8).copy()).cuda()


def states(count):
    rng = np.random.default_rng(3)
    out = [rng.integers(0, 256, (N, CS), dtype=np.uint8)]
    for k in range(1, count):
        x = out[-1].copy()
        x[20 * k:20 * k + 30] = rng.integers(0, 256, (30, CS), dtype=np.uint8)
        out.append(x)
    return [x.reshape(-1) for x in out]


def diffs_of(bufs, baselines=(0,)):
    g = TreeDeduplicator(CS)
    out = [g.checkpoint(to_dev(b), k in baselines) for k, b in enumerate(bufs)]
    g.close()
    return out


def restart(g, out, entries, last):
    """b2d_restart_device with (address, size) entries, on the handle's stream"""
    ptrs = (ctypes.c_void_p * len(entries))(*[a for a, _ in entries])
    sizes = (ctypes.c_uint64 * len(entries))(*[n for _, n in entries])
    return lib().b2d_restart_device(g._h, ctypes.c_void_p(out.data_ptr()), out.numel(), ptrs, sizes, len(entries), last)


def entries_of(tensors):
    return [(t.data_ptr(), t.numel()) for t in tensors]


@pytest.mark.parametrize("at", [3, 1, 0])
def test_pageable_entry_is_refused(cuda, at):
    """a diff in memory that is not the device's: an error, and the handle goes on"""
    import torch

    bufs = states(4)
    diffs = diffs_of(bufs)
    dev = [to_dev(d) for d in diffs]
    host = np.frombuffer(diffs[at], np.uint8).copy()
    entries = entries_of(dev)
    entries[at] = (host.ctypes.data, host.size)
    g = TreeDeduplicator(CS)
    out = torch.zeros(N * CS, dtype=torch.uint8, device="cuda")
    assert restart(g, out, entries, 3) == B2D_ERR_CUDA
    assert restart(g, out, entries_of(dev), 3) == 0
    assert np.array_equal(out.cpu().numpy(), bufs[3])
    g.close()


@pytest.mark.parametrize("entry", ["null", "short"])
def test_entries_off_the_chain_are_not_read(cuda, entry):
    """a chain that an older diff ends early (a baseline that stands for those before it): what the
    list holds below it does not matter"""
    import torch

    bufs = states(4)
    mixed = diffs_of(bufs)[:2] + [diffs_of(bufs[:3], (0, 2))[2], diffs_of(bufs)[3]]
    dev = [to_dev(d) for d in mixed]
    entries = entries_of(dev)
    for k in (0, 1):
        entries[k] = (None, 4096) if entry == "null" else (dev[k].data_ptr(), 31)
    g = TreeDeduplicator(CS)
    out = torch.zeros(N * CS, dtype=torch.uint8, device="cuda")
    assert restart(g, out, entries, 3) == 0
    assert np.array_equal(out.cpu().numpy(), bufs[3])
    # on the chain they do
    entries = entries_of([to_dev(d) for d in diffs_of(bufs)])
    entries[1] = (None, 4096) if entry == "null" else (dev[1].data_ptr(), 31)
    assert restart(g, out, entries, 3) == B2D_ERR_FORMAT
    g.close()


@pytest.mark.parametrize("count", [8, 9, 64, 65, 73, 140])
def test_long_chains(cuda, count):
    """chains of one and of several header reads"""
    import torch

    bufs = states(count)
    dev = [to_dev(d) for d in diffs_of(bufs)]
    g = TreeDeduplicator(CS)
    for last in (count - 1, count - 2):
        out = torch.zeros(N * CS, dtype=torch.uint8, device="cuda")
        assert restart(g, out, entries_of(dev), last) == 0
        assert np.array_equal(out.cpu().numpy(), bufs[last]), last
    g.close()


@pytest.mark.parametrize("stream", ["other", "own"])
def test_follows_the_default_stream(cuda, stream):
    """diffs that the default stream is still copying when the restart is called"""
    import torch

    bufs = states(4)
    src = [to_dev(d) for d in diffs_of(bufs)]
    g = TreeDeduplicator(CS)
    other = torch.cuda.Stream()
    assert lib().b2d_set_stream(g._h, ctypes.c_void_p(other.cuda_stream if stream == "other" else None)) == 0
    for _ in range(3):
        dst = [torch.zeros_like(x) for x in src]
        out = torch.zeros(N * CS, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)   # about 10 ms before the copies start
        for x, y in zip(dst, src):
            x.copy_(y)
        assert restart(g, out, entries_of(dst), 3) == 0
        assert np.array_equal(out.cpu().numpy(), bufs[3])
    g.close()
