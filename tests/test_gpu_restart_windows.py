"""Restarts whose diffs are resolved in windows of any size, and what a handle holds after one.

A chain's diffs are expanded and resolved a window at a time (src/tree_approach.cpp:966-1128 goes
through them one by one); the buffer rebuilt does not depend on the window.
"""
import numpy as np
import pytest

from oracle import oracle as O
from reproducibility_icpp23_scalable_gpu_deduplication_b200 import ListDeduplicator, TreeDeduplicator, synth

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def to_dev(a):
    import torch

    return torch.from_numpy(np.frombuffer(a, np.uint8).copy()).cuda()


@pytest.mark.parametrize("approach", ["tree", "list"])
@pytest.mark.parametrize("window", [0, 1, 2, 3, 8])
def test_windows(cuda, approach, window):
    import torch

    tree = approach == "tree"
    cs, nbytes = 128, 128 * 3001 - 5
    s = synth.ByteSeries(nbytes, cs, lambda r, n: synth.plan_varied(r, n, 16), 9, buf_id=1)
    g = (TreeDeduplicator if tree else ListDeduplicator)(cs)
    diffs = [g.checkpoint(torch.from_numpy(np.ascontiguousarray(s.next())).cuda(), k == 0) for k in range(12)]
    g.set_param("restart_window", window)
    dev = [to_dev(d) for d in diffs]
    for last in (0, 1, 11):
        want, orc = (O.restart if tree else O.list_restart)(diffs, last)
        for run, chain in ((g.restart, diffs), (g.restart_device, dev)):
            out = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
            rc = run(out, chain, last, check_status=False)
            assert (rc == 0) == (orc == 0), (last, rc, orc)
            assert out.cpu().numpy().tobytes() == want.tobytes(), last
    g.close()


def test_memory_of_a_host_restart(cuda):
    """a chain of large diffs in host memory passes through a bounded part of the device's"""
    import torch

    n = 64 * MIB
    states = [torch.empty(n, dtype=torch.uint8, device="cuda").random_(0, 256) for _ in range(7)]
    with TreeDeduplicator(128) as g:
        diffs = [np.frombuffer(g.checkpoint(x, k == 0), np.uint8) for k, x in enumerate(states)]
    held = []
    for window in (0, 1):
        with TreeDeduplicator(128) as g:
            g.set_param("restart_window", window)
            out = torch.zeros(n, dtype=torch.uint8, device="cuda")
            g.restart(out, diffs, 6)
            assert torch.equal(out, states[6])
            held.append(g.memory())
    # at most 256 MiB of diffs, a slot of 13 bytes per chunk and diff, 9 bytes per chunk, and lists
    assert held[0] < 256 * MIB + (n // 128) * (13 * 5 + 9) + 8 * MIB
    # one diff at a time: the largest of them and one slot
    assert held[1] < len(max(diffs, key=len)) + (n // 128) * (13 + 9) + 8 * MIB


def plain_chain(nbytes, cs, count):
    """states that only rewrite chunks (no moves): restarts are whole for any chunk count"""
    import torch

    rng = np.random.default_rng(cs)
    x = rng.integers(0, 256, nbytes, dtype=np.uint8)
    states, diffs = [], []
    with ListDeduplicator(cs) as g:
        for k in range(count):
            x = x.copy()
            x[k * 5000 * cs:(k * 5000 + 3000) * cs] = rng.integers(0, 256, 3000 * cs, dtype=np.uint8)
            states.append(x)
            diffs.append(np.frombuffer(g.checkpoint(torch.from_numpy(x).cuda(), k == 0), np.uint8))
    return states, diffs


@pytest.mark.parametrize("kind", ["pageable", "page-locked", "mixed"])
@pytest.mark.parametrize("stream", [None, 1, 2])
def test_uploads(cuda, kind, stream):
    """host diffs of several upload pieces, in pageable and page-locked memory, on the handle's own, the
    legacy default and the per-thread default stream"""
    import ctypes

    import torch

    from reproducibility_icpp23_scalable_gpu_deduplication_b200._lib import lib

    states, diffs = plain_chain(40 * MIB + 77, 128, 4)
    keep = []
    for k, d in enumerate(diffs):
        if kind == "page-locked" or (kind == "mixed" and k % 2):
            t = torch.empty(d.size, dtype=torch.uint8, pin_memory=True)
            t.copy_(torch.from_numpy(d.copy()))
            keep.append(t)
            diffs[k] = t.numpy()
    ptrs = (ctypes.c_void_p * 4)(*[d.ctypes.data for d in diffs])
    sizes = (ctypes.c_uint64 * 4)(*[d.size for d in diffs])
    with ListDeduplicator(128) as g:
        assert lib().b2d_set_stream(g._h, ctypes.c_void_p(stream)) == 0
        for last in (3, 0, 2):
            out = torch.zeros(states[0].size, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            assert lib().b2d_restart(g._h, ctypes.c_void_p(out.data_ptr()), out.numel(), ptrs, sizes, 4, last, None) == 0
            assert np.array_equal(out.cpu().numpy(), states[last]), last


@pytest.mark.parametrize("cs", [64, 100, 128, 256])
@pytest.mark.parametrize("offset", [0, 1, 4, 8])
def test_output_alignments(cuda, cs, offset):
    """outputs of 2^15 chunks and more that do not start on 16 bytes"""
    import torch

    nbytes = cs * 33333 - 9
    states, diffs = plain_chain(nbytes, cs, 4)
    dev = [to_dev(d) for d in diffs]
    with ListDeduplicator(cs) as g:
        for run, chain in ((g.restart, diffs), (g.restart_device, dev)):
            mem = torch.full((nbytes + 64,), 7, dtype=torch.uint8, device="cuda")
            run(mem[offset:offset + nbytes], chain, 3)
            assert np.array_equal(mem[offset:offset + nbytes].cpu().numpy(), states[3])
            assert bool((mem[:offset] == 7).all()) and bool((mem[offset + nbytes:] == 7).all())


@pytest.mark.parametrize("cs", [64, 80, 96, 112, 128, 144])
@pytest.mark.parametrize("nbytes", [32 * MIB - 5, 33 * MIB + 5])
def test_large_walks(cuda, cs, nbytes):
    """outputs on both sides of the size and the chunk sizes from which copies are staged, from diffs at
    several alignments, in one window and in several"""
    import torch

    states, diffs = plain_chain(nbytes, cs, 4)
    with ListDeduplicator(cs) as g:
        for window in (0, 1):
            g.set_param("restart_window", window)
            for shift in (0, 1, 4, 8):
                mems = [torch.zeros(d.size + 16, dtype=torch.uint8, device="cuda") for d in diffs]
                dev = []
                for m, d in zip(mems, diffs):
                    v = m[shift:shift + d.size]
                    v.copy_(torch.from_numpy(d.copy()))
                    dev.append(v)
                out = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
                g.restart_device(out, dev, 3)
                assert np.array_equal(out.cpu().numpy(), states[3]), (window, shift)
            out.zero_()
            g.restart(out, diffs, 3)
            assert np.array_equal(out.cpu().numpy(), states[3]), window
