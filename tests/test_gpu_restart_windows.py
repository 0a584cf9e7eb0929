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
