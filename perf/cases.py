"""Timed cases: checkpoint series and restarts through the public entry points.

A case is one of five kinds of pass:

  device        one series as a simulation writes it: a baseline checkpoint of the buffer, then an
                incremental checkpoint of each later state, every diff kept in device memory
  host          the same series with every diff returned to the host (``checkpoint``)
  batch         the same series for several buffers at once (``CheckpointBatch``)
  restart       the last state rebuilt from a chain of diffs in device memory
  restart_host  the last state rebuilt from a chain of diffs in host memory

A handle is kept from one series to the next, as a long-running program keeps it; a series starts
with a baseline, so every pass does the same work.
"""
import math

import numpy as np
import torch

from reproducibility_icpp23_scalable_gpu_deduplication_b200.batch import CheckpointBatch
from reproducibility_icpp23_scalable_gpu_deduplication_b200.tree import (
    HASH_MD5,
    HASH_MURMUR3,
    ListDeduplicator,
    TreeDeduplicator,
)

MIB = 1 << 20
MAX_ID = 8190   # checkpoint ids of one handle; a longer-lived program opens a new handle


def _case(name, kind, nbytes, chunk=128, ckpts=4, approach="tree", hash="murmur3", content="bytes", change=0.01,
          run=64, shift=0.005, zero=0.0, offset=0, count=1):
    return {"name": name, "kind": kind, "nbytes": nbytes, "chunk": chunk, "ckpts": ckpts, "approach": approach,
            "hash": hash, "content": content, "change": change, "run": run, "shift": shift, "zero": zero,
            "offset": offset, "count": count}


def listed():
    return [
        # the smallest buffer of the batched and served workloads, checkpointed alone with its diffs
        # taken to the host: launches and host work, little data
        _case("host_1m", "host", MIB, change=0.05, shift=0.01),
        # the 64 MiB configuration: 5 % rewritten in short runs, 2 % moved, 1 % zeroed
        _case("tree_64m", "device", 64 * MIB, ckpts=5, change=0.05, run=64, shift=0.02, zero=0.01),
        # an application's buffer: no power of two, a short last chunk, the batched change rate
        _case("tree_ragged", "device", 400_000_123, change=0.10, run=256, shift=0.01),
        # the headline size, 1 % changed per checkpoint
        _case("tree_4g", "device", 4096 * MIB),
        # the smallest and the largest chunk size of the 4 GiB configuration
        _case("tree_cs64", "device", 1024 * MIB, chunk=64),
        _case("tree_cs4096", "device", 1024 * MIB, chunk=4096),
        # training state: float32, MD5, noise on 30 % of the 64 KiB blocks, zero pages
        _case("md5_float", "device", 1024 * MIB, chunk=256, hash="md5", content="float", change=0.30, shift=0.05,
              zero=0.10),
        # records of a size that no vector width divides, from a view into a larger allocation
        _case("tree_records", "device", 150_000_000, chunk=1000, change=0.05, run=32, offset=8),
        # the list approach
        _case("list_512m", "device", 512 * MIB, approach="list", change=0.05, shift=0.02),
        # several ranks' or fields' buffers per call, uneven sizes, up to 256 MiB each
        _case("batch_12", "batch", 256 * MIB, change=0.10, run=256, shift=0.01, count=12),
        # recovery from diffs kept on the device, and from diffs read back into host memory
        _case("restart_1g", "restart", 1024 * MIB, ckpts=5, change=0.05),
        _case("restart_host", "restart_host", 128 * MIB - 100, change=0.05),
    ]


def draw(rng):
    kind = rng.choice(["host", "device", "device", "device", "device", "batch", "restart", "restart_host"])
    top = {"host": 64, "device": 1024, "batch": 128, "restart": 1024, "restart_host": 128}[kind] * MIB
    nbytes = int(math.exp(rng.uniform(math.log(MIB), math.log(top))))
    if rng.random() < 0.3:
        nbytes = 1 << round(math.log2(nbytes))   # many buffers are powers of two
    chunk = rng.choice([64, 128, 128, 256, 512, 1024, 4096, 48, 100, 200, 1000])
    if chunk % 16:
        nbytes = min(nbytes, 200 * MIB)
    content = rng.choice(["bytes", "bytes", "float"])
    approach = rng.choice(["tree", "tree", "tree", "list"])
    if kind.startswith("restart") and approach == "tree":
        # a tree restart is whole where the number of chunks is a power of two; the last may be short
        nbytes = chunk * (1 << round(math.log2(nbytes / chunk))) - rng.choice([0, 0, 4, chunk // 2 + 1])
    return {
        "kind": kind, "nbytes": nbytes, "chunk": chunk, "ckpts": rng.randint(2, 5),
        "approach": approach, "hash": rng.choice(["murmur3", "murmur3", "md5"]), "content": content,
        "change": 0.30 if content == "float" else math.exp(rng.uniform(math.log(0.005), math.log(0.2))),
        "run": rng.choice([8, 32, 64, 256]), "shift": rng.choice([0.0, 0.005, 0.02]),
        "zero": rng.choice([0.0, 0.01, 0.1]), "offset": rng.choice([0, 0, 0, 0, 4, 8]),
        "count": rng.randint(3, 12) if kind == "batch" else 1,
    }


# ------------------------------------------------------------------------------------------ inputs
def _sizes(case):
    """Buffer sizes of a case: one, or `count` spread evenly over the logarithm from 1 MiB up."""
    if case["count"] == 1:
        return [case["nbytes"]]
    lo, hi = math.log(MIB), math.log(max(case["nbytes"], 2 * MIB))
    return [int(math.exp(lo + (hi - lo) * i / (case["count"] - 1))) // 4 * 4 for i in range(case["count"])]


def _randint(hi, n, gen):
    return torch.randint(0, hi, (n,), generator=gen, device="cuda")


def _new_buffer(nbytes, offset):
    return torch.empty(nbytes + offset, dtype=torch.uint8, device="cuda")[offset:]


def _first_state(case, nbytes, gen):
    buf = _new_buffer(nbytes, case["offset"])
    if case["content"] == "float":   # float32 values N(0, 0.02)
        step = 256 * MIB
        for lo in range(0, nbytes, step):
            hi = min(nbytes, lo + step)
            v = torch.randn((hi - lo + 3) // 4, generator=gen, device="cuda") * 0.02
            buf[lo:hi] = v.view(torch.uint8)[:hi - lo]
        _zero_pages(case, buf, gen.initial_seed())
    else:
        buf.random_(0, 256, generator=gen)
    return buf


def _zero_pages(case, buf, seed):
    """A fixed part of the 4 KiB pages is zero in every state of a float series."""
    pages = buf.numel() // 4096
    if case["zero"] and pages:
        fixed = torch.Generator(device="cuda").manual_seed(seed + 1)
        rows = torch.unique(_randint(pages, int(case["zero"] * pages), fixed))
        buf[:pages * 4096].view(pages, 4096)[rows] = 0


def _next_state(case, old, gen):
    """A copy of `old` with part of its chunks rewritten in runs, moved from elsewhere or zeroed."""
    buf = _new_buffer(old.numel(), case["offset"])
    buf.copy_(old)
    cs = case["chunk"]
    m = buf.numel() // cs
    if m == 0:
        return buf
    rows, was = buf[:m * cs].view(m, cs), old[:m * cs].view(m, cs)
    if case["content"] == "float":   # fresh values on a part of the 64 KiB blocks
        block = 64 << 10
        blocks = max(1, buf.numel() // block)
        block = min(block, buf.numel() // 4 * 4)
        at = torch.unique(_randint(blocks, max(1, int(-math.log(1 - case["change"]) * blocks)), gen))
        values = torch.randn((at.numel(), block // 4), generator=gen, device="cuda") * 0.02
        buf[:blocks * block].view(blocks, block)[at] = values.view(torch.uint8)
    else:
        runs = max(1, round(case["change"] * m / ((1 + case["run"]) / 2)))
        lens, starts = _randint(case["run"], runs, gen) + 1, _randint(m, runs, gen)
        at = torch.repeat_interleave(starts, lens)
        at += torch.arange(at.numel(), device="cuda") - torch.repeat_interleave(torch.cumsum(lens, 0) - lens, lens)
        at = torch.unique(at.clamp_(max=m - 1))
        rows[at] = torch.randint(0, 256, (at.numel(), cs), dtype=torch.uint8, generator=gen, device="cuda")
    moved = int(case["shift"] * m)
    if moved:
        at = torch.unique(_randint(m, moved, gen))
        rows[at] = was[_randint(m, at.numel(), gen)]
    if case["content"] == "float":
        _zero_pages(case, buf, gen.initial_seed())
    elif case["zero"]:
        rows[torch.unique(_randint(m, int(case["zero"] * m), gen))] = 0
    return buf


def _series(case, nbytes, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    states = [_first_state(case, nbytes, gen)]
    while len(states) < case["ckpts"]:
        states.append(_next_state(case, states[-1], gen))
    return states


# ---------------------------------------------------------------------------------------- handles
class _Handle:
    """A deduplicator that a program keeps from series to series."""

    def __init__(self, case):
        self.make = TreeDeduplicator if case["approach"] == "tree" else ListDeduplicator
        self.args = case["chunk"], HASH_MD5 if case["hash"] == "md5" else HASH_MURMUR3
        self.dedup, self.ids = self.make(*self.args), 0

    def begin(self, ckpts):
        """The deduplicator for the next `ckpts` checkpoints."""
        if self.ids + ckpts > MAX_ID:
            self.dedup.close()
            self.dedup, self.ids = self.make(*self.args), 0
        self.ids += ckpts
        return self.dedup


class _DeviceBytes:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _room(case, nbytes):
    """Bytes that the diffs of a series take at most: header, region and shift tables, chunk data."""
    cs, run = case["chunk"], case["run"]
    n = -(-nbytes // cs)
    full = 4096 + 16 * n + n * cs
    if case["content"] == "float":
        later = MIB + 24 * n + int(0.45 * nbytes)
    else:
        later = 2 * MIB // 16 + 8 * n + max(1, round(case["change"] * n / ((1 + run) / 2))) * run * (cs + 4)
    return [full] + [min(full, later)] * (case["ckpts"] - 1)


def _keep(dedup, room):
    """Copies the last checkpoint's diff into memory of the program's own; returns its length."""
    ptr, n = dedup.diff_device()
    room[:n].copy_(torch.as_tensor(_DeviceBytes(ptr, n), device="cuda"))
    return n


def _device_series(dedup, states, rooms):
    lengths = []
    for k, (data, room) in enumerate(zip(states, rooms)):
        dedup.checkpoint_device(data, make_baseline=k == 0)
        lengths.append(_keep(dedup, room))
    return lengths


def _host_series(dedup, states, rooms):
    lengths = []
    for k, (data, room) in enumerate(zip(states, rooms)):
        diff = dedup.checkpoint(data, make_baseline=k == 0, copy=False)
        room[:diff.size] = diff
        lengths.append(diff.size)
    return lengths


# ------------------------------------------------------------------------------------------ passes
def prepare(case, seed):
    sizes = _sizes(case)
    buffers = [_series(case, n, seed * 1000 + i) for i, n in enumerate(sizes)]
    on_host = case["kind"] in ("host", "restart_host")
    make = (lambda n: np.zeros(n, np.uint8)) if on_host else lambda n: torch.zeros(n, dtype=torch.uint8, device="cuda")
    state = {"kind": case["kind"], "buffers": buffers, "handles": [_Handle(case) for _ in sizes],
             "rooms": [[make(n) for n in _room(case, size)] for size in sizes]}
    if case["kind"] == "batch":
        state["batch"] = CheckpointBatch()
    if case["kind"].startswith("restart"):
        dedup, rooms = state["handles"][0].begin(case["ckpts"]), state.pop("rooms")[0]
        lengths = (_host_series if on_host else _device_series)(dedup, buffers[0], rooms)
        dedup.close()
        state["diffs"] = [room[:n] if on_host else room[:n].clone() for room, n in zip(rooms, lengths)]
        state["out"] = _new_buffer(sizes[0], case["offset"]).zero_()
        state["last"] = case["ckpts"] - 1
        state["restarter"] = _Handle(case).dedup   # a program that recovers starts with a handle of its own
        del state["buffers"], state["handles"]
    return state


def run(state):
    kind = state["kind"]
    if kind == "restart":
        state["restarter"].restart_device(state["out"], state["diffs"], state["last"])
        return state["out"]
    if kind == "restart_host":
        state["restarter"].restart(state["out"], state["diffs"], state["last"])
        return state["out"]
    buffers, rooms = state["buffers"], state["rooms"]
    ckpts = len(buffers[0])
    dedups = [h.begin(ckpts) for h in state["handles"]]
    if kind == "device":
        lengths = _device_series(dedups[0], buffers[0], rooms[0])
    elif kind == "host":
        lengths = _host_series(dedups[0], buffers[0], rooms[0])
    else:
        lengths = []
        for k in range(ckpts):
            state["batch"].checkpoint(dedups, [b[k] for b in buffers], make_baseline=k == 0)
            lengths += [_keep(d, room[k]) for d, room in zip(dedups, rooms)]
    return {"lengths": np.array(lengths), "diffs": rooms}


def work(case):
    """Every state read once, every diff written once, and the digests that a series cannot do
    without: one written per chunk by the baseline, one read per chunk by each later checkpoint.
    A restart reads each chunk's data once and writes it once."""
    total = sum(_sizes(case))
    if case["kind"].startswith("restart"):
        return {"bytes": 2 * total, "flops": 0}
    chunks = total / case["chunk"]
    later = case["ckpts"] - 1
    states = (1 + later) * (total + 16 * chunks)
    return {"bytes": states + total + later * case["change"] * total, "flops": 0}
