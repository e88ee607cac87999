"""The work a user of this library has it do, as cases that can be timed.

Four kinds of case, each through the public Python entry points:

* ``series``: a running application's period -- some incremental checkpoints
  of a buffer that changed between them, each archived in device memory (or
  fetched to the host), then the next baseline;
* ``batch``: the same period for many buffers of uneven sizes at once;
* ``restart``: one checkpoint rebuilt from its chain, held in device or in
  host memory;
* ``hash``: the digests of every chunk of a buffer.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program has in hand before the call, ``run`` is one
pass and returns what it computes, ``work`` is what a pass cannot do without
and ``exact`` is a restart's buffer as the application wrote it.
"""
import math

import numpy as np
import torch

import mtcheck_gb300 as mc
from mtcheck_gb300 import workloads

APPROACH = {"basic": mc.BASIC, "list": mc.LIST, "tree": mc.TREE, "tree_ref": mc.TREE_LOW_OFFSET_REF}
HASH = {"murmur3": mc.MURMUR3, "md5": mc.MD5}
# chunk sizes of the configurations and tests: powers of two, and sizes that
# are no multiple of a 16-byte word
CHUNKS = (16, 32, 64, 128, 128, 256, 256, 512, 512, 4096)
ODD_CHUNKS = (24, 48, 100, 640)


def _series(name, nbytes, chunk, approach="tree", hash="murmur3", steps=4, rate=0.02, run_max=4096, dup=0.0,
            offset=0, host=False):
    return {"name": name, "kind": "series", "nbytes": nbytes, "chunk": chunk, "approach": approach, "hash": hash,
            "steps": steps, "rate": rate, "run_max": run_max, "dup": dup, "offset": offset, "host": host}


def _restart(name, nbytes, chunk, approach, chain, hash="murmur3", rate=0.02, run_max=4096, host=False):
    return {"name": name, "kind": "restart", "nbytes": nbytes, "chunk": chunk, "approach": approach, "hash": hash,
            "steps": chain - 1, "rate": rate, "run_max": run_max, "dup": 0.0, "offset": 0, "host": host}


def listed():
    return [
        # a small state checkpointed often, each checkpoint written out by the
        # host: launches and latency count; the last chunk is short
        _series("tree_1mb_to_host", 1_000_000, 128, steps=4, run_max=32, host=True),
        # the plain series: 64 MiB in 128 B chunks, a fifth of the chunks
        # copies of others, 1% rewritten in short runs, ten checkpoints
        _series("tree_64mib", 64 << 20, 128, steps=9, rate=0.01, run_max=32, dup=0.2),
        # a large single buffer, sparse and long changes and shifted copies
        _series("tree_4gib", 4 << 30, 512, steps=5, rate=0.025),
        # the same pattern with MD5 digests
        _series("tree_md5_1gib", 1 << 30, 512, hash="md5", steps=4, rate=0.025),
        # the hash-list approach in the smallest chunks of the mixed workload,
        # a size that fills no tile
        _series("list_200mb", 200_000_000, 64, approach="list", steps=4, run_max=256),
        # records of 100 bytes: chunks that are no multiple of a word
        _series("basic_odd_64mb", 64_000_003, 100, approach="basic", steps=4, run_max=256),
        # many buffers of uneven sizes, chunk sizes and digests in one call
        {"name": "batch_24", "kind": "batch", "members": 24, "median_mib": 12.0, "hi_mib": 64, "mix": 4, "steps": 4},
        # the last of 31 checkpoints of a large buffer, chain on the device
        _restart("restart_tree_1gib", 1 << 30, 256, "tree", 31, rate=0.025),
        # the last of 10, its chain as files leave it: in host memory
        _restart("restart_list_64mib_host", 64 << 20, 128, "list", 10, rate=0.01, run_max=32, host=True),
        # records of 100 bytes again
        _restart("restart_basic_odd_64mb", 64_000_000, 100, "basic", 8, run_max=256),
        # digests alone, as a program that verifies a buffer takes them
        {"name": "hash_4k_256mib", "kind": "hash", "nbytes": 256 << 20, "chunk": 4096, "hash": "murmur3", "offset": 0},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choices(("series", "restart", "hash", "batch"), (10, 5, 3, 2))[0]
    chunk = rng.choice(CHUNKS if rng.random() < 0.75 else ODD_CHUNKS)
    hash = rng.choice(("murmur3", "murmur3", "md5"))
    offset = rng.choice((0, 0, 0, 4, 8, 16))  # where in its allocation the buffer starts
    if kind == "hash":
        nbytes = min(_log_int(rng, 1 << 14, 2 << 30), chunk << 24)
        return {"kind": kind, "nbytes": nbytes, "chunk": chunk, "hash": hash, "offset": offset}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(4, 32), "median_mib": round(rng.uniform(2.0, 14.0), 2),
                "hi_mib": 64, "mix": rng.randint(1, 1000), "steps": rng.randint(2, 4)}
    rate = round(rng.uniform(0.002, 0.05), 4)
    run_max = rng.choice((32, 256, 4096))
    if kind == "restart":
        approach = rng.choice(("tree", "tree", "list", "basic"))
        nbytes = min(_log_int(rng, 1 << 18, 512 << 20), chunk << 21)
        if approach == "tree":  # a power of two of whole chunks, for which a tree restart gives every chunk back
            nbytes = chunk << max(8, (nbytes // chunk).bit_length() - 1)
        c = _restart("", nbytes, chunk, approach, rng.randint(2, 16), hash, rate, run_max, rng.random() < 0.3)
    else:
        approach = rng.choice(("tree", "tree", "tree", "list", "basic", "tree_ref"))
        nbytes = min(_log_int(rng, 1 << 16, 1536 << 20), chunk << 22)
        host = nbytes < (4 << 20) and rng.random() < 0.5
        c = _series("", nbytes, chunk, approach, hash, rng.randint(1, 5), rate, run_max,
                    rng.choice((0.0, 0.0, 0.2)), offset, host)
    c.pop("name")
    return c


class _View:
    """A handle's device memory as an array, which keeps the handle."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _diff(dedup):
    ptr, n = dedup.diff_device()
    return torch.as_tensor(_View(dedup, ptr, n), device="cuda")


def _buffer(nbytes, offset=0):
    return torch.empty(nbytes + offset, dtype=torch.uint8, device="cuda")[offset:]


def _changes(rng, n, rate, run_max):
    """The chunks that one step of the update pattern writes: `rate` of them
    changed, half single chunks and half runs of up to `run_max`, and a tenth
    as many overwritten by copies of chunks at earlier offsets."""
    count = max(2, int(rate * n))
    single = rng.integers(0, n, count // 2)
    lens = rng.integers(1, run_max + 1, count)
    lens = lens[:int(np.searchsorted(np.cumsum(lens), count - count // 2)) + 1]
    lens[-1] -= int(lens.sum()) - (count - count // 2)
    starts = (rng.random(lens.size) * np.maximum(1, n - lens)).astype(np.int64)
    within = np.arange(int(lens.sum())) - np.repeat(np.cumsum(lens) - lens, lens)
    runs = np.minimum(np.repeat(starts, lens) + within, n - 1)
    dst = np.unique(rng.integers(1, n, max(1, count // 10)))
    return np.unique(np.concatenate([single, runs])), dst, (rng.random(dst.size) * dst).astype(np.int64)


def _states(case, seed):
    """The buffer's states: the first, then one per incremental checkpoint.
    Which chunks change goes by the case, every byte written by the seed, so
    that the checkpoints of two seeds have one size."""
    cs, where = case["chunk"], np.random.default_rng([case["nbytes"], case["chunk"], case["steps"]])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))

    def fresh(*shape):
        return torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=gen)

    def at(index):
        return torch.from_numpy(index).cuda()

    full = case["nbytes"] // cs
    buf = _buffer(case["nbytes"], case["offset"])
    buf.copy_(fresh(case["nbytes"]))
    rows = buf[:full * cs].view(full, cs)
    if case["dup"] and full > 1:
        dst = np.unique(where.integers(full // 2, full, int(case["dup"] * full)))
        rows[at(dst)] = rows[at(where.integers(0, full // 2, dst.size))]
    yield buf
    for _ in range(case["steps"]):
        nxt = _buffer(case["nbytes"], case["offset"])
        nxt.copy_(buf)
        changed, dst, src = _changes(where, full, case["rate"], case["run_max"])
        rows, old = nxt[:full * cs].view(full, cs), buf[:full * cs].view(full, cs)
        rows[at(changed)] = fresh(changed.size, cs)
        rows[at(dst)] = old[at(src)]
        yield nxt
        buf = nxt


def _members(case, seed):
    mix = workloads.batch_mix(case["members"], seed=case["mix"], median_mib=case["median_mib"], hi_mib=case["hi_mib"])
    return [{"nbytes": m["nbytes"], "chunk": m["chunk_size"], "hash": m["hash"], "rate": m["rate"], "steps": case["steps"],
             "run_max": 4096, "dup": 0.0, "offset": 0, "seed": seed * 1000 + i} for i, m in enumerate(mix)]


def _chain(case, seed):
    """A handle, its chain of checkpoints (device tensors or host bytes) and the last state."""
    dedup = mc.Deduplicator(case["chunk"], HASH[case["hash"]], approach=APPROACH[case["approach"]])
    chain, last = [], None
    for i, buf in enumerate(_states(case, seed)):
        if case["host"]:
            chain.append(dedup.checkpoint(buf, i == 0))
        else:
            dedup.checkpoint_device(buf, i == 0)
            chain.append(_diff(dedup).clone())
        last = buf
    return dedup, chain, last


def prepare(case, seed):
    if case["kind"] == "hash":
        buf = _buffer(case["nbytes"], case["offset"])
        gen = torch.Generator(device="cuda")
        gen.manual_seed(int(seed))
        buf.copy_(torch.randint(0, 256, (case["nbytes"],), dtype=torch.uint8, device="cuda", generator=gen))
        out = torch.empty(-(-case["nbytes"] // case["chunk"]) * 16, dtype=torch.uint8, device="cuda")
        return {"case": case, "buf": buf, "out": out}
    if case["kind"] == "restart":
        dedup, chain, _ = _chain(case, seed)
        out = torch.zeros(case["nbytes"], dtype=torch.uint8, device="cuda")
        where = chain if case["host"] else [(c.data_ptr(), c.numel()) for c in chain]
        return {"case": case, "dedup": dedup, "chain": chain, "where": where, "out": out}
    if case["kind"] == "batch":
        members = _members(case, seed)
        states = list(zip(*[list(_states(m, m["seed"])) for m in members]))
        batch = mc.Batch([(mc.TREE, m["hash"], m["chunk"]) for m in members])
        batch.checkpoint(states[0], make_baseline=True)
        return {"case": case, "batch": batch, "states": states}
    dedup = mc.Deduplicator(case["chunk"], HASH[case["hash"]], approach=APPROACH[case["approach"]])
    states = list(_states(case, seed))
    # the first baseline, as a program has taken it before its main loop
    dedup.checkpoint_device(states[0], True)
    return {"case": case, "dedup": dedup, "states": states}


def run(state):
    case = state["case"]
    if case["kind"] == "hash":
        return mc.hash_chunks(HASH[case["hash"]], state["buf"], case["chunk"], out=state["out"])
    if case["kind"] == "restart":
        dedup, last = state["dedup"], case["steps"]
        if case["host"]:
            dedup.restart(state["out"], state["where"], last)
        else:
            dedup.restart_device(state["out"], state["where"], last)
        return state["out"]
    states = state["states"]
    if case["kind"] == "batch":
        batch, out = state["batch"], []
        for bufs in states[1:]:
            batch.checkpoint(bufs)
            out.append(torch.cat([_diff(m) for m in batch.members]))
        batch.checkpoint(states[0], make_baseline=True)
        return out + [torch.cat([_diff(m) for m in batch.members])]
    dedup, out = state["dedup"], []
    if case["host"]:
        for buf in states[1:]:
            out.append(np.frombuffer(dedup.checkpoint(buf, False), np.uint8))
        return out + [np.frombuffer(dedup.checkpoint(states[0], True), np.uint8)]
    for buf in states[1:]:
        dedup.checkpoint_device(buf, False)
        out.append(_diff(dedup).clone())
    dedup.checkpoint_device(states[0], True)
    return out + [_diff(dedup)]


def _series_bytes(nbytes, chunk, steps, rate):
    """Every checkpoint reads its state and reads and writes a digest per
    chunk; an incremental one writes the changed chunks, a baseline all."""
    n = -(-nbytes // chunk)
    return (steps + 1) * (nbytes + 32 * n) + steps * rate * nbytes + nbytes


def work(case):
    if case["kind"] == "hash":
        return {"bytes": case["nbytes"] + 16 * -(-case["nbytes"] // case["chunk"]), "flops": 0}
    if case["kind"] == "restart":  # every byte comes from one checkpoint of the chain, and is written once
        n = -(-case["nbytes"] // case["chunk"])
        return {"bytes": 2 * case["nbytes"] + 8 * case["rate"] * n * (case["steps"] + 1), "flops": 0}
    if case["kind"] == "batch":
        return {"bytes": sum(_series_bytes(m["nbytes"], m["chunk"], m["steps"], m["rate"]) for m in _members(case, 0)),
                "flops": 0}
    return {"bytes": _series_bytes(case["nbytes"], case["chunk"], case["steps"], case["rate"]), "flops": 0}


def exact(case, seed):
    """A restart gives back the buffer that the application wrote; digests and
    checkpoints are whole numbers that have no other value than the library's."""
    if case["kind"] != "restart":
        return None
    last = None
    for last in _states(case, seed):
        pass
    return last
