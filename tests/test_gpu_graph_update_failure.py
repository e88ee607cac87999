"""A failing query or update of a captured sequence's nodes (injected on the host):
the call reports it, and no later call replays a sequence of which only some
nodes follow the input.  Every checkpoint that succeeds is the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CS = 128


def states(rng, n, count):
    state = rng.integers(0, 256, (n, CS), dtype=np.uint8)
    for _ in range(count):
        yield state.reshape(-1).copy()
        pick = rng.random(n) < 0.1
        state[pick] = rng.integers(0, 256, (int(pick.sum()), CS), dtype=np.uint8)


@pytest.mark.parametrize("approach", [2, 3, 4], ids=["basic", "list", "tree"])
@pytest.mark.parametrize("op", range(1, 10))
def test_lone_handle(cuda, mtc, oracle, monkeypatch, approach, op):
    monkeypatch.setenv("MTCHECK_FAIL_GRAPH_OP", str(op))
    ref, gpu = oracle.Deduplicator(approach, CS, 0), mtc.Deduplicator(CS, 0, approach=approach)
    monkeypatch.delenv("MTCHECK_FAIL_GRAPH_OP")
    n, failed = 1000, 0
    bufs = [cuda.zeros(n * CS, dtype=cuda.uint8, device="cuda") for _ in range(2)]
    for step, state in enumerate(states(np.random.default_rng(op), n, 9)):
        buf = bufs[(0, 0, 1, 0, 1, 1, 0, 1, 0)[step]]
        buf.copy_(cuda.from_numpy(state))
        try:
            got = gpu.checkpoint(buf, step == 0)
        except mtc.MtcError:
            failed += 1
            continue
        assert got == ref.checkpoint(state, step == 0), step
    assert failed == 1


@pytest.mark.parametrize("op", range(1, 6))
def test_batch(cuda, mtc, oracle, monkeypatch, op):
    monkeypatch.setenv("MTCHECK_FAIL_GRAPH_OP", str(op))
    sizes = (1000, 5000)
    batch = mtc.Batch([(4, 0, CS) for _ in sizes])
    monkeypatch.delenv("MTCHECK_FAIL_GRAPH_OP")
    refs = [oracle.Deduplicator(4, CS, 0) for _ in sizes]
    bufs = [[cuda.zeros(n * CS, dtype=cuda.uint8, device="cuda") for n in sizes] for _ in range(3)]
    failed = 0
    for step, row in enumerate(zip(*[states(np.random.default_rng(n), n, 9) for n in sizes])):
        for buf, state in zip(bufs[step % 3], row):
            buf.copy_(cuda.from_numpy(state))
        try:
            batch.checkpoint(bufs[step % 3], make_baseline=step == 0)
        except mtc.MtcError:
            failed += 1
            continue
        for m, ref, state in zip(batch.members, refs, row):
            host = np.empty(m.diff_device()[1], np.uint8)
            m.copy_diff(host)
            assert host.tobytes() == ref.checkpoint(state, step == 0), step
    assert failed == len(sizes)
    batch.close()
