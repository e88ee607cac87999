"""Checkpoints whose changed chunks repeat each other's and earlier contents, so
that inserts of one digest meet within a warp, a block and the launch: the
lowest chunk keeps the entry and every other one is a shifted duplicate, in the
oracle's bytes.  Also with the id not advanced, where entries of earlier calls
carry the current id."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approach,advance", [(3, True), (4, True), (5, True), (3, False), (4, False)],
                         ids=["list", "tree", "tree_ref", "list-same_id", "tree-same_id"])
@pytest.mark.parametrize("n,palette", [(2, 1), (33, 1), (64, 3), (700, 40), (3000, 1), (20000, 7), (20000, 6000)])
def test_insert_duplicates(cuda, mtc, oracle, approach, advance, n, palette):
    cs = 64
    rng = np.random.default_rng(n + palette)
    colours = rng.integers(0, 256, (palette, cs), dtype=np.uint8)
    state = rng.integers(0, 256, (n, cs), dtype=np.uint8)
    ref, gpu = oracle.Deduplicator(approach, cs, 0), mtc.Deduplicator(cs, 0, approach=approach)
    for step in range(5):
        want = ref.checkpoint(state.reshape(-1), step == 0, increment=advance)
        got = gpu.checkpoint(cuda.from_numpy(state.reshape(-1).copy()).cuda(), step == 0, advance=advance)
        assert got == want, step
        old = state.copy()
        pick = rng.random(n) < (0.3, 0.9, 0.1, 0.5)[step % 4]
        state[pick] = colours[rng.integers(0, palette, int(pick.sum()))]
        if step == 1:  # a run, and chunks of earlier steps moved down and up
            state[n // 4:n // 2] = colours[0]
        if step >= 2:
            state[n // 2:] = old[rng.integers(0, n, n - n // 2)]


@pytest.mark.parametrize("copies", [1, 2, 5])
def test_list_bins_of_many_checkpoints(cuda, mtc, oracle, copies):
    """A few shift entries with sources among many checkpoints: the sort's bins are
    fewer than the keys, so keys share them."""
    cs, n = 64, 400
    rng = np.random.default_rng(copies)
    state = rng.integers(0, 256, (n, cs), dtype=np.uint8)
    ref, gpu = oracle.Deduplicator(3, cs, 0), mtc.Deduplicator(cs, 0, approach=3)
    for step in range(220):
        want = ref.checkpoint(state.reshape(-1), step == 0)
        assert gpu.checkpoint(cuda.from_numpy(state.reshape(-1).copy()).cuda(), step == 0) == want, step
        old = state.copy()
        state[step] = rng.integers(0, 256, cs, dtype=np.uint8)  # this checkpoint's own content
        state[300 + rng.choice(100, copies, replace=False)] = old[rng.integers(0, step + 1, copies)]
