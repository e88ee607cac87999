"""A baseline's forest in one traversal, at the edges of its spans and with the
contents that decide its labels: unique chunks, runs of equal chunks, aligned
copies (pairs of shifted duplicates) and scattered copies.  The checkpoint that
follows copies runs of old chunks, so that its sources are the interior nodes
the baseline put into the map."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("content", ["unique", "zeros", "aligned", "scattered"])
@pytest.mark.parametrize("n", [2, 3, 64, 511, 2047, 2048, 2049, 4096, 4100, 8191, 12289, 40000])
def test_baseline_forest(cuda, mtc, oracle, kind, content, n):
    cs = 32
    rng = np.random.default_rng(n + 7 * kind)
    state = rng.integers(0, 256, n * cs, dtype=np.uint8)
    rows = state.reshape(n, cs)
    if content == "zeros":
        rows[n // 4:n // 4 + n // 2] = 0
    elif content == "aligned":
        k = 1 << max(0, (n // 4).bit_length() - 1)
        rows[n - k:] = rows[:k]
        rows[k:2 * k] = rows[:k]
    elif content == "scattered":
        dst = rng.integers(n // 2, n, n // 5 + 1)
        rows[dst] = rows[rng.integers(0, n // 2 + 1, dst.size)]
    ref, gpu = oracle.Deduplicator(4, cs, kind), mtc.TreeDeduplicator(cs, kind)

    def step(baseline):
        assert gpu.checkpoint(cuda.from_numpy(state).cuda(), baseline) == ref.checkpoint(state, baseline)

    step(True)
    for rep in range(2):
        for _ in range(4):
            ln = int(rng.integers(1, max(2, n // 8)))
            a, b = (int(x) for x in rng.integers(0, n - ln + 1, 2))
            rows[a:a + ln] = rows[b:b + ln].copy()
        step(False)
    step(True)  # on the buffers of the first one
    rows[: n // 3 + 1] = rows[n - n // 3 - 1:].copy()
    step(False)
