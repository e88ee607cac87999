"""The chunk gather at the edges of its tiles: slot counts around a tile's,
chunks shorter than a word, longer than a tile, no multiple of a word, buffers
that start anywhere, one long region, single chunks and short runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("approach", [2, 3, 4], ids=["basic", "list", "tree"])
@pytest.mark.parametrize("cs,n,tail,offset", [
    (128, 256, 0, 0), (128, 257, 5, 0), (128, 1023, 127, 4), (64, 513, 1, 0), (16, 700, 9, 0), (4096, 17, 4000, 16),
    (100, 256, 0, 0), (100, 769, 99, 1), (127, 300, 3, 8), (129, 600, 1, 0), (640, 130, 0, 4), (1, 700, 0, 0),
    (7, 523, 4, 3), (15, 257, 2, 0), (32768, 5, 1, 0), (40000, 9, 39999, 2), (40000, 1, 0, 0),
])
def test_gather_tile_edges(cuda, mtc, oracle, approach, cs, n, tail, offset):
    nbytes = cs * n - (cs - tail if tail else 0)
    rng = np.random.default_rng(cs * 1000 + n)
    state = rng.integers(0, 256, nbytes, dtype=np.uint8)
    ref, gpu = oracle.Deduplicator(approach, cs, 0), mtc.Deduplicator(cs, 0, approach=approach)
    buf = cuda.empty(nbytes + offset + 16, dtype=cuda.uint8, device="cuda")[offset:offset + nbytes]
    for step in range(4):
        buf.copy_(cuda.from_numpy(state))
        assert gpu.checkpoint(buf, step == 0) == ref.checkpoint(state, step == 0), step
        # single chunks and runs, the last chunk among them every second time
        for c in rng.integers(0, n, max(1, n // 7)):
            state[c * cs:(c + 1 + int(c) % 3) * cs] ^= 1 + step
        if step % 2:
            state[-1] ^= 0x80
