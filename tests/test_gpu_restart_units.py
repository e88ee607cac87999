"""The restart copy in 16-byte units: chunk sizes around and below a word, no
multiple of one, and outputs that start anywhere; bytes the chain does not
restore keep what the buffer held."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FILL = 0xA5


@pytest.mark.parametrize("approach", [2, 3, 4], ids=["basic", "list", "tree"])
@pytest.mark.parametrize("offset", [0, 1, 8])
@pytest.mark.parametrize("cs,n,tail", [(1, 100, 0), (7, 64, 3), (15, 33, 0), (16, 70, 5), (17, 97, 16), (100, 64, 0), (100, 161, 9),
                                       (129, 40, 1), (640, 33, 600), (5000, 9, 0)])
def test_restart_units(cuda, mtc, oracle, approach, offset, cs, n, tail):
    if approach == 4:  # a power of two of whole chunks, of which a tree restart gives every one back
        n, tail = 1 << (n.bit_length() - 1), 0
    nbytes = cs * n - (cs - tail if tail else 0)
    rng = np.random.default_rng(cs * 31 + n)
    state = rng.integers(0, 256, nbytes, dtype=np.uint8)
    gpu, diffs = mtc.Deduplicator(cs, 0, approach=approach), []
    for step in range(4):
        diffs.append(gpu.checkpoint(cuda.from_numpy(state).cuda(), step == 0))
        a, b = (int(x) * cs for x in rng.integers(0, n - 1, 2))
        state[a:a + cs] = state[b:b + cs].copy()
        state[int(rng.integers(0, nbytes))] ^= 0x55
    for i in range(4):
        want = np.full(nbytes, FILL, np.uint8)
        assert oracle.restart(approach, diffs[: i + 1], i, want) == 0
        buf = cuda.full((nbytes + 32,), FILL, dtype=cuda.uint8, device="cuda")
        gpu.restart(buf[offset:offset + nbytes], diffs, i)
        got = buf.cpu().numpy()
        assert np.array_equal(got[offset:offset + nbytes], want), i
        assert (got[:offset] == FILL).all() and (got[offset + nbytes:] == FILL).all(), i
