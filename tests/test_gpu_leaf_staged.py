"""Chunk digests through the hashing kernels for chunk sizes that are no box width
and buffers off a 16-byte boundary (whole tiles, staged panels, direct reads) at
the edges of their tiles, panels, words and ranges, against the oracle; and a
checkpoint series on such a buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("offset", [0, 1, 4, 8, 15])
@pytest.mark.parametrize("cs,n,tail", [(1, 300, 0), (15, 128, 0), (24, 129, 7), (63, 257, 0), (64, 130, 63), (100, 1, 0),
                                       (100, 385, 99), (127, 127, 1), (128, 128, 5), (129, 131, 128), (192, 200, 0),
                                       (255, 129, 64), (300, 64, 1), (512, 257, 511), (4096, 130, 200), (5000, 3, 4999),
                                       (48, 257, 47), (65, 128, 64), (436, 129, 3), (440, 257, 0), (441, 129, 2)])
def test_staged_digests(cuda, mtc, oracle, kind, offset, cs, n, tail):
    nbytes = cs * n - (cs - tail if tail else 0)
    host = np.random.default_rng(cs * 7 + n).integers(0, 256, nbytes, dtype=np.uint8)
    buf = cuda.empty(nbytes + offset, dtype=cuda.uint8, device="cuda")[offset:]
    buf.copy_(cuda.from_numpy(host))
    got = mtc.hash_chunks(kind, buf, cs).cpu().numpy().reshape(-1, 16)
    for c in range(n):
        assert got[c].tobytes() == bytes(oracle.digest(host[c * cs:(c + 1) * cs], kind)), c


@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("cs,offset,n", [(100, 0, 500_003), (100, 3, 500_003), (436, 8, 100_000), (24, 0, 1_000_001)])
def test_many_tiles(cuda, mtc, oracle, kind, cs, offset, n):
    # several tiles per block, so that every stage is filled again; a sample of the chunks
    nbytes = cs * n - 5
    host = np.random.default_rng(n).integers(0, 256, nbytes, dtype=np.uint8)
    buf = cuda.empty(nbytes + offset, dtype=cuda.uint8, device="cuda")[offset:]
    buf.copy_(cuda.from_numpy(host))
    got = mtc.hash_chunks(kind, buf, cs).cpu().numpy().reshape(-1, 16)
    for c in [*np.random.default_rng(1).integers(0, n, 2000), 0, n - 2, n - 1]:
        assert got[c].tobytes() == bytes(oracle.digest(host[c * cs:(c + 1) * cs], kind)), c


@pytest.mark.parametrize("approach", [2, 3, 4], ids=["basic", "list", "tree"])
@pytest.mark.parametrize("cs,offset", [(256, 4), (100, 1), (40, 0)])
def test_staged_series(cuda, mtc, oracle, approach, cs, offset):
    nbytes = cs * 700 + 17
    rng = np.random.default_rng(cs)
    state = rng.integers(0, 256, nbytes, dtype=np.uint8)
    ref, gpu = oracle.Deduplicator(approach, cs, 0), mtc.Deduplicator(cs, 0, approach=approach)
    bufs = [cuda.empty(nbytes + offset + 16 * i, dtype=cuda.uint8, device="cuda")[offset + 16 * i:] for i in range(2)]
    for step in range(4):  # the replayed sequence follows a moved input
        bufs[step % 2].copy_(cuda.from_numpy(state))
        assert gpu.checkpoint(bufs[step % 2], step == 0) == ref.checkpoint(state, step == 0), step
        state[int(rng.integers(0, nbytes))] ^= 1
        state[cs * 5:cs * 9] = state[cs * 20:cs * 24].copy()
