"""Chunk digests of a partial last chunk beside whole ones (chunk sizes that are
box widths, 16-byte aligned buffers): tails at the edges of words, of 16 bytes,
of 64-byte pieces and of the chunk, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("cs,tails", [(16, (1, 3, 8, 9, 15)), (32, (1, 16, 17, 31)), (64, (1, 4, 47, 55, 56, 63)),
                                      (128, (1, 63, 64, 65, 120, 127)),
                                      (4096, (1, 64, 127, 128, 129, 191, 192, 1000, 3840, 4087, 4095))])
def test_tail_digests(cuda, mtc, oracle, kind, cs, tails):
    rng = np.random.default_rng(cs)
    for tail in tails:
        host = rng.integers(0, 256, 3 * cs + tail, dtype=np.uint8)
        buf = cuda.empty(host.size + 64, dtype=cuda.uint8, device="cuda")
        buf.fill_(0xa5)  # what follows the buffer is not hashed
        buf[:host.size].copy_(cuda.from_numpy(host))
        got = mtc.hash_chunks(kind, buf[:host.size], cs).cpu().numpy().reshape(-1, 16)
        for c in range(4):
            assert got[c].tobytes() == bytes(oracle.digest(host[c * cs:(c + 1) * cs], kind)), (tail, c)
