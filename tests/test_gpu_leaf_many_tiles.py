"""The hashing kernels with several tiles per block, so that stages are filled
again, rows at a tile's edge come from inner tiles and the changed chunks of one
tile wait for the next: digests of a sample of the chunks against the oracle on
both sides of the lines between the staged and the direct kernel, and series
whose increments change a few percent."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffer(cuda, host, offset):
    buf = cuda.empty(host.size + offset, dtype=cuda.uint8, device="cuda")[offset:]
    buf.copy_(cuda.from_numpy(host))
    return buf


# staged: 512 chunks per SM at a time; boxes off a boundary: up to 768
@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("cs,offset,per_sm,n", [
    (441, 0, 512, 100_003), (441, 3, 512, 100_003), (160, 1, 512, 170_003), (192, 4, 512, 100_003), (448, 8, 512, 160_001),
    (600, 8, 512, 100_003),                                  # staged
    (160, 4, 256, 77_000), (160, 4, 512, 170_003), (516, 0, 256, 50_001), (516, 0, 512, 240_001), (1004, 0, 384, 60_001),
    (1004, 0, 1536, 240_001), (2004, 0, 768, 120_001), (504, 0, 512, 80_003),  # read directly, or either side of it
    (64, 4, 768, 200_003), (128, 8, 768, 200_003), (128, 1, 768, 130_001)])     # boxes
def test_digests(cuda, mtc, oracle, kind, cs, offset, per_sm, n):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    assert n > per_sm * sms, "more chunks than are in flight at once"
    host = np.random.default_rng(n).integers(0, 256, cs * n - 5, dtype=np.uint8)
    got = mtc.hash_chunks(kind, buffer(cuda, host, offset), cs).cpu().numpy().reshape(-1, 16)
    for c in [*np.random.default_rng(1).integers(0, n, 2000), 0, n - 2, n - 1]:
        assert got[c].tobytes() == bytes(oracle.digest(host[c * cs:(c + 1) * cs], kind)), c


@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("approach", [3, 4], ids=["list", "tree"])
@pytest.mark.parametrize("cs,offset,n", [(100, 1, 400_003), (64, 4, 200_003), (441, 1, 100_003), (516, 4, 100_003)])
def test_series(cuda, mtc, oracle, approach, kind, cs, offset, n):
    rng = np.random.default_rng(cs)
    state = rng.integers(0, 256, cs * n - 7, dtype=np.uint8)
    ref, gpu = oracle.Deduplicator(approach, cs, kind), mtc.Deduplicator(cs, kind, approach=approach)
    for step in range(3):
        got = gpu.checkpoint(buffer(cuda, state, offset), step == 0)
        assert got == ref.checkpoint(state, step == 0), step
        for c in rng.integers(0, n - 1, n // 30):  # single chunks
            state[c * cs] ^= 1
        a, b = rng.integers(0, n - 3000, 2)  # and a moved run
        state[a * cs:(a + 2000) * cs] = state[b * cs:(b + 2000) * cs].copy()
