"""Buffers that keep digests of their own chunks: a 32-byte chunk equal to the
pair of digests an interior node hashes has that node's digest, so leaves and
interior nodes, and first occurrences of two depths, meet in the map.  Which of
them owns the digest (and is a region of the diff) is the serial order's to
decide: the oracle's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CS = 32


def pair(oracle, kind, x, y):
    return np.frombuffer(oracle.digest(x.tobytes(), kind) + oracle.digest(y.tobytes(), kind), np.uint8)


def groups(rng, n, count):
    """Leaves (a, b, z1, z2) under one node two levels up and two sibling leaves
    (c, y) elsewhere: chunks c = [a b] and y = [z1 z2] give the node above c and y
    the digest of the node above the four."""
    first = n - 1  # node of leaf 0
    out = []
    for _ in range(20 * count):
        k, q = (int(x) | 1 for x in rng.integers(first, 2 * n - 2, 2))  # left children
        p = (k - 1) // 2
        four = (2 * p + 1 - first, 2 * p + 2 - first, 2 * p + 3 - first, 2 * p + 4 - first)
        c = q - first
        if p % 2 == 0 or four[0] < 0 or four[3] >= n or c < 0 or c + 1 >= n or c in four:
            continue
        out.append((four, c))
        if len(out) == count:
            break
    return out


def states(oracle, kind, n, seed):
    """Six states of n chunks with planted groups; a third of them get their digests
    a step before their data, which then also come as moved chunks."""
    rng = np.random.default_rng(seed)
    few = rng.integers(0, 256, (5, CS), dtype=np.uint8)
    rows = few[rng.integers(0, 5, n)]  # mostly duplicates: the planted nodes are roots
    later = []
    for _ in range(6):
        for (a, b, z1, z2), c, content in later:
            rows[[a, b, z1, z2]] = content
            d = groups(rng, n, 1)
            if d:
                rows[d[0][1]:d[0][1] + 2] = rows[c:c + 2].copy()
        later = []
        for i, (four, c) in enumerate(groups(rng, n, max(1, min(200, n // 64)))):
            content = rng.integers(0, 256, (4, CS), dtype=np.uint8)
            rows[c], rows[c + 1] = pair(oracle, kind, *content[:2]), pair(oracle, kind, *content[2:])
            if i % 3 == 2:
                later.append((four, c, content))
            else:
                rows[list(four)] = content
        yield rows.reshape(-1).copy()


@pytest.mark.parametrize("kind", [0, 1], ids=["murmur3", "md5"])
@pytest.mark.parametrize("approach", [4, 5, 6], ids=["tree", "tree_ref", "tree_low_offset"])
@pytest.mark.parametrize("n", [8, 64, 2048, 2049, 5000, 40000, 1 << 18])
def test_chunks_of_digest_pairs(cuda, mtc, oracle, approach, kind, n):
    if n > 40000 and (approach != 4 or kind):
        pytest.skip("one large tree is enough: its inserts may run on a second stream")
    if approach == 5 and n & (n - 1):
        pytest.skip("leaves on two levels put both nodes of a pair on one, where this approach's reference goes down")
    ref, gpu = oracle.Deduplicator(approach, CS, kind), mtc.Deduplicator(CS, kind, approach=approach)
    for step, state in enumerate(states(oracle, kind, n, n + approach)):
        baseline = step in (0, 4)
        want = ref.checkpoint(state, baseline)
        assert gpu.checkpoint(cuda.from_numpy(state).cuda(), baseline) == want, step


def test_batch_of_digest_pairs(cuda, mtc, oracle):
    """Members of a batch, whose later checkpoints are replayed inside its graph."""
    sizes, kinds = (64, 3000, 20000), (0, 1, 0)
    batch = mtc.Batch([(4, k, CS) for k in kinds])
    refs = [oracle.Deduplicator(4, CS, k) for k in kinds]
    for step, row in enumerate(zip(*[states(oracle, k, n, n) for k, n in zip(kinds, sizes)])):
        batch.checkpoint([cuda.from_numpy(s).cuda() for s in row], make_baseline=step == 0)
        for m, ref, state in zip(batch.members, refs, row):
            host = np.empty(m.diff_device()[1], np.uint8)
            m.copy_diff(host)
            assert host.tobytes() == ref.checkpoint(state, step == 0), step
    batch.close()


@pytest.mark.parametrize("n", [8, 300, 5000])
def test_last_chunk_of_a_digest_pair(cuda, mtc, oracle, n):
    """Longer chunks, the partial last one a pair of digests."""
    cs = 128
    rng = np.random.default_rng(n)
    few = rng.integers(0, 256, (3, cs), dtype=np.uint8)
    state = np.empty(n * cs + 32, np.uint8)
    rows = state[:n * cs].reshape(n, cs)
    rows[:] = few[rng.integers(0, 3, n)]
    ref, gpu = oracle.Deduplicator(4, cs, 0), mtc.TreeDeduplicator(cs)
    for step in range(4):
        a = int(rng.integers(0, (n - 2) // 2)) * 2
        a += (n + a + 1) % 2  # node n + a (n + 1 leaves) is a left child
        rows[a:a + 2] = rng.integers(0, 256, (2, cs), dtype=np.uint8)
        state[n * cs:] = pair(oracle, 0, rows[a], rows[a + 1])
        want = ref.checkpoint(state, step in (0, 2))
        assert gpu.checkpoint(cuda.from_numpy(state.copy()).cuda(), step in (0, 2)) == want, step


@pytest.mark.parametrize("use_graph", [True, False], ids=["graph", "eager"])
def test_served_digest_pairs(cuda, mtc, oracle, use_graph):
    srv = mtc.Server(use_graph=use_graph)
    pid, ref = srv.add_process(4, 0, CS), oracle.Deduplicator(4, CS, 0)
    for step, state in enumerate(states(oracle, 0, 5000, 5)):
        buf = cuda.from_numpy(state).cuda()
        srv.submit_checkpoint(pid, buf, make_baseline=step == 0)
        srv.drain()
        assert srv.diff(pid, step) == ref.checkpoint(state, step == 0), step
    srv.close()
