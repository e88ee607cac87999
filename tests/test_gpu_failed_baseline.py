"""A baseline that fails for want of device memory leaves no state to go on from:
the next checkpoint, whatever was asked for, is a baseline of its own buffer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CS, N = 1 << 20, 6


@pytest.mark.parametrize("approach", [2, 3, 4, 5], ids=["basic", "list", "tree", "tree_ref"])
@pytest.mark.parametrize("before", [0, 2], ids=["first", "later"])
def test_next_checkpoint_is_a_baseline(cuda, mtc, oracle, approach, before):
    rng = np.random.default_rng(approach)
    ref, gpu = oracle.Deduplicator(approach, CS, 0), mtc.Deduplicator(CS, 0, approach=approach)

    def step(baseline, want_baseline):
        state = rng.integers(0, 256, CS * N - 100, dtype=np.uint8)
        got = gpu.checkpoint(cuda.from_numpy(state).cuda(), baseline)
        assert got == ref.checkpoint(state, want_baseline)

    for i in range(before):
        step(i == 0, i == 0)
    buf = cuda.zeros(64, dtype=cuda.uint8, device="cuda")
    # 4 TiB: refused while its buffers are allocated, before anything reads it
    with pytest.raises(mtc.MtcError) as e:
        gpu.checkpoint_device((buf.data_ptr(), 1 << 42), True)
    assert e.value.code == 3
    step(False, True)
    step(False, False)
