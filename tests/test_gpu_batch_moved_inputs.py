"""A batch's counters tell inputs that moved, which its graph follows in place,
from sequences that were captured again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CS, SIZES, STEPS = 128, (1000, 3000, 5000), 6


@pytest.mark.parametrize("moving", [(), (1,), (0, 1, 2)], ids=["none", "one", "all"])
def test_moved_inputs(cuda, mtc, moving):
    rng = np.random.default_rng(1)
    batch = mtc.Batch([(2, 0, CS) for _ in SIZES])  # basic: no map that grows
    bufs = [cuda.from_numpy(rng.integers(0, 256, n * CS, dtype=np.uint8)).cuda() for n in SIZES]
    kept = list(bufs)
    for step in range(STEPS):
        if step:
            bufs = [b.clone() if i in moving else b for i, b in enumerate(bufs)]
            kept += bufs  # no address comes back
        batch.checkpoint(bufs, make_baseline=step == 0)
    # captured in the first increment with that step's buffers, moved in the others
    assert batch.moved_inputs() == (STEPS - 2) * len(moving)
    assert batch.info().graph_captures - batch.moved_inputs() == len(SIZES)
    batch.close()
