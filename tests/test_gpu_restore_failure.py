"""A restore of a spilled state that fails (injected on the host) is reported, and
the state stays spilled, whole: the process's later requests are served as if the
failed one had not been made."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# (approach, hash, chunk size, bytes)
PROCS = [(4, 0, 128, 1 << 20), (3, 0, 512, 3 << 19), (2, 1, 256, 1 << 20), (4, 1, 512, 1 << 20), (5, 0, 128, 1 << 19)]
STEPS = 5


def test_failed_restore_is_retried(cuda, mtc, oracle, monkeypatch):
    monkeypatch.setenv("MTCHECK_FAIL_RESTORE", "1")
    srv = mtc.Server(hbm_budget=8 << 20, max_inflight=1)  # one or two of the states fit
    pids = [srv.add_process(a, h, cs) for a, h, cs, _ in PROCS]
    monkeypatch.delenv("MTCHECK_FAIL_RESTORE")
    refs = [oracle.Deduplicator(a, cs, h) for a, h, cs, _ in PROCS]
    rng = np.random.default_rng(1)
    states = [rng.integers(0, 256, n, dtype=np.uint8) for *_, n in PROCS]
    failed = 0
    for step in range(STEPS):
        for i, pid in enumerate(pids):
            at = rng.integers(0, states[i].size - 3000, 40)
            for x in at:
                states[i][x] ^= 1
            a, b = at[:2]
            states[i][a:a + 3000] = states[i][b:b + 3000].copy()
            buf = cuda.from_numpy(states[i]).cuda()
            while True:
                srv.submit_checkpoint(pid, buf, make_baseline=step == 0)
                done = []
                while not done:
                    done = srv.poll(wait_ms=100)
                if done[0]["status"] == 0:
                    break
                failed += 1
                assert failed <= len(PROCS), (step, i, done)
            assert srv.diff(pid, step) == refs[i].checkpoint(states[i], step == 0), (step, i)
    st = srv.stats()
    assert st["restored_states"] > 0 and 0 < failed == st["failed"]
    srv.close()
