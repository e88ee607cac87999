"""mtc_hash_chunks from many host threads: calls that run at one time do not
share their error words, and a thread that ends leaves nothing behind."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def resident_kb():
    return next(int(line.split()[1]) for line in open("/proc/self/status") if line.startswith("VmRSS"))


def test_ended_threads_leave_nothing(cuda, mtc):
    buf = cuda.zeros(4096, dtype=cuda.uint8, device="cuda")
    out = cuda.empty(512, dtype=cuda.uint8, device="cuda")

    def calls(count):
        for _ in range(count):
            t = threading.Thread(target=mtc.hash_chunks, args=(0, buf, 128, out))
            t.start()
            t.join()

    calls(200)
    before = resident_kb()
    calls(2000)
    # a pinned word and a device word kept by each thread: 2.7 KB of the driver's
    # memory, 5 MB in all
    assert resident_kb() - before < 1500


def test_threads_at_once(cuda, mtc, oracle):
    cs, n = 100, 3000
    hosts = [np.random.default_rng(i).integers(0, 256, cs * n, dtype=np.uint8) for i in range(8)]
    bufs = [cuda.from_numpy(h).cuda() for h in hosts]
    outs = [cuda.empty(16 * n, dtype=cuda.uint8, device="cuda") for _ in hosts]
    streams = [cuda.cuda.Stream() for _ in hosts]
    cuda.cuda.synchronize()
    wrong = []

    def work(i):
        try:
            for _ in range(50):
                mtc.hash_chunks(i & 1, bufs[i], cs, out=outs[i], stream=streams[i].cuda_stream)
            got = outs[i].cpu().numpy().reshape(n, 16)
            wrong.extend((i, c) for c in range(0, n, 7)
                         if got[c].tobytes() != bytes(oracle.digest(hosts[i][c * cs:(c + 1) * cs], i & 1)))
        except Exception as e:
            wrong.append((i, e))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(hosts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
