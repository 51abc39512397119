"""The streams and device memory kept between calls, shared by several threads and given back while
calls are in flight: residues stay those of lone calls, and batches that are launched again, or
destroyed without being read, leave nothing behind that a later call would see."""
import threading

import pytest

pytestmark = pytest.mark.gpu


def test_release_while_threads_call(gpu, oracle):
    ps = [61, 127, 251, 257, 521, 1279, 2203, 9689, 36847, 44497]
    want = {p: oracle.ll_gmp(p, min(p - 2, 400))[2] for p in ps}
    bad, stop = [], threading.Event()

    def caller(k):
        for i in range(12):
            p = ps[(i * 7 + k) % len(ps)]
            got = gpu.run(p, iters=400, want_words=True)["words"]
            if got != want[p]:
                bad.append(("run", p))
            batch = ps[k % 3::3]
            for p, r in zip(batch, gpu.run_batch(batch, iters=400, want_words=True)):
                if r["words"] != want[p]:
                    bad.append(("batch", p))

    def releaser():
        while not stop.is_set():
            gpu.release_cached()

    threads = [threading.Thread(target=caller, args=(k,)) for k in range(6)]
    extra = threading.Thread(target=releaser)
    extra.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    extra.join()
    assert not bad


def test_batch_again_and_unread(gpu, oracle):
    ps = [2, 4, 127, 521, 2203, 9689, 44497]
    b = gpu.Batch(ps, 300, flags=gpu.Batch.KEEP_WORDS)
    try:
        for _ in range(3):
            b.launch()
            for p, r in zip(ps, b.results(want_words=True)):
                if p > 4:
                    assert r["words"] == oracle.ll_gmp(p, min(p - 2, 300))[2], p
    finally:
        b.close()
    unread = gpu.Batch(ps, 300)
    unread.launch()
    unread.close()
    assert gpu.run(9689, iters=300, want_words=True)["words"] == oracle.ll_gmp(9689, 300)[2]
