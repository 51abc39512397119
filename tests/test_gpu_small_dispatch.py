"""The whole-test FP64 kernel takes more threads a test when each test has its SM to itself: both
forms at every length, full residues against each other and the oracle, and the
per-squaring round-off log of the form that runs in one warp."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1 << k for k in range(5, 14)] + [3072, 5120, 6144, 10240, 12288])
def test_alone_and_batch_forms_agree(gpu, oracle, n):
    sms = gpu.device_info()[1]
    lo = max(257, int(17.2 * n))
    ps = [p for p in range(lo | 1, 18 * n) if p % 2 and gpu.fft_length(p) == n]
    if len(ps) <= sms:  # the shortest lengths hold few exponents: repeat them
        ps = (ps or [18 * n - 1]) * (sms // max(1, len(ps)) + 1)
    ps = ps[: sms + 1]
    k = 40
    batch = gpu.run_batch(ps, iters=k, want_words=True)      # one test too many for one per SM
    alone = gpu.run_batch(ps[:3], iters=k, want_words=True)  # one test per SM
    for p, a, b in zip(ps[:3], alone, batch):
        assert a["status"] == b["status"] == 0 and a["n"] == b["n"] == n
        assert a["words"] == b["words"] == oracle.ll_gmp(p, k)[2], (p, n)
    assert batch[-1]["words"] == oracle.ll_gmp(ps[-1], k)[2]


@pytest.mark.parametrize("p", [521, 2203, 4423, 9689])  # N = 32, 128, 256 (one warp), 1024
def test_errlog_of_every_squaring(gpu, p):
    b = gpu.Batch([p], 200, flags=gpu.Batch.ERRLOG)
    try:
        b.launch()
        r = b.results()[0]
        log = b.errlog()
    finally:
        b.close()
    assert len(log) == 200 and all(0.0 <= e < 0.5 for e in log)
    assert max(log) == pytest.approx(r["max_err"], rel=1e-6)
    assert sum(e > 0 for e in log) > 150  # every squaring but the first few, whose digits are tiny
