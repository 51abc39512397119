"""A resident two-pass test started again on the same object: the epochs, and with them the tags of
the carries that row tiles hand on, begin anew, and nothing the earlier run published may be taken
for the new run's. Reads in between resume at the same epoch. Against plain integers (the longer lengths:
against a fresh test on the exact NTT engine)."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _square_on(s, p, k):
    m = (1 << p) - 1
    for _ in range(k):
        s = s * s - 2
        while s > m:
            s = (s & m) + (s >> p)
        if s < 0:
            s += m
    return 0 if s == m else s


def _words(gpu, s, p):
    b = s.to_bytes(8 * gpu.nwords(p), "little")
    return [int.from_bytes(b[i:i + 8], "little") for i in range(0, len(b), 8)]


# the smallest length, the first that lets the next pass launch late, a one-wave and a several-wave
# one, and the R0 x 2^k length whose tiles run at five blocks an SM
@pytest.mark.parametrize("engine,n", [("fp64", 1 << 14), ("fp64", 1 << 17), ("fp64", 1 << 18), ("fp64", 1 << 19),
                                      ("fp64", 5 << 18), ("ntt", 1 << 14), ("ntt", 1 << 17)])
def test_restarted_test_repeats_exactly(gpu, engine, n):
    p = int(16.3 * n) | 1
    rng = random.Random(n)
    t = gpu.Test(p, n, engine=engine)
    try:
        for _ in range(3):
            s = rng.getrandbits(p)
            words = _words(gpu, s, p)
            t.load(words, 7)
            mid = t.read()
            t.iterate(1)
            again = t.read(want_words=True)
            if n <= 1 << 17:
                first = _square_on(s, p, 1)
                want = (first & (2**64 - 1), _words(gpu, _square_on(first, p, 1), p))
            else:
                u = gpu.Test(p, 0, engine="ntt")
                u.load(words, 7)
                first = u.read()["res64"]
                u.iterate(1)
                want = (first, u.read(want_words=True)["words"])
                u.close()
            assert (mid["res64"], again["words"]) == want
    finally:
        t.close()
