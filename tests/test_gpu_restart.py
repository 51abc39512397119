"""A resident two-pass test started again on the same object: the epochs, and with them the tags of
the carries that row tiles hand on, begin anew, and nothing the earlier run published may be taken
for the new run's. Reads in between resume at the same epoch. Against plain integers."""
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
            words = [(s >> (64 * i)) & (2**64 - 1) for i in range(gpu.nwords(p))]
            t.load(words, 7)
            mid = t.read()
            t.iterate(1)
            again = t.read(want_words=True)
            want = _square_on(s, p, 1)
            assert mid["res64"] == want & (2**64 - 1)
            want = _square_on(want, p, 1)
            assert sum(w << (64 * i) for i, w in enumerate(again["words"])) == want
    finally:
        t.close()
