"""The two-pass NTT engine from residues whose digits sit at the edges of the carry (all ones, one,
minus one, alternating runs, a lone top digit), one and two squarings on, against plain integers."""
import random

import pytest

pytestmark = pytest.mark.gpu


def _residues(p):
    m = (1 << p) - 1
    rng = random.Random(p)
    return {
        "one": 1,
        "minus one": m - 1,
        "zero as 2^p - 1": m,
        "top bit": 1 << (p - 1),
        "alternating": int("01" * (p // 2 + 1), 2) & m,
        "runs": int(("0" * 61 + "1" * 67) * (p // 128 + 1), 2) & m,
        "random": rng.getrandbits(p),
    }


# N = 2^14: rows of 2^7 (one warp row group); 2^16: 2^8; 2^17: 2^8 rows of 2^9 columns; the widest
# digits the field holds and about 9 bits
@pytest.mark.parametrize("logn,bits", [(14, 24), (14, 9), (16, 23), (17, 9)])
def test_ntt_two_pass_edge_digits(gpu, logn, bits):
    n = 1 << logn
    p = bits * n - 1
    m = (1 << p) - 1
    t = gpu.Test(p, n, engine="ntt")
    try:
        for name, s in _residues(p).items():
            words = [(s >> (64 * i)) & (2**64 - 1) for i in range(gpu.nwords(p))]
            t.load(words, 1)
            t.iterate(1)
            r = t.read(want_words=True)
            want = (s * s - 2) % m
            want = (want * want - 2) % m
            got = sum(w << (64 * i) for i, w in enumerate(r["words"]))
            assert got == want, (name, p)
            assert r["is_zero"] == int(want == 0)
    finally:
        t.close()
