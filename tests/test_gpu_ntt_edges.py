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


def _square(s, p):
    m = (1 << p) - 1
    s = s * s - 2
    while s > m:
        s = (s & m) + (s >> p)
    return s + m if s < 0 else 0 if s == m else s


# N = 2^14: rows of 2^7 (one warp row group); 2^16: 2^8; 2^17: 2^8 rows of 2^9 columns; the widest
# digits the field holds and about 9 bits
@pytest.mark.parametrize("logn,bits", [(14, 24), (14, 9), (16, 23), (17, 9)])
def test_ntt_two_pass_edge_digits(gpu, logn, bits):
    n = 1 << logn
    p = bits * n - 1
    t = gpu.Test(p, n, engine="ntt")
    try:
        for name, s in _residues(p).items():
            b = s.to_bytes(8 * gpu.nwords(p), "little")
            words = [int.from_bytes(b[i:i + 8], "little") for i in range(0, len(b), 8)]
            t.load(words, 1)
            t.iterate(1)
            r = t.read(want_words=True)
            want = _square(_square(s, p), p)
            got = int.from_bytes(b"".join(w.to_bytes(8, "little") for w in r["words"]), "little")
            assert got == want, (name, p)
            assert r["is_zero"] == int(want == 0)
    finally:
        t.close()
