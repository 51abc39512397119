"""The work this engine is used for, as timed cases: single Lucas-Lehmer calls, batches over ranges
of exponents, and long-running tests of one large exponent, on the FP64 and the exact NTT engine.

A case is one of three kinds:

  call   one exponent through `llgpu.run` (what `lucaslehmer.lucas_lehmer*_res` and
         `fft_res64_after` do): a whole test, or its first `iters` squarings, from s_0 = 4. The
         exponent is one of the primes that follow `p`, so another seed is another exponent.
  batch  the primes of [lo, hi] (a random `share` of them) through the C-ABI's `llg_run_batch`
         (what `lucaslehmer_cuda.lucas_lehmer_batch` calls): whole tests, or `iters` squarings each.
  test   a resident test of one exponent (`llgpu.Test`), as a program that runs a large exponent
         for days keeps it: its residue is random digits, as in the middle of a test; a pass is
         `iters` squarings and a full read of the residue (a checkpoint).

Outputs are residues: whole numbers, equal bit for bit whatever computes them.
"""
import ctypes
import math
import random

import numpy as np

from mersenneprime_python_cpp_gmp_benchmark_b200 import llgpu


def listed():
    return [
        # the smallest call: an exponent below 256 (exact word kernel), all launch and host latency
        {"name": "call_word", "kind": "call", "p": 127, "iters": 0, "engine": "fp64"},
        # a driver thread's call on a small exponent: one short whole test on one SM
        {"name": "call_small", "kind": "call", "p": 2203, "iters": 0, "engine": "fp64"},
        # a driver thread's call on an ordinary exponent: the latency of one squaring, 21,701 times
        {"name": "call_mid", "kind": "call", "p": 21701, "iters": 0, "engine": "fp64"},
        # the same call on the exact engine (`lucas_lehmer`, the driver's --engine gmp)
        {"name": "call_exact", "kind": "call", "p": 9689, "iters": 0, "engine": "ntt"},
        # a first look at an exponent of the two-pass lengths: tables, buffers, squarings, residue
        {"name": "call_interim", "kind": "call", "p": 859433, "iters": 1000, "engine": "fp64"},
        # the lower part of the range benchmark (every prime p <= 100001), whole tests
        {"name": "range_tests", "kind": "batch", "lo": 3, "hi": 20011, "share": 0.9, "iters": 0, "engine": "fp64"},
        # the upper part of it, where nearly all of its time goes: 1000 squarings of every test
        {"name": "range_slice", "kind": "batch", "lo": 20011, "hi": 100001, "share": 0.9, "iters": 1000, "engine": "fp64"},
        # a range double-checked on the exact engine
        {"name": "range_exact", "kind": "batch", "lo": 401, "hi": 40009, "share": 0.3, "iters": 1000, "engine": "ntt"},
        # the single-exponent benchmark's exponent, at the length that benchmark asks for
        {"name": "test_1257787", "kind": "test", "p": 1257787, "n": 65536, "iters": 1000, "engine": "fp64"},
        # an exponent of the [20M, 25M] sweep (N = 5 x 2^18)
        {"name": "test_22685363", "kind": "test", "p": 22685363, "iters": 1000, "engine": "fp64"},
        # the headline benchmark's exponent (N = 2^23)
        {"name": "test_136279841", "kind": "test", "p": 136279841, "iters": 1000, "engine": "fp64"},
        # the sweep exponent on the exact engine (N = 2^21)
        {"name": "test_exact_22685363", "kind": "test", "p": 22685363, "iters": 200, "engine": "ntt"},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(["call", "batch", "batch", "test", "test", "test"])
    engine = rng.choice(["fp64", "fp64", "ntt"])
    slow = 5 if engine == "ntt" else 1  # squarings on the exact engine cost several times as much
    if kind == "call":
        if rng.random() < 0.6:  # whole tests
            p = _log_uniform(rng, 61, 24000) if engine == "fp64" else _log_uniform(rng, 401, 12000)
            return {"kind": kind, "p": p, "iters": 0, "engine": engine}
        p = _log_uniform(rng, 24000, 4000000)
        return {"kind": kind, "p": p, "iters": _log_uniform(rng, 100, 1000) // slow, "engine": engine}
    if kind == "batch":
        hi = _log_uniform(rng, 1000, 100001 // (2 if slow > 1 else 1))
        lo = rng.randrange(3 if engine == "fp64" else 401, hi // 2)
        share = round(rng.uniform(0.1, 0.9) / (2 if slow > 1 else 1), 3)
        return {"kind": kind, "lo": lo, "hi": hi, "share": share, "iters": _log_uniform(rng, 50, 800) // slow, "engine": engine}
    p = _log_uniform(rng, 270000, 150000000)
    iters = min(_log_uniform(rng, 100, 2000), 10**11 // p) // slow
    return {"kind": kind, "p": p, "iters": max(20, iters), "engine": engine}


# ---- inputs ----------------------------------------------------------------------------------


def _is_prime(n):
    if n < 4:
        return n > 1
    if n % 2 == 0:
        return False
    for d in range(3, math.isqrt(n) + 1, 2):
        if n % d == 0:
            return False
    return True


def _prime_from(n, skip=0):
    """The (skip + 1)-th prime >= n."""
    n |= 1
    while True:
        if _is_prime(n):
            if skip == 0:
                return n
            skip -= 1
        n += 2


def _primes(lo, hi):
    comp = bytearray(hi + 1)
    for i in range(2, math.isqrt(hi) + 1):
        if not comp[i]:
            comp[i * i::i] = b"\x01" * len(range(i * i, hi + 1, i))
    return [i for i in range(max(lo, 3), hi + 1) if not comp[i]]


def _exponent(case, seed):
    if case["kind"] == "test":
        return _prime_from(case["p"])
    return _prime_from(case["p"], random.Random(seed).randrange(8))


def _batch_exponents(case, seed):
    ps = _primes(case["lo"], case["hi"])
    return sorted(random.Random(seed).sample(ps, max(1, int(len(ps) * case["share"]))))


def _residue_words(p, seed):
    """ceil(p/64) random words below 2^p."""
    w = np.random.default_rng(seed).integers(0, 1 << 64, llgpu.nwords(p), dtype=np.uint64)
    if p % 64:
        w[-1] &= np.uint64((1 << (p % 64)) - 1)
    return w


def _word_room(case):
    """Words that hold the residues of any seed's exponents (the rest stays zero)."""
    if case["kind"] == "batch":
        ps = _primes(case["lo"], case["hi"])
        return sum(llgpu.nwords(p) for p in ps[-max(1, int(len(ps) * case["share"])):])
    return llgpu.nwords(_prime_from(case["p"], 7 if case["kind"] == "call" else 0))


def prepare(case, seed):
    state = {"case": case}
    if case["kind"] == "call":
        state["p"] = _exponent(case, seed)
        state["words"] = np.zeros(_word_room(case), dtype=np.uint64)
        return state
    if case["kind"] == "batch":
        ps = _batch_exponents(case, seed)
        state["count"] = len(ps)
        state["ps"] = (ctypes.c_uint64 * len(ps))(*ps)
        state["out"] = (llgpu.LlgResult * len(ps))()
        state["words"] = np.zeros(_word_room(case), dtype=np.uint64)
        return state
    p = _exponent(case, seed)
    t = llgpu.Test(p, n=case.get("n", 0), engine=case["engine"])
    t.load(_residue_words(p, seed).tolist(), 1000)
    state.update(p=p, test=t, words=np.zeros(llgpu.nwords(p), dtype=np.uint64))
    return state


# ---- one pass --------------------------------------------------------------------------------


def _pointer(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))


def _check(rc):
    if rc:
        raise llgpu.LlgError(rc, (llgpu.lib().llg_last_error() or b"").decode())


def run(state):
    case = state["case"]
    if case["kind"] == "call":
        r = llgpu.run(state["p"], iters=case["iters"], engine=case["engine"], want_words=True)
        words = state["words"]
        words[:len(r["words"])] = r["words"]
        return {"zero": r["is_zero"], "words": words.view(np.int64)}
    if case["kind"] == "batch":
        out, words = state["out"], state["words"]
        _check(llgpu.lib().llg_run_batch(state["ps"], state["count"], case["iters"], llgpu.ENGINES[case["engine"]], out,
                                         _pointer(words), words.size))
        return {"zero": np.array([r.is_zero for r in out], dtype=np.int64), "words": words.view(np.int64)}
    t, words = state["test"], state["words"]
    t.iterate(case["iters"])
    r = llgpu.LlgResult()
    _check(llgpu.lib().llg_test_read(t.h, None, ctypes.byref(r), _pointer(words), words.size))
    return {"zero": r.is_zero, "words": words.view(np.int64)}


# ---- what a pass cannot do without -------------------------------------------------------------


def _squaring_flops(p, engine):
    """One squaring of p bits by a transform pair over the digits of the engine's own size: 5 n log2 n
    operations (FP64, n = p / 18), or n log2 n products and as many sums in the field (NTT)."""
    if p < 256:
        return 2.0 * ((p + 63) // 64) ** 2
    if engine == "fp64":
        n = p / 18.0
        return 5.0 * n * math.log2(n)
    n = p / ((63.0 - math.log2(p / 22.0)) / 2.0)
    return 2.0 * n * math.log2(n)


def work(case):
    if case["kind"] == "batch":
        ps = _primes(case["lo"], case["hi"])
        share = case["share"]
    else:
        ps, share = [case["p"]], 1.0
    flops = sum((case["iters"] or p - 2) * _squaring_flops(p, case["engine"]) for p in ps) * share
    residue = sum(llgpu.nwords(p) * 8 for p in ps) * share  # read (a test's start) or written once
    return {"bytes": residue * (2 if case["kind"] == "test" else 1), "flops": flops}


# ---- exact results -----------------------------------------------------------------------------


def _square_on(s, p, iters):
    m = (1 << p) - 1
    for _ in range(iters):
        s = s * s - 2
        while s > m:
            s = (s & m) + (s >> p)
        if s < 0:
            s += m
    return 0 if s == m else s


def _words_of(s, p):
    return np.frombuffer(s.to_bytes(llgpu.nwords(p) * 8, "little"), dtype=np.uint64).view(np.int64)


def exact(case, seed):
    """Plain integer arithmetic, where it takes a few seconds at most."""
    if case["kind"] == "batch":
        ps = _batch_exponents(case, seed)
    else:
        ps = [_exponent(case, seed)]
    if sum((case["iters"] or p - 2) * (1e-6 + 2.5e-9 * (p / 30.0) ** 1.585) for p in ps) > 8.0:
        return None
    if case["kind"] == "test":
        p = ps[0]
        s = int.from_bytes(_residue_words(p, seed).tobytes(), "little")
        # loading a residue starts the next squaring, which the pass's read includes
        s = _square_on(s, p, 1 + case["iters"])
        return {"zero": int(s == 0), "words": _words_of(s, p)}
    done = [_square_on(4 % ((1 << p) - 1), p, case["iters"] or p - 2) for p in ps]
    words = np.concatenate([_words_of(s, p) for s, p in zip(done, ps)])
    words = np.concatenate([words, np.zeros(_word_room(case) - words.size, dtype=np.int64)])
    zero = [int(s == 0) for s in done]
    return {"zero": np.array(zero, dtype=np.int64) if case["kind"] == "batch" else zero[0], "words": words}
