"""The library's host code against a CUDA runtime that is as late as the documentation allows
(fake_cudart.cpp, linked with the library's own objects): copies read their source when the stream
gets to them, legacy-stream work stays pending until something waits for it, two devices. No GPU."""
import ctypes
import glob
import os
import subprocess

import pytest

from conftest import PKG, ROOT

FP64, NTT, KEEP_WORDS, ERRLOG = 0, 1, 1, 2


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    from mersenneprime_python_cpp_gmp_benchmark_b200 import llgpu
    out = tmp_path_factory.mktemp("fake")
    objs = ["_build/" + os.path.splitext(os.path.basename(f))[0] + ".o"
            for f in sorted(glob.glob(os.path.join(PKG, "csrc", "llg_*.c*"))) if f.endswith((".cu", ".cpp"))]
    subprocess.run(["make", "-s", "-j8", "-C", PKG, *objs], check=True)
    so = str(out / "libfake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), *[os.path.join(PKG, o) for o in objs],
                    "-lpthread", "-o", so], check=True)
    L = ctypes.CDLL(so)
    u64, u32, i, sz, vp, P = (ctypes.c_uint64, ctypes.c_uint32, ctypes.c_int, ctypes.c_size_t, ctypes.c_void_p,
                              ctypes.POINTER)
    L.llg_batch_create.argtypes = [P(u64), sz, u64, i, i, P(vp)]
    L.llg_batch_launch.argtypes = [vp, vp]
    L.llg_batch_results.argtypes = [vp, P(llgpu.LlgResult), P(u64), sz]
    L.llg_batch_destroy.argtypes = [vp]
    L.llg_run.argtypes = [u64, u64, i, u32, P(llgpu.LlgResult), P(u64), sz]
    L.llg_test_create.argtypes = [u64, u32, i, P(vp)]
    L.llg_test_start.argtypes = [vp, vp]
    L.llg_test_iterate.argtypes = [vp, u64, vp]
    L.llg_test_load.argtypes = [vp, P(u64), sz, u64, vp]
    L.llg_test_destroy.argtypes = [vp]
    L.llg_run_noalloc.argtypes = [u64, u64, u32, vp, P(ctypes.c_double), vp]
    L.fake_violations.restype = ctypes.c_char_p
    L.fake_in_use.restype = L.fake_host_news.restype = u64
    L.fake_set_free.argtypes = [u64]
    L.Result = llgpu.LlgResult
    return L


@pytest.fixture
def fake(fake_lib):
    fake_lib.fake_set_device(0)
    fake_lib.fake_reset()
    yield fake_lib
    fake_lib.fake_set_device(0)


def _batch(L, ps, iters=20, engine=FP64, flags=0):
    b = ctypes.c_void_p()
    assert L.llg_batch_create((ctypes.c_uint64 * len(ps))(*ps), len(ps), iters, engine, flags, ctypes.byref(b)) == 0
    return b


def _results(L, b, n):
    out = (L.Result * n)()
    assert L.llg_batch_results(b, out, None, 0) == 0
    return out


# one word test, whole tests of one and of several lengths, with the word offsets of kept residues
@pytest.mark.parametrize("ps,flags", [([127], 0), ([2203], 0), ([127, 521, 2203, 9689, 44497], KEEP_WORDS)])
@pytest.mark.parametrize("engine", [FP64, NTT])
def test_job_lists_live_until_their_copy_ran(fake, ps, flags, engine):
    b = _batch(fake, ps, engine=engine, flags=flags)
    churn = [ctypes.create_string_buffer(256) for _ in range(64)]  # reuses what the call has freed
    assert fake.llg_batch_launch(b, None) == 0
    _results(fake, b, len(ps))
    fake.llg_batch_destroy(b)
    del churn
    assert b"source of an asynchronous copy" not in fake.fake_violations()


# tables built on first use by every kind of test, one-exponent batches with a round-off log, and the
# objects of both two-pass engines (power-of-two and R0 x 2^k lengths)
def test_no_kernel_starts_beside_pending_setup(fake):
    for p in (127, 521, 2203, 9689, 44497, 80021):
        for engine in (FP64, NTT):
            b = _batch(fake, [p], engine=engine, flags=ERRLOG)
            assert fake.llg_batch_launch(b, None) == 0
            _results(fake, b, 1)
            fake.llg_batch_destroy(b)
    for p, n, engine in ((300007, 1 << 14, FP64), (300007, 1 << 14, NTT), (14000017, 3 << 18, FP64)):
        t = ctypes.c_void_p()
        assert fake.llg_test_create(p, n, engine, ctypes.byref(t)) == 0
        assert fake.llg_test_start(t, None) == 0
        assert fake.llg_test_iterate(t, 3, None) == 0
        fake.llg_test_destroy(t)
    assert b"legacy-stream work is pending" not in fake.fake_violations()


def test_loaded_residue_is_the_callers_again_on_return(fake):
    p, n = 300007, 1 << 14
    for engine in (FP64, NTT):
        t = ctypes.c_void_p()
        assert fake.llg_test_create(p, n, engine, ctypes.byref(t)) == 0
        words = (ctypes.c_uint64 * ((p + 63) // 64))(*range(1, (p + 63) // 64 + 1))
        words[-1] = 0
        assert fake.llg_test_load(t, words, len(words), 5, None) == 0
        words[0] = 99  # the call is over: the buffer may be reused
        assert fake.llg_test_iterate(t, 2, None) == 0
        fake.llg_test_destroy(t)  # waits
    assert b"source of an asynchronous copy" not in fake.fake_violations()


def test_redone_tests_stay_on_the_batchs_device(fake):
    """A batch collected by a thread whose current device is another one: its round-off redo runs on the
    batch's device, and the stream it used is not handed to later calls of the wrong device."""
    b = _batch(fake, [521])
    assert fake.llg_batch_launch(b, None) == 0
    fake.fake_script_status(1, 1)  # round-off above the limit: redone at the next length
    fake.fake_set_device(1)
    out = _results(fake, b, 1)
    assert out[0].escalations == 1
    fake.llg_batch_destroy(b)
    ps = [127, 521, 2203, 9689]  # a group and a stream each
    for dev in (0, 1, 0):
        fake.fake_set_device(dev)
        b = _batch(fake, ps)
        assert fake.llg_batch_launch(b, None) == 0
        _results(fake, b, len(ps))
        fake.llg_batch_destroy(b)
    assert b"device" not in fake.fake_violations()


def test_noalloc_allocates_no_host_memory_either(fake):
    out = (ctypes.c_int32 * 65536)()  # the fake's device memory is host memory
    err = ctypes.c_double()
    for p, n in ((300007, 1 << 14), (600011, 1 << 15), (1257787, 1 << 16)):
        before = fake.fake_host_news()
        assert fake.llg_run_noalloc(p, 3, n, out, ctypes.byref(err), None) == 0
        assert fake.fake_host_news() == before, n
