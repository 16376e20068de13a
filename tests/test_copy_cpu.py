"""The shared copy (csrc/host/ff_copy.c): every byte, at sizes around its piece and its sharing threshold, at odd
addresses, with pools of several owners at work."""
import ctypes as C
import os
import signal
import subprocess
import sys
import threading

import numpy as np
import pytest

import fastface_b200 as ff


@pytest.fixture(scope="module")
def lib(built_lib):
    L = ff.load_library()
    L.ff_copy_pool_create.restype = C.c_void_p
    L.ff_copy_pool_create.argtypes = [C.c_int]
    L.ff_copy_pool_destroy.restype = None
    L.ff_copy_pool_destroy.argtypes = [C.c_void_p]
    L.ff_copy.restype = None
    L.ff_copy.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
    return L


SIZES = [1, 63, 255, 256, 257, 319, 4095, (512 << 10) - 1, 512 << 10, (512 << 10) + 1, (640 << 10) - 3, 1 << 20, 2408448, 5_000_001]


def copies(lib, pool, seed, rounds):
    rng = np.random.default_rng(seed)
    for _ in range(rounds):
        for n in SIZES:
            so, do = int(rng.integers(0, 70)), int(rng.integers(0, 70))
            src = rng.integers(0, 256, n + 200, dtype=np.uint8)
            dst = np.full(n + 200, 0xA5, np.uint8)
            lib.ff_copy(pool, dst.ctypes.data + do, src.ctypes.data + so, n, int(rng.integers(0, 2)))
            assert np.array_equal(dst[do:do + n], src[so:so + n])
            assert np.all(dst[:do] == 0xA5) and np.all(dst[do + n:] == 0xA5)


@pytest.mark.parametrize("helpers", [-1, 0, 1, 3, 100])
def test_copies_every_byte(lib, helpers):
    pool = lib.ff_copy_pool_create(helpers)
    copies(lib, pool, helpers + 5, 4)
    lib.ff_copy_pool_destroy(pool)


def test_no_pool_and_unused_pool(lib):
    copies(lib, None, 1, 1)
    lib.ff_copy_pool_destroy(lib.ff_copy_pool_create(3))
    lib.ff_copy_pool_destroy(None)


def test_pools_of_several_threads(lib):
    bad = []

    def work(k):
        try:
            for _ in range(3):
                pool = lib.ff_copy_pool_create(3)
                copies(lib, pool, k, 3)
                lib.ff_copy_pool_destroy(pool)
        except AssertionError as e:
            bad.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(5)]
    [t.start() for t in ts]
    [t.join(timeout=120) for t in ts]
    assert not bad and not any(t.is_alive() for t in ts)


FORKED = """
import ctypes as C, os, sys, time
L = C.CDLL(sys.argv[1])
L.ff_copy_pool_create.restype = C.c_void_p
L.ff_copy_pool_create.argtypes = [C.c_int]
L.ff_copy_pool_destroy.argtypes = [C.c_void_p]
L.ff_copy.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_int]
n = 4 << 20
src, dst, again = C.create_string_buffer(os.urandom(n), n), C.create_string_buffer(n), C.create_string_buffer(n)
pool = L.ff_copy_pool_create(3)
L.ff_copy(pool, dst, src, n, 0)
time.sleep(0.05)                       # the helpers sleep by now
bad = 0
for first_copies in (0, 1):
    pid = os.fork()
    if pid == 0:
        if first_copies:
            L.ff_copy(pool, again, src, n, 1)
        L.ff_copy_pool_destroy(pool)
        os._exit(0 if again.raw == src.raw or not first_copies else 1)
    bad |= os.waitpid(pid, 0)[1]
L.ff_copy(pool, again, src, n, 0)      # the parent's pool is as it was
L.ff_copy_pool_destroy(pool)
sys.exit(0 if bad == 0 and dst.raw == src.raw and again.raw == src.raw else 1)
"""


def test_forked_process_copies_and_destroys(lib):
    """A child forked after the helpers have started has none of them: it must neither wait for them nor for the
    locks they left (a program that forks workers and lets them drop the object they inherited)."""
    p = subprocess.Popen([sys.executable, "-W", "ignore", "-c", FORKED, ff.LIB_PATH], start_new_session=True)
    try:
        assert p.wait(timeout=20) == 0
    finally:
        if p.poll() is None:
            os.killpg(p.pid, signal.SIGKILL)           # parent and the child that hangs
            p.wait()
