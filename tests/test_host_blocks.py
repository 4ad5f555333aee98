"""The pool of page-locked blocks (csrc/host_blocks.cpp) and the blocks a context lends to its batches (csrc/block_cache.h),
built against a stand-in for the CUDA runtime: sizes, references, bounds, the device the locking happens on, and what a forked
child sees."""
import ctypes as C
import os
import random
import subprocess
import sys
import threading

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "datago_b200", "csrc")
MB = 1 << 20
E_TOO_LARGE = 11


@pytest.fixture(scope="session")
def library(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libhost_blocks.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "fake_cuda.cpp"), os.path.join(CSRC, "host_blocks.cpp"), "-o", out], check=True)
    return out


@pytest.fixture
def pool(library, tmp_path, monkeypatch):
    monkeypatch.setenv("DATAGO_B200_HOST_BLOCKS_MB", "8")
    private = str(tmp_path / "lib.so")  # a copy of its own: the pool starts empty
    with open(library, "rb") as f, open(private, "wb") as g:
        g.write(f.read())
    L = C.CDLL(private)
    L.hb_acquire.argtypes = [C.c_size_t, C.c_int, C.POINTER(C.c_void_p)]
    L.dg_host_alloc.argtypes = [C.c_uint64, C.POINTER(C.c_void_p)]
    L.dg_host_release.argtypes = L.hb_retain.argtypes = L.fake_locked_on.argtypes = [C.c_void_p]
    L.fake_locked_bytes.restype = L.fake_device_bytes.restype = C.c_size_t
    L.bc_new.restype = C.c_void_p
    L.bc_acquire.argtypes, L.bc_release.argtypes, L.bc_delete.argtypes = [C.c_void_p, C.c_size_t], [C.c_void_p, C.c_int], [C.c_void_p]
    L.fake_device_limit.argtypes = [C.c_size_t]
    return L


def take(L, n, optional=1):
    p = C.c_void_p()
    assert L.hb_acquire(n, optional, C.byref(p)) == 0
    return p.value


def test_blocks_are_reused_counted_and_given_back(pool):
    pool.hb_context(0, 1)
    a = take(pool, 3 * MB - 5)
    C.memset(a, 1, 3 * MB - 5)
    b = take(pool, 100)
    pool.hb_retain(a)
    pool.dg_host_release(a)
    assert take(pool, 3 * MB) != a                # one reference is left
    pool.dg_host_release(a)
    assert take(pool, 3 * MB - 5) == a            # idle now
    pool.dg_host_release(b)
    assert take(pool, 2 * MB) != b                # far too small
    pool.dg_host_release(a)
    pool.dg_host_release(a)                       # once too often: nothing happens
    before = pool.fake_locked_bytes()
    pool.hb_context(0, -1)                        # the last context: idle blocks go, referenced ones stay
    assert 0 < pool.fake_locked_bytes() < before


def test_limits_hold_for_what_is_referenced_and_for_what_is_idle(pool):
    pool.hb_context(0, 1)
    held = [take(pool, MB) for _ in range(8)]
    p = C.c_void_p()
    assert not pool.hb_scarce()
    assert pool.dg_host_alloc(1, C.byref(p)) == E_TOO_LARGE and not p.value
    more = [take(pool, 2 * MB, 0) for _ in range(3)]  # a caller without an alternative gets its block
    assert pool.hb_scarce()
    for x in more + held:
        pool.dg_host_release(x)
    assert not pool.hb_scarce() and pool.fake_locked_bytes() <= 8 * MB
    assert pool.dg_host_alloc(8 * MB, C.byref(p)) == 0


def test_a_feeder_keeps_the_blocks_its_batches_need(pool):
    pool.hb_context(0, 1)
    pool.hb_feeder(1)
    for i in range(10):  # 24 MB a batch, two at a time, over a limit of 8
        batch = [take(pool, 4 * MB, 0) for _ in range(6)]
        if i:
            for x in last:
                pool.dg_host_release(x)
        last = batch
        if i == 1:
            locks = pool.fake_locks()
    assert pool.fake_locks() == locks and pool.fake_locked_bytes() == 48 * MB
    p = C.c_void_p()
    assert pool.dg_host_alloc(MB, C.byref(p)) == E_TOO_LARGE  # others are bounded as before
    for x in last:
        pool.dg_host_release(x)
    assert pool.dg_host_alloc(MB, C.byref(p)) == 0
    pool.dg_host_release(p)
    pool.hb_feeder(-1)
    assert pool.fake_locked_bytes() <= 8 * MB


def test_locking_happens_on_a_device_that_has_a_context(pool):
    pool.hb_context(3, 1)  # (this thread has never made a CUDA call: its current device is 0)
    a, b = take(pool, 100), take(pool, 5 * MB)
    assert pool.fake_locked_on(a) == pool.fake_locked_on(b) == 3
    pool.dg_host_release(a)
    pool.hb_context(3, -1)
    pool.dg_host_release(b)
    assert pool.fake_locked_bytes() == 0 and not pool.fake_contexts(0)


def test_threads_at_once(pool):
    pool.hb_context(0, 1)

    def work(seed):
        for i in range(300):
            p = C.c_void_p()
            if pool.hb_acquire(1 + (i * seed) % (2 * MB), 1, C.byref(p)) == 0:
                C.memset(p.value, seed, 16)
                pool.hb_retain(p)
                pool.dg_host_release(p)
                assert C.string_at(p.value, 16) == bytes([seed]) * 16
                pool.dg_host_release(p)

    threads = [threading.Thread(target=work, args=(k,)) for k in (3, 7, 11, 201)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    pool.hb_context(0, -1)
    assert pool.fake_locked_bytes() == 0


@pytest.mark.parametrize("nbytes", [1000, 1 * MB - 1])
def test_a_forked_child_keeps_its_own_copy(pool, nbytes):
    script = """
import ctypes as C, os, sys
L = C.CDLL(sys.argv[1]); n = int(sys.argv[2])
L.hb_acquire.argtypes = [C.c_size_t, C.c_int, C.POINTER(C.c_void_p)]
p = C.c_void_p()
assert L.hb_acquire(n, 1, C.byref(p)) == 0
C.memset(p.value, 7, n)
idle = C.c_void_p()
L.hb_context(0, 1)
L.dg_host_release.argtypes = [C.c_void_p]
for _ in range(2):  # made, handed back, lent again, handed back: idle blocks stay behind (a fork would copy them)
    assert L.hb_acquire(4 * n, 1, C.byref(idle)) == 0 and idle.value != p.value
    L.dg_host_release(idle)
r, w = os.pipe()
pid = os.fork()
if pid == 0:
    os.read(r, 1)
    ok = C.string_at(p.value, n) == bytes([7]) * n
    C.memset(p.value, 9, n)
    ranges = [[int(x, 16) for x in line.split()[0].split("-")] for line in open("/proc/self/maps")]
    ok = ok and not any(lo <= idle.value < hi for lo, hi in ranges)
    L.dg_host_release(p)
    os._exit(0 if ok else 1)
C.memset(p.value, 8, n)  # the pool has handed the block on
os.write(w, b"x")
_, status = os.waitpid(pid, 0)
assert L.hb_acquire(4 * n, 1, C.byref(idle)) == 0
C.memset(idle.value, 5, 4 * n)
pid = os.fork()
if pid == 0:
    os._exit(0 if C.string_at(idle.value, 4 * n) == bytes([5]) * (4 * n) else 1)
status += os.waitpid(pid, 0)[1]
sys.exit(0 if status == 0 and C.string_at(p.value, n) == bytes([8]) * n else 1)
"""
    subprocess.run([sys.executable, "-c", script, pool._name, str(nbytes)], check=True)


class Cache:
    """Batches that borrow some blocks at once, and hand them back."""

    def __init__(self, L):
        self.L, self.c = L, L.bc_new()

    def batch(self, *sizes):
        got = [self.L.bc_acquire(self.c, n) for n in sizes]
        assert len(set(got)) == len(got)
        return got

    def done(self, got):
        for i in got:
            self.L.bc_release(self.c, i)


def test_a_smaller_batch_borrows_what_is_there(pool):
    cache = Cache(pool)
    cache.done(cache.batch(4000 * MB, 700 * MB))
    n = pool.fake_allocations()
    for scale in (1, 3, 40, 5000):
        cache.done(cache.batch(4000 * MB // scale, 700 * MB // scale))
    assert pool.fake_allocations() == n
    pool.bc_delete(cache.c)
    assert pool.fake_device_bytes() == 0


@pytest.mark.parametrize("in_flight", [1, 2])
def test_batches_of_many_sizes_neither_pile_up_blocks_nor_allocate_for_ever(pool, in_flight):
    rng = random.Random(5)
    sizes = [tuple(int(2 ** rng.uniform(20, 32)) for _ in range(3)) for _ in range(40)]
    most = max(max(s) for s in sizes)
    cache, flying = Cache(pool), []
    for i in range(3000):
        if i == 2000:
            n = pool.fake_allocations()
        flying.append(cache.batch(*rng.choice(sizes)))
        if len(flying) > in_flight - 1:
            cache.done(flying.pop(0))
        assert pool.fake_device_bytes() <= 3 * in_flight * (most + most // 8 + 4096)
    assert pool.fake_allocations() == n


def test_idle_blocks_go_before_an_allocation_fails(pool):
    pool.fake_device_limit(1000 * MB)
    cache = Cache(pool)
    cache.done(cache.batch(300 * MB, 300 * MB, 200 * MB))
    big, = cache.batch(800 * MB)
    assert big >= 0
    assert cache.batch(300 * MB) == [-1]
    cache.done([big])
    assert cache.batch(300 * MB, 50 * MB)[0] >= 0
