"""Device memory: handles and batches step with what they hold when nothing more is to be had for
tables formed ahead, a batch forms them beyond one step only within its allowance, and the server
counts them.  An allocation that fails is reported by its call and by no later one."""
import ctypes as C
from contextlib import ExitStack

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

USED = 7  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT


class _Location(C.Structure):
    _fields_ = [("type", C.c_int), ("id", C.c_int)]


class _Props(C.Structure):
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("location", _Location), ("security", C.c_void_p),
                ("maxSize", C.c_size_t), ("reserved", C.c_ubyte * 56)]


class _Pool:
    """The device's memory pool for as long as this is open: one of at most `size` bytes."""

    def __init__(self, size):
        self.cu = C.CDLL("libcuda.so.1")
        self.old, self.pool, self.held = C.c_void_p(), C.c_void_p(), []
        self._ok(self.cu.cuInit(0))
        self._ok(self.cu.cuDeviceGetMemPool(C.byref(self.old), 0))
        p = _Props(allocType=1, location=_Location(1, 0), maxSize=size)
        self._ok(self.cu.cuMemPoolCreate(C.byref(self.pool), C.byref(p)))
        self._ok(self.cu.cuDeviceSetMemPool(0, self.pool))

    @staticmethod
    def _ok(e):
        assert e == 0, e

    def used(self):
        v = C.c_uint64()
        self._ok(self.cu.cuMemPoolGetAttribute(self.pool, USED, C.byref(v)))
        return v.value

    def fill(self, keep=0):
        """Takes all but `keep` bytes, in pieces of 4 KB and more."""
        kept = C.c_uint64()
        if keep:
            self._ok(self.cu.cuMemAllocAsync(C.byref(kept), C.c_size_t(keep), None))
        n = 1 << 26
        while n >= 1 << 12:
            d = C.c_uint64()
            if self.cu.cuMemAllocAsync(C.byref(d), C.c_size_t(n), None) == 0:
                self.held.append(d)
                assert len(self.held) < 10000
            else:
                n //= 2
        if keep:
            self._ok(self.cu.cuMemFreeAsync(kept, None))
        self._ok(self.cu.cuStreamSynchronize(None))

    def empty(self):
        for d in self.held:
            self._ok(self.cu.cuMemFreeAsync(d, None))
        self._ok(self.cu.cuStreamSynchronize(None))
        self.held = []

    def __enter__(self):
        return self

    def __exit__(self, *a):
        self.empty()
        self._ok(self.cu.cuDeviceSetMemPool(0, self.old))
        self._ok(self.cu.cuCtxSynchronize())
        if self.used() == 0:  # not while a handle is left in it
            self._ok(self.cu.cuMemPoolDestroy(self.pool))


def _oblique(n, precision):
    """Tables over whole faces: twelve sets of two planes."""
    kw = dict(isPlanar=0, Nx=n, Ny=n + 1, Nz=n + 2, precision=precision, cpml_mode=1)
    kw.update(cases.pw((cases.S3, cases.S3, cases.S3), (cases.S2, 0, -cases.S2), ((6, n - 7), (6, n - 6), (6, n - 5)), off=6.0))
    return cases.make(**kw, **cases.pml(4))


def _fields(s):
    return [s.field(c) for c in range(6)] + [np.array(s.max_e2())]


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_steps_alone_without_memory_for_tables_ahead(engine, precision):
    from luxum_gb300 import Sim

    p = _oblique(40, precision)
    with Sim(p) as s:
        s.step(30)
        want = _fields(s)
    with _Pool(96 << 20) as pool, Sim(p) as s:
        pool.fill()
        s.step(13)
        s.step(17)
        pool.empty()
        for a, b in zip(want, _fields(s)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_batch_steps_without_memory_for_tables_ahead(engine, precision):
    from luxum_gb300 import Batch, Sim

    ps = [_oblique(n, precision) for n in (40, 33, 50)]
    want = []
    for p in ps:
        with Sim(p) as s:
            s.step(30)
            want.append(_fields(s))
    with _Pool(256 << 20) as pool, ExitStack() as held:
        sims = [held.enter_context(Sim(p)) for p in ps]
        batch = Batch(chunk=10)
        held.callback(batch.close)
        for s in sims:
            batch.add(s)
        pool.fill(1 << 18)  # a batch of three takes less than this besides its tables
        batch.step(10)
        batch.step(20)
        pool.empty()
        for w, s in zip(want, sims):
            for a, b in zip(w, _fields(s)):
                assert np.array_equal(a, b)


def test_batch_tables_stay_within_their_allowance(engine):
    """Members whose tables of one step take more than half the allowance: no second copy of them."""
    from luxum_gb300 import Batch, Sim

    n, count = 230, 4
    face = (n - 12) ** 2
    assert count * 24 * face * 8 > 17 << 20
    with _Pool(8 << 30) as pool, ExitStack() as held:
        sims = [held.enter_context(Sim(_oblique(n, 0))) for _ in range(count)]
        batch = Batch()
        held.callback(batch.close)
        for s in sims:
            batch.add(s)
        before = pool.used()
        batch.step(1)
        assert pool.used() - before < 4 << 20


def test_server_counts_the_tables_of_its_batch(engine):
    """A budget for two requests, but not for the tables that a batch of the two forms ahead, runs
    one at a time; with the batch's allowance on top of it, both."""
    from luxum_gb300 import Server, device_bytes

    p = _oblique(60, 1)
    for extra, most in ((1 << 20, 1), (32 << 20, 2)):
        with Server(chunk=20, budget_bytes=2 * device_bytes(p) + extra) as srv:
            ids = [srv.submit(p, 2000) for _ in range(2)]
            assert all(srv.wait(r, 120.0) == "done" for r in ids)
            assert srv.stats()["peak_running"] == most


def test_a_failed_allocation_is_reported_once(engine):
    """A handle too large for the memory left fails to create; the next calls go on."""
    from luxum_gb300 import Batch, LuxumError, Sim

    with _Pool(64 << 20) as pool, ExitStack() as held:
        for _ in range(2):
            with pytest.raises(LuxumError):
                Sim(_oblique(200, 0))
            s = held.enter_context(Sim(_oblique(24, 0)))
            s.step(5)
            assert s.max_e2() > 0
        batch = Batch()
        held.callback(batch.close)
        batch.add(s)
        with pytest.raises(LuxumError):
            Sim(_oblique(200, 0))
        batch.step(5)
        assert s.t == 10 and pool.used() > 0
