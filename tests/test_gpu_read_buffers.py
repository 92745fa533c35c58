"""lx_sim_read_field into every kind of host buffer: fresh (its pages populated first), used, offset
from a page boundary, pinned, and sizes around the limits of that population."""
import ctypes as C

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(30, 40), (181, 181), (256, 129), (512, 1025), (1200, 1800)])
def test_read_field_buffers(engine, nx, nz):
    from luxum_gb300 import Sim

    p = cases.make(isPlanar=1, Nx=nx, Ny=1, Nz=nz, precision=1)
    s = Sim(p)
    a = np.random.default_rng(nx).standard_normal(s.shape(1))
    s.set_field(1, a)
    want = a.astype(np.float32).astype(np.float64)
    dp = C.POINTER(C.c_double)

    def read(out):
        s._check(s.lib.lx_sim_read_field(s.h, 1, out.ctypes.data_as(dp), out.size))
        assert np.array_equal(out, want)

    fresh = np.empty(a.shape)
    read(fresh)
    fresh[:] = -1.0
    read(fresh)  # resident pages
    for off in (1, 7, 513):  # off a page boundary, with neighbours that must keep their values
        buf = np.full(a.size + off + 9, 5.0)
        read(buf[off:off + a.size].reshape(a.shape))
        assert (buf[:off] == 5.0).all() and (buf[off + a.size:] == 5.0).all()
    ptr = C.c_void_p()
    s._check(s.lib.lx_host_alloc(a.nbytes, C.byref(ptr)))
    read(np.ctypeslib.as_array(C.cast(ptr, dp), shape=(a.size,)).reshape(a.shape))
    s.lib.lx_host_free(ptr)
    s.close()
