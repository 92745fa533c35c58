"""Grids near the limits of the kernels' launches and offsets.  With the point source a few cells
from the far corner, the first steps around it are those of a small grid with the source as far from
its far corner, whose profiles and coefficients there are the same numbers: the probes agree bit for
bit."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _probes(n, precision, pml, steps, at):
    """Probe rows of a grid of n points whose source and probes sit at distances from the far corner."""
    from luxum_gb300 import Sim

    far = lambda d: tuple(max(v - 1 - x, 0) for v, x in zip(n, d))  # noqa: E731
    src = far((7, 8, 9))
    planar = n[1] == 1
    s = Sim(cases.make(isPlanar=int(planar), Nx=n[0], Ny=n[1], Nz=n[2], precision=precision, cpml_mode=1, usePS=1,
                       source_kind=1, Nx_source=src[0], Ny_source=src[1], Nz_source=src[2], amp_source=1.0,
                       omega_source=2.0e11, src_t0=2.0, src_tw=2.0, **cases.pml(pml)))
    lo, hi = far((5, 5, 5)), far((2, 2, 2))
    s.set_eps_box(lo, (hi[0], hi[1] + 1 if planar else hi[1], hi[2]), 3.0)
    s.set_probes([far(d) for d in at], steps)
    s.step(steps)
    rows, top, t = s.probes(), s.max_e2(), s.t
    s.close()
    assert rows.shape[0] == t == steps
    return rows, top


# the launch's grid of rows is at most 65535 blocks high
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("rows", [3145680, 3145681, 8388480])
def test_tall_planar_grids(engine, precision, rows):
    at = [(i, 0, k) for i in (0, 1, 3, 6, 8, 11) for k in (0, 1, 4, 9, 10, 18)]
    a, am = _probes((rows, 1, 35), precision, 5, 14, at)
    b, bm = _probes((333, 1, 35), precision, 5, 14, at)
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
    assert am == bm > 0


# 32-bit byte offsets reach FP32 arrays of 2^29 elements and FP16 ones of 2^30 (4-byte coefficients):
# the largest grids below, in packed rows too, and the smallest beyond
@pytest.mark.parametrize("precision, n", [(1, (1023, 1024, 509)), (1, (2047, 2048, 100)), (1, (1024, 1025, 510)),
                                          (2, (1023, 2048, 509)), (2, (1025, 2048, 509))])
def test_3d_grids_at_the_reach_of_offsets(engine, precision, n):
    from luxum_gb300 import trim_device_memory

    row = 128 // (4 if precision == 1 else 2)
    padded = n[0] * n[1] * (-(-n[2] // row) * row)
    assert abs(padded / (1 << (29 if precision == 1 else 30)) - 1) < 2e-3
    at = [(i, j, k) for i in (0, 3, 6, 9) for j in (0, 4, 8, 10) for k in (0, 5, 9, 12)]
    a, am = _probes(n, precision, 5, 14, at)
    trim_device_memory()
    b, bm = _probes((45, 46, 47), precision, 5, 14, at)
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
    assert am == bm > 0
