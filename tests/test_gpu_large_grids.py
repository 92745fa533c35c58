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
