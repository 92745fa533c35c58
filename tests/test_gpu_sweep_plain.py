"""Planar float grids without CPML: the single sweep's form without psi against the two-sweep kernels,
bit for bit, at the edges of its tiles and runs of rows."""
import pytest

import cases
from test_gpu_sweep import _pair, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("tf, dz", [(0, 1e-3), (1, 1e-3), (1, 0.8e-3)])
@pytest.mark.parametrize("n, m", [(3, 3), (17, 31), (16, 32), (33, 33), (50, 64), (2000, 65), (65, 2000), (513, 300), (1300, 1311)])
def test_planar_without_cpml_equals_two_sweep(engine, precision, tf, dz, n, m):
    kw = dict(isPlanar=1, Nx=n, Ny=1, Nz=m, dz=dz, precision=precision, usePS=1, source_kind=1, Nx_source=n // 2,
              Nz_source=m // 2, amp_source=1.0, omega_source=2.0e11, src_t0=6.0, src_tw=4.0)
    if tf:
        kw.update(cases.pw((0.6, 0, 0.8), (0, 1, 0), ((1 + n // 5, n - 2 - n // 5), (0, 0), (1 + m // 5, m - 2 - m // 5)), off=4.0))
    a, b = _pair(cases.make(**kw), [((n // 3, 0, m // 3), (n // 2 + 1, 1, m // 2 + 1), 3.0)], dft=False)
    for steps in (17, 12):
        a.step(steps)
        b.step(steps)
        _same(a, b)
    assert a.max_e2() == b.max_e2() and (n < 5 or a.max_e2() > 0)
    a.close()
    b.close()
