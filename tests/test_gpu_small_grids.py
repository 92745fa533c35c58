"""3-D grids whose kernels issue every load ahead and pack rows that fill their tiles badly: the bits
of the members of a batch, which march through the general cell code, or of the single sweep.  DFT planes that
split their frequencies over blocks: the bits of a batch's accumulation, which walks them in order."""
import numpy as np
import pytest

import cases
from test_gpu_sweep import _big3, _pair, _same

pytestmark = pytest.mark.gpu


def _sim(n, precision, pml, tf, dy=1e-3):
    from luxum_gb300 import Sim

    kw = dict(isPlanar=0, Nx=n[0], Ny=n[1], Nz=n[2], dy=dy, precision=precision, usePS=1, source_kind=1,
              Nx_source=n[0] // 2, Ny_source=n[1] // 2, Nz_source=n[2] // 2, amp_source=1.0, omega_source=2.0e11,
              src_t0=6.0, src_tw=4.0, monitor_every=3)
    if pml:
        kw.update(cases.pml(pml, kappa=5.0, a_max=0.05))
    if tf:
        kw.update(cases.pw((1, 0, 0), (0, 0, 1), tuple((v // 4, v - 1 - v // 4) for v in n), off=4.0))
    s = Sim(cases.make(**kw))
    s.set_eps_box((n[0] // 3, n[1] // 3, n[2] // 3), (n[0] // 2, n[1] // 2, n[2] // 2), 4.0)
    return s


def _march(make, steps=19):
    """The same handle alone and as a member of a batch beside a twin (a lone large member of a
    batch would march in a lane of its own)."""
    from luxum_gb300 import Batch

    alone, a, b = make(), make(), make()
    batch = Batch()
    batch.add(a)
    batch.add(b)
    batch.step(steps)
    batch.close()
    alone.step(steps)
    for c in range(6):
        assert np.array_equal(alone.field(c), a.field(c)), c
    assert alone.max_e2() == a.max_e2() > 0
    b.close()
    return alone, a


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("n, pml, tf, dy", [
    ((9, 8, 7), 0, 0, 1e-3), ((12, 12, 25), 3, 1, 1e-3), ((13, 11, 26), 3, 1, 1.25e-3), ((16, 9, 31), 4, 0, 1e-3),
    ((17, 14, 32), 5, 1, 1.25e-3), ((14, 15, 33), 3, 1, 1e-3), ((11, 30, 64), 3, 0, 1e-3), ((40, 38, 64), 6, 1, 1e-3),
    ((46, 47, 45), 6, 1, 1e-3), ((46, 47, 46), 6, 0, 1e-3), ((63, 64, 65), 0, 1, 1.25e-3), ((64, 64, 64), 0, 0, 1e-3)])
def test_small_grids_equal_batch_members(engine, precision, n, pml, tf, dy):
    for s in _march(lambda: _sim(n, precision, pml, tf, dy)):
        s.close()


# Larger float grids: both halves, E only, packed, neither or E only again; against the independently written single sweep.
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("uniform, n", [(True, (101, 103, 105)), (False, (129, 128, 128)), (True, (150, 149, 151)),
                                        (False, (176, 175, 177)), (True, (260, 259, 65)), (True, (180, 176, 190)),
                                        (False, (176, 191, 180))])
def test_loads_ahead_equal_single_sweep(engine, precision, uniform, n):
    p, boxes = _big3(precision, uniform, n)
    a, b = _pair(p, boxes)
    a.step(37)
    b.step(37)
    _same(a, b)
    assert a.max_e2() == b.max_e2() > 0
    a.close()
    b.close()


# 128 x 152 cells fill the 304 blocks from which a plane walks its frequencies in order
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nfreq, na, nb", [(1, 20, 33), (3, 20, 33), (4, 20, 33), (5, 20, 33), (33, 128, 151),
                                           (33, 128, 152), (256, 16, 16)])
def test_split_dft_planes_equal_batch(engine, precision, nfreq, na, nb):
    w = 2 * np.pi * np.linspace(1e10, 1.5e11, nfreq)

    def make():
        s = _sim((10, na, nb), precision, 0, 0)
        s.add_dft_plane(0, 4, w, every=2)
        return s

    alone, a = _march(make)
    x = alone.dft(0)
    assert np.array_equal(x, a.dft(0)) and np.abs(x).max() > 0
    alone.close()
    a.close()
