"""A batch's planar float members step in their two buffers while they are few, in place otherwise:
the bits of their solo twins in either mode and across a change of mode at an odd step."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _sim(k, precision, side):
    from luxum_gb300 import Sim

    n, m = side + k % 5, side - 2 + k % 7
    p = cases.make(isPlanar=1, Nx=n, Ny=1, Nz=m, precision=precision, **cases.pml(6),
                   **cases.pw((1, 0, 0), (0, 1, 0), ((9, n - 10), (0, 0), (9, m - 10)), off=4.0 + k % 3))
    s = Sim(p)
    if k % 9 == 1:
        s.add_dft_plane(0, n // 2, [2e10, 5e10, 9e10], 2)
    return s


def _same(a, b):
    for c in (1, 3, 5):
        assert np.array_equal(a.field(c), b.field(c)), c
    for plane in getattr(a, "_dft", {}):
        assert np.array_equal(a.dft(plane), b.dft(plane))
    assert a.t == b.t and a.max_e2() == b.max_e2() > 0


# 48 members share a sweep launch; FP16 storage sweeps up to 2^22 cells together
@pytest.mark.parametrize("precision, side, first, then", [(1, 40, 48, 3), (2, 40, 47, 4), (2, 700, 8, 2)])
def test_members_keep_their_bits_across_modes(engine, precision, side, first, then):
    from luxum_gb300 import Batch

    members = [_sim(k, precision, side) for k in range(first + then)]
    twins = [_sim(k, precision, side) for k in range(first + then)]
    b = Batch(chunk=4)
    for s in members[:first]:
        b.add(s)
    b.step(13)
    for s in members[first:]:
        b.add(s)
    b.step(10)
    for s in members[:then]:
        b.remove(s)
    b.step(15)
    b.close()
    for k, s in enumerate(twins):
        s.step(13 * (k < first) + 10 + 15 * (k >= then))
        _same(members[k], s)
