"""Float 3-D grids with CPML beyond those whose half steps issue every load ahead (FP32 H to 5 * 2^20
cells unless their rows are packed, FP16 H to 2^21 and E to 2^22): blocks in one CPML slab take a path
of their own.  The same bits as the independently written single-sweep kernel, at odd sizes with equal
and unequal spacing; and the largest grids that batches step in the general cell code, without CPML."""
import numpy as np
import pytest

from test_gpu_small_grids import _march, _sim
from test_gpu_sweep import _big3, _pair, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("uniform, n", [(False, (177, 191, 157)), (True, (201, 187, 160)), (False, (161, 180, 203)),
                                        (True, (40, 700, 190))])
def test_slab_paths_equal_single_sweep_beyond_loads_ahead(engine, precision, uniform, n):
    assert np.prod(n) > 5 << 20 and 5 * n[2] > 4 * ((n[2] + 31) & ~31)
    p, boxes = _big3(precision, uniform, n)
    a, b = _pair(p, boxes)
    for steps in (31, 16):
        a.step(steps)
        b.step(steps)
        _same(a, b)
    assert a.max_e2() == b.max_e2() > 0
    a.close()
    b.close()


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("n, pml, tf", [((63, 64, 64), 0, 0), ((62, 64, 66), 6, 1)])
def test_grids_just_below_the_lanes_equal_batch_members(engine, precision, n, pml, tf):
    assert np.prod(n) < 1 << 18
    for s in _march(lambda: _sim(n, precision, pml, tf)):
        s.close()
