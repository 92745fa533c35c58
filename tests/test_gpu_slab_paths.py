"""Float 3-D grids of 2^20 cells or more, whose blocks in one CPML slab take a path of their own:
the same bits as the independently written single-sweep kernel, at odd sizes with unequal spacing."""
import numpy as np
import pytest

from test_gpu_sweep import _big3, _pair, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("uniform, n", [(False, (161, 133, 203)), (True, (129, 261, 127)), (True, (101, 103, 105)),
                                        (False, (33, 420, 83))])
def test_slab_paths_equal_single_sweep(engine, precision, uniform, n):
    assert np.prod(n) >= 1 << 20
    p, boxes = _big3(precision, uniform, n)
    a, b = _pair(p, boxes)
    for steps in (40, 23):
        a.step(steps)
        b.step(steps)
        _same(a, b)
    assert a.max_e2() == b.max_e2() > 0
