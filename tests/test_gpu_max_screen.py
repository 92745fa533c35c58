"""The FP64 max|E|^2 monitor leaves out cells whose bound lies below the maximum found so far: the
result is the exact maximum at every magnitude a double holds, and non-finite fields still stop
the run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [dict(isPlanar=0, Nx=70, Ny=41, Nz=75), dict(isPlanar=1, Nx=130, Ny=1, Nz=97)]


def _sim(shape):
    from luxum_gb300 import Sim, params

    return Sim(params(dx=1e-3, dy=1e-3, dz=1e-3, S=0.5, num_timesteps=9, monitor_every=1, **shape))


def _fill(s, scale, rng, flat):
    for c in range(3):
        shp = s.shape(c)
        if np.prod(shp) == 0:
            continue
        a = rng.standard_normal(shp)
        if flat:  # nearly equal cells: the bound cannot tell them apart
            a = 1.0 + 1e-9 * a
        s.set_field(c, a * scale)


@pytest.mark.parametrize("shape", SHAPES, ids=["3d", "planar"])
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("scale", [1e-170, 1e-150, 1e-60, 1e-25, 3e-19, 1.0, 1e19, 1e80, 1e150])
def test_max_is_exact(engine, shape, flat, scale):
    """Squares below the smallest double (1e-170) round to zero on both sides."""
    s = _sim(shape)
    rng = np.random.default_rng(3)
    _fill(s, scale, rng, flat)
    s.step(3)
    if shape["isPlanar"]:
        want = (s.field(1) ** 2).max()
    else:
        n = (s.p.Nx - 1, s.p.Ny - 1, s.p.Nz - 1)
        e = [s.field(c)[: n[0], : n[1], : n[2]].astype(np.longdouble) for c in range(3)]
        want = float((e[0] ** 2 + e[1] ** 2 + e[2] ** 2).max())
    assert s.max_e2() == pytest.approx(want, rel=1e-15, abs=5e-324)
    s.close()


@pytest.mark.parametrize("shape", SHAPES, ids=["3d", "planar"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e200])
def test_non_finite_maximum_stops_the_run(engine, shape, bad):
    from luxum_gb300 import LuxumError

    s = _sim(shape)
    _fill(s, 1.0, np.random.default_rng(4), False)
    c = 1
    a = s.field(c)
    a[-2, 0 if shape["isPlanar"] else 20, 50] = bad
    s.set_field(c, a)
    with pytest.raises(LuxumError, match="not finite"):
        s.step(1)
    s.close()
