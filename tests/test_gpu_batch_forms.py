"""The forms in which a batch steps its planar float members, at the edges of the rules that choose
among them.  Every member equals, bit for bit, its twin stepped alone."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _lens(n, m, precision, k=0):
    kw = dict(isPlanar=1, Nx=n, Ny=1, Nz=m, precision=precision, cpml_mode=1)
    if k % 4 == 1:
        kw.update(usePS=1, source_kind=1, Nx_source=n // 2, Ny_source=0, Nz_source=m // 2, amp_source=1.0,
                  omega_source=4e10, src_t0=9.0, src_tw=5.0)
    else:
        kw.update(cases.pw((0.6, 0, 0.8), (0, 1, 0), ((9, n - 10), (0, 0), (9, m - 10)), off=8.0))
    return cases.make(**kw, **cases.pml(5 + k % 3))


def _sim(p):
    from luxum_gb300 import Sim

    s = Sim(p)
    s.set_eps_box((p.Nx // 3, 0, p.Nz // 3), (p.Nx // 2, 1, p.Nz // 2), 3.0)
    return s


def _compare(ps, runs=(17, 8, 8, 9), chunk=8, before=0):
    from luxum_gb300 import Batch

    sims = [_sim(p) for p in ps]
    batch = Batch(chunk=chunk)
    for k, s in enumerate(sims):
        s.step(k % 3 if before else 0)
        batch.add(s)
    for n in runs:
        batch.step(n)
    for k, (p, s) in enumerate(zip(ps, sims)):
        twin = _sim(p)
        twin.step(sum(runs) + (k % 3 if before else 0))
        for c in (1, 3, 5):
            assert np.array_equal(s.field(c), twin.field(c)), (p.Nx, p.Nz, c)
        assert s.max_e2() == twin.max_e2() > 0
        twin.close()
    batch.close()
    for s in sims:
        s.close()


# 54 members fill the parameters of one batched sweep; one more takes the half steps
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("count", [1, 49, 54, 55])
def test_members_of_one_sweep_launch(engine, precision, count):
    _compare([_lens(24 + 3 * (k % 11), 30 + 7 * (k % 5), precision, k) for k in range(count)])


def test_the_tuner_takes_members_of_the_half_steps(engine):
    """Planar float members of 2^19 cells and more never step in the half-step launches: the tuner
    has no pick for them, in a batch or for one handle."""
    from luxum_gb300 import Batch

    small, large = _sim(_lens(300, 311, 1)), _sim(_lens(725, 724, 1))
    double = _sim(_lens(725, 724, 0))
    batch = Batch()
    batch.add(small)
    batch.add(large)
    assert batch.tune_member(large, 2) == 0 and batch.tune_table() == []
    batch.autotune(2)
    assert [dict(e, march=0) for e in batch.tune_table()] == [dict(small.tune_class(), march=0)]
    assert batch.tune_member(small, 2) in (1, 2, 4, 8)
    batch.close()
    other = Batch()
    other.add(double)
    other.autotune(2)
    assert len(other.tune_table()) == 1
    other.close()
    for s in (small, large, double):
        s.close()


# the sweep's rows a warp: 1 to 4, 6, 8 (4 at most in FP16), by the rows of all its members
@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("count, n, m", [(1, 130, 127), (1, 300, 511), (1, 301, 513), (1, 520, 700), (2, 450, 577), (3, 513, 640),
                                         (8, 480, 700), (8, 640, 800)])
def test_rows_of_the_batched_sweep(engine, precision, count, n, m):
    _compare([_lens(n + k, m - 5 * k, precision, k) for k in range(count)])


# members one by one in lanes, at 2, 5, 6 and 8 rows a warp (FP16 4, 6 and 8): FP32 from 2^19 cells beside more members
# than one sweep holds, FP16 beside few cells
SOLO = [(731, 740), (811, 835), (1001, 903), (1201, 1103)]


@pytest.mark.parametrize("precision, small", [(1, 55), (2, 0)])
def test_rows_of_members_in_lanes(engine, precision, small):
    ps = [_lens(n, m, precision, k) for k, (n, m) in enumerate(SOLO + SOLO[::-1][:2])]
    _compare(ps + [_lens(24 + k % 7, 40 + k % 9, precision, k) for k in range(small)], runs=(5, 8, 8, 4), before=1)


# FP16: lanes for members of 620 K cells and more beside the half steps of the others, from 6 M cells
# of the batch on; half steps for all from 27 M
@pytest.mark.parametrize("sides", [[(1300, 1111)] * 4 + [(701, 803), (90, 77)], [(1901, 1853)] * 7 + [(2100, 1900), (300, 333)]])
def test_fp16_members_by_the_cells_of_the_batch(engine, sides):
    _compare([_lens(n + k, m - k, 2, k) for k, (n, m) in enumerate(sides)], runs=(5, 8, 8, 4), before=1)


# FP16 cubes of 2^18 cells and more: lanes filled (the general kernels) and not (every load ahead)
@pytest.mark.parametrize("count", [2, 4])
def test_fp16_cubes_in_lanes(engine, count):
    from luxum_gb300 import Batch, Sim

    def cube(n, k):
        kw = dict(isPlanar=0, Nx=n, Ny=n + 1, Nz=n + 3, precision=2, cpml_mode=1)
        kw.update(cases.pw((1, 0, 0), (0, 0, 1), ((9, n - 10), (9, n - 9), (9, n - 7)), off=8.0))
        return cases.make(**kw, **cases.pml(5 + k))

    ps = [cube(n, k) for k, n in enumerate((64, 71, 90, 101)[:count])]
    sims = [Sim(p) for p in ps]
    batch = Batch(chunk=8)
    for s in sims:
        batch.add(s)
    for n in (5, 8, 8, 4):
        batch.step(n)
    for p, s in zip(ps, sims):
        twin = Sim(p)
        twin.step(25)
        for c in range(6):
            assert np.array_equal(s.field(c), twin.field(c)), (p.Nx, c)
        assert s.max_e2() == twin.max_e2() > 0
        twin.close()
    batch.close()
    for s in sims:
        s.close()


# members one by one with point sources (each in its lane), beside grouped members with and without
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("hard", [0, 1])
def test_sources_of_members_in_lanes(engine, precision, hard):
    from luxum_gb300 import Batch, Sim

    def cube(n, k):
        kw = dict(isPlanar=0, Nx=n, Ny=n + 1, Nz=n + 3, precision=precision, cpml_mode=1)
        if k != 1:
            kw.update(usePS=1, source_kind=0 if hard else 1, Nx_source=n // 2, Ny_source=n // 2, Nz_source=n // 2,
                      amp_source=5.0, omega_source=2e9 if hard else 4e10, src_t0=9.0, src_tw=5.0)
        else:
            kw.update(cases.pw((1, 0, 0), (0, 0, 1), ((9, n - 10), (9, n - 9), (9, n - 7)), off=8.0))
        return cases.make(**kw, **(cases.pml(5) if k % 2 else {}))

    ps = [cube(n, k) for k, n in enumerate((64, 70, 67, 81, 30, 41))]
    ps += [_lens(1101, 1013, precision, 1), _lens(40, 50, precision, 1)]
    sims = [Sim(p) for p in ps]
    batch = Batch(chunk=8)
    for k, s in enumerate(sims):
        s.step(k % 2)
        batch.add(s)
    for n in (5, 8, 8, 18):
        batch.step(n)
    for k, (p, s) in enumerate(zip(ps, sims)):
        twin = Sim(p)
        twin.step(39 + k % 2)
        for c in range(6):
            if np.prod(s.shape(c)):
                assert np.array_equal(s.field(c), twin.field(c)), (p.Nx, c)
        assert s.max_e2() == twin.max_e2() > 0
        twin.close()
    batch.close()
    for s in sims:
        s.close()
