"""Batches over the forms their launches take: more planar float members than one batched sweep
launch holds, members at odd and even steps, point sources (amplitudes formed ahead), large members
in lanes of their own with DFT planes, tables too large to form many steps ahead, captured and
directly launched chunks.  Every member equals, bit for bit, its twin stepped alone."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _planar(n, m, precision, source):
    kw = dict(isPlanar=1, Nx=n, Ny=1, Nz=m, precision=precision, cpml_mode=1)
    if source:
        kw.update(usePS=1, source_kind=1, Nx_source=n // 2, Ny_source=0, Nz_source=m // 2, amp_source=1.0,
                  omega_source=4e10, src_t0=12.0, src_tw=5.0)
    else:
        kw.update(cases.pw((0.6, 0, 0.8), (0, 1, 0), ((9, n - 10), (0, 0), (9, m - 10)), off=8.0))
    return cases.make(**kw, **cases.pml(5)), [((n // 3, 0, m // 3), (n // 2, 1, m // 2), 3.0)]


def _cube(n, precision, source):
    kw = dict(isPlanar=0, Nx=n, Ny=n + 1, Nz=n + 3, precision=precision, cpml_mode=1)
    if source:
        kw.update(usePS=1, Nx_source=n // 2, Ny_source=n // 2, Nz_source=n // 2, amp_source=5.0, omega_source=2e9)
    else:
        kw.update(cases.pw((cases.S3, cases.S3, cases.S3), (cases.S2, 0, -cases.S2), ((8, n - 9), (8, n - 9), (8, n - 9)), off=10.0))
    return cases.make(**kw, **cases.pml(5)), [((n // 3, n // 3, n // 3), (n // 2, n // 2, n // 2), 4.0)]


def _specs(precision, sources):
    rng = np.random.default_rng(11)
    specs = [_planar(int(rng.integers(26, 90)), int(rng.integers(26, 120)), precision, sources and q % 3 == 0)
             for q in range(53)]
    specs += [_planar(1030, 1025, precision, False)]  # a lane of its own
    specs += [_cube(n, precision, sources and n % 2 == 0) for n in (30, 41, 64, 66, 71)]
    return specs


def _make(p, boxes, k):
    from luxum_gb300 import Sim

    s = Sim(p)
    for lo, hi, eps in boxes:
        s.set_eps_box(lo, hi, eps)
    planes = [s.add_dft_plane(0, p.Nx // 2, [2e10, 6e10], 1 + k % 4)] if k % 5 == 3 else []
    s.step(k % 3)
    return s, planes


@pytest.mark.parametrize("precision,sources,chunk", [(1, True, 24), (1, False, 7), (2, False, 12), (0, True, 24)])
def test_members_equal_twins(engine, precision, sources, chunk):
    from luxum_gb300 import Batch

    specs = _specs(precision, sources)
    pairs = [(_make(p, b, k), _make(p, b, k)) for k, (p, b) in enumerate(specs)]
    batch = Batch(chunk=chunk)
    for (a, _), _ in pairs:
        batch.add(a)
    for n in (37, 2 * chunk, 1, 3 * chunk):
        batch.step(n)
        for _, (b, _) in pairs:
            b.step(n)
    for (a, qa), (b, qb) in pairs:
        assert a.t == b.t and a.max_e2() == b.max_e2()
        for c in range(6):
            if np.prod(a.shape(c)):
                assert np.array_equal(a.field(c), b.field(c)), (a.p.Nx, a.p.Nz, c)
        for x, y in zip(qa, qb):
            assert np.array_equal(a.dft(x), b.dft(y)), a.p.Nx
    # stepped alone inside the batch, then with it again; the chunk length changes
    for k in (0, 5, 54):
        pairs[k][0][0].step(3)
        pairs[k][1][0].step(3)
    lib = batch.lib
    batch._check(lib.lx_batch_set_chunk(batch.h, 5))
    batch.step(17)
    for (a, _), (b, _) in pairs:
        b.step(17)
        assert np.array_equal(a.field(1), b.field(1))
    batch.close()
