"""The kernel counter of batched members: the launches that a member has part in."""
import pytest

import cases

pytestmark = pytest.mark.gpu


def _params(planar, precision, n, source):
    kw = dict(isPlanar=int(planar), Nx=n, Ny=1 if planar else n, Nz=n, precision=precision, cpml_mode=1)
    if source:
        kw.update(usePS=1, source_kind=1, Nx_source=n // 2, Ny_source=0 if planar else n // 2, Nz_source=n // 2,
                  amp_source=1.0, omega_source=4e10, src_t0=12.0, src_tw=5.0)
    return cases.make(**kw, **cases.pml(5))


# Launches of tables ahead (16 steps each) and of the step counters (one a run): chunks of 20 steps are
# runs of their own where a plane's period divides them, else 45 steps are one run.
# Planar float members of 2^21 cells and more step in one launch, FP64 and 3-D members in two.
@pytest.mark.parametrize("every, common", [(3, (2 + 1) + (3 + 1)), (4, 3 * (2 + 1) + (1 + 1))])
@pytest.mark.parametrize("planar, precision, n, update", [(True, 0, 60, 2), (True, 1, 1449, 1), (False, 0, 30, 2), (False, 1, 70, 2)])
def test_batched_members_count_their_launches(engine, planar, precision, n, update, every, common):
    from luxum_gb300 import Batch, Sim

    sims = [Sim(_params(planar, precision, n, source)) for source in (False, True)]
    sims[0].add_dft_plane(0, n // 2, [2e10], every)
    batch = Batch(chunk=20)
    for s in sims:
        batch.add(s)
    at = [s.counters()[0] for s in sims]
    batch.step(20)
    batch.step(45)
    steps = 65
    samples = len([t for t in range(steps) if t % every == 0])
    got = [s.counters()[0] - a for s, a in zip(sims, at)]
    assert got == [common + update * steps + 2 * samples, common + (update + 1) * steps]
    batch.close()
    for s in sims:
        s.close()
