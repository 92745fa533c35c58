"""Replayed step sequences: a long call (captured sequences of steps, TF/SF tables and source
amplitudes formed ahead) leaves the same bits as the same steps taken in short calls, which are
launched one by one: fields, DFT accumulators, probe rows, the max|E|^2 series and max_e2."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

# case, precision, monitor_every, DFT cadence, probes, series; the source cases have a point source
RUNS = [("planar_pml_axis", 0, 1, 0, True, True), ("planar_pml_axis", 1, 4, 3, True, True),
        ("planar_oblique", 1, 0, 5, False, True), ("planar_pml_std_oblique", 2, 0, 0, False, False),
        ("3d_pml_axis", 0, 2, 4, True, True), ("3d_oblique", 0, 0, 0, False, False),
        ("3d_pml_point_cw", 1, 0, 7, True, False), ("3d_pml_pulse_nonuniform", 0, 3, 0, True, True),
        ("3d_pml_pulse_nonuniform", 2, 17, 2, True, True), ("planar_pml_axis", 1, 0, 17, True, False)]


def _run(name, precision, monitor, every, probes, series, calls):
    from luxum_gb300 import Sim

    p, _, boxes = cases.build(name)
    p.precision = precision
    p.monitor_every = monitor
    s = Sim(p)
    for lo, hi, eps in boxes:
        s.set_eps_box(lo, hi, eps)
    planes = [s.add_dft_plane(0, p.Nx // 3, [1e10, 3e10, 7e10], every)] if every else []
    if probes:
        s.set_probes([[p.Nx // 2, 0 if p.isPlanar else p.Ny // 2, p.Nz // 2], [3, 0, 4]], 90)
    if series:
        s.set_max_series(60)
    for n in calls:
        s.step(n)
    out = {c: s.field(c) for c in range(6) if np.prod(s.shape(c))}
    out["t"], out["max"] = s.t, s.max_e2()
    for q in planes:
        out["dft"] = s.dft(q)
    if probes:
        out["probes"] = s.probes()
    if series:
        out["steps"], out["series"] = s.max_series()
    s.close()
    return out


@pytest.mark.parametrize("name,precision,monitor,every,probes,series", RUNS)
def test_sequences_equal_single_steps(engine, name, precision, monitor, every, probes, series):
    """One call of 100 steps, calls that start and end off a sequence's boundary, and 100 calls of
    one step.  The series is compared on the steps that monitor_every asks for: every call's last
    step is recorded besides."""
    ones = _run(name, precision, monitor, every, probes, series, [1] * 100)
    for calls in ([100], [3, 60, 37], [5, 0, 31, 64]):
        got = _run(name, precision, monitor, every, probes, series, calls)
        assert got.keys() == ones.keys()
        for k in ones:
            if k in ("steps", "series"):
                continue
            assert np.array_equal(got[k], ones[k]), (calls, k)
        if series:
            ends = np.cumsum(calls) - 1
            want = [t for t in range(100) if (monitor and (t + 1) % monitor == 0) or t in ends][:60]
            assert got["steps"].tolist() == want
            ref = dict(zip(ones["steps"].tolist(), ones["series"]))  # the first 60 steps
            for t, v in zip(got["steps"].tolist(), got["series"]):
                assert t not in ref or v == ref[t], t


def test_sequence_follows_configuration_changes(engine):
    """What a captured sequence was given may change between calls: a DFT plane, probes, the series,
    the stream and a reset."""
    import torch

    from luxum_gb300 import Sim

    p, _, boxes = cases.build("planar_pml_axis")
    p.precision = 1

    def run(chunked):
        s = Sim(p)
        step = (lambda n: s.step(n)) if chunked else (lambda n: [s.step(1) for _ in range(n)])
        step(64)
        q = s.add_dft_plane(2, 20, [2e10], 4)
        step(48)
        s.set_probes([[20, 0, 30]], 40)
        step(40)
        a = (s.dft(q), s.probes(), s.field(1))
        st = torch.cuda.Stream()
        s.set_stream(st.cuda_stream)
        step(40)
        s.set_stream(None)
        step(48)
        b = (s.field(3), s.dft(q))
        s.reset()
        step(56)
        c = (s.field(1), s.dft(q), s.probes())
        s.close()
        return a + b + c

    for x, y in zip(run(True), run(False)):
        assert np.array_equal(x, y)
