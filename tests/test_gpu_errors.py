"""Error paths of the CUDA engine that are tested without faulting a GPU.

* A bounded wait that runs out: the marching kernel's test hook arms one
  ring barrier with more expected bytes than its copies deliver (every copy
  lands; the phase never completes), its waits give up after 20 ms, the
  block sets the timeout flag and returns. The next check reports
  EMS_ERR_TIMEOUT; the handle and the context stay usable.
* The same of the resident kernel: its first barrier waits for a block more
  than there is; every read reports it, once.
* Divergence: a NaN uploaded into a field makes the next marching step write
  non-finite values; the next check reports EMS_ERR_DIVERGED, and the run
  loop ends with the Diverged outcome (src/engine/run.rs:156-161).
"""
import numpy as np
import pytest

import ems_b200 as E
from ems_b200 import workloads as W
from oracle import OracleEngine
from helpers import assert_fields_equal

pytestmark = pytest.mark.gpu


def _box():
    return W.dispersive_box(n=40, radius=6, slab=3, cpml=4, steps=200)


def test_bounded_wait_runs_out_and_reports_timeout():
    w = _box()
    g = E.Engine(w.model)
    g.set_schedule(7)
    g.run(3)
    g.check()
    g.test_wait_timeout(20_000_000)
    g.run(1)
    with pytest.raises(E.EngineError) as ei:
        g.check()
    assert ei.value.status == E.ERR_TIMEOUT
    # The flag was cleared; the handle steps on.
    g.run(5)
    g.check()
    # The context is usable: a new engine on it matches the oracle.
    h = E.Engine(w.model)
    h.set_schedule(7)
    o = OracleEngine(w.model, threads=4)
    h.run(30)
    o.run(30)
    h.check()
    assert_fields_equal(h, o, "after a bounded wait ran out")


def test_nan_field_reports_divergence():
    w = _box()
    g = E.Engine(w.model)
    g.set_schedule(7)
    g.run(4)
    g.check()
    u = g.field(0, 2)
    u[20, 20, 20] = np.nan
    g.set_field(0, 2, u)
    g.run(2)
    with pytest.raises(E.EngineError) as ei:
        g.check()
    assert ei.value.status == E.ERR_DIVERGED


def test_run_loop_ends_diverged_on_nan():
    w = _box()
    g = E.Engine(w.model)
    g.set_schedule(7)
    g.run(10)
    u = g.field(1, 0)
    u[10, 12, 14] = np.inf
    g.set_field(1, 0, u)
    out = E.run_until(g, E.energy_decay_limits(2000, -40.0, w.model.dt))
    assert out.reason == 2  # Diverged
    assert out.checks == 1


def _resident():
    m = E.Model.uniform([40, 30, 33], [1e-3] * 3)
    m.build(courant=0.95)
    m.add_cpml([4] * 6)
    src = m.add_source_table(E.SOFT_E, [(E.Z, (20, 15, 16), 1.0)], np.sin(0.3 * np.arange(100)))
    return m, src, m.add_probe(E.VOLTAGE, [(E.Z, (21, 15, 16), 1.0)])


@pytest.mark.parametrize("read", ["check", "last_sample", "samples", "field", "energy"])
def test_resident_wait_runs_out_and_every_read_reports_it(read):
    m, _, probe = _resident()
    g = E.Engine(m)
    g.run(3)
    g.last_sample(probe)
    g.test_wait_timeout(5_000_000)
    g.run(2)
    call = {"check": g.check, "last_sample": lambda: g.last_sample(probe), "samples": lambda: g.samples(probe),
            "field": lambda: g.field(0, 2), "energy": g.step_with_energy}[read]
    with pytest.raises(E.EngineError) as ei:
        call()
    assert ei.value.status == E.ERR_TIMEOUT
    # Reported once; the handle and the device step on.
    for _ in range(2):
        g.run(2)
        g.last_sample(probe)
        call()
    h, o = E.Engine(m), OracleEngine(m, threads=4)
    h.run(30)
    o.run(30)
    h.check()
    assert_fields_equal(h, o, "after a bounded wait ran out")


@pytest.mark.parametrize("read", ["samples", "field", "energy"])
def test_batch_wait_runs_out_and_every_read_reports_it(read):
    m, _, probe = _resident()
    b = E.Batch([m, m], max_steps=100)
    b.run(3)
    b.test_wait_timeout(5_000_000)
    b.run(2)
    call = {"samples": lambda: b.samples(0, probe), "field": lambda: b.field(0, 0, 2), "energy": b.step_with_energy}[read]
    with pytest.raises(E.EngineError) as ei:
        call()
    assert ei.value.status == E.ERR_TIMEOUT
    b.run(2)
    call()
    assert b.samples(1, probe).size == b.timestep(1)


@pytest.mark.parametrize("schedule", [0, 4])
@pytest.mark.parametrize("grown", [0, 1, 2, 3, 4])
def test_no_room_for_samples_loses_none(schedule, grown):
    """Memory runs out while the series grow (some of them moved already): the
    run is refused before any of its steps, the counts stay, and steps that
    need no more room go on with every sample in place."""
    m, _, first = _resident()
    amp = np.cos(0.1 * np.arange(50))
    port = m.add_lumped_port_table(E.Y, [9, 9, 9], [9, 11, 9], 50.0, amp)
    second = m.add_probe(E.CURRENT, [(E.X, (20, 15, 16), 1.0)])
    series = [(first, 0), (port, 0), (port, 1), (port, 2), (second, 0)]
    g, want = E.Engine(m), E.Engine(m)
    for e in (g, want):
        e.set_schedule(schedule)
        e.run(1000)  # series hold 1024 samples
    if schedule:
        g.run(24)
        want.run(24)
    g.test_fail_alloc(1 + grown)
    with pytest.raises(E.EngineError) as ei:
        g.run(30)
    assert ei.value.status == E.ERR_NOMEM
    assert g.timestep == want.timestep and all(g.samples(*q).size == g.timestep for q in series)
    for n in (20, 60):
        g.run(n)
        want.run(n)
        for q in series:
            x, y = g.samples(*q), want.samples(*q)
            assert x.size == y.size == g.timestep and np.array_equal(x.view(np.uint64), y.view(np.uint64)), (n, q)
    assert_fields_equal(g, want, "after running out of memory")
