"""Resident steps (many steps per launch, the automatic schedule on small
grids) against the split schedule's kernels, one step at a time: every
operator they run, odd and tiny grids, short and long runs, energy steps,
uploads, amplitudes fed while running and schedule switches between them.
Fields and series must agree bit for bit."""
import numpy as np
import pytest

import ems_b200 as E
from ems_b200 import workloads as W
from helpers import assert_fields_equal, graded, mixed_model

pytestmark = pytest.mark.gpu


def _cavity(n, kappa=0.003, layers=0):
    m = E.Model(*[graded(q * 1e-3, q, 0.2) for q in n])
    h = [q // 2 for q in n]
    m.fill(m.cells().box([0, 0, 0], [n[0], n[1], max(1, h[2])]), m.material(eps_r=3.0, kappa=kappa))
    m.build(courant=0.99)
    if layers:
        m.add_cpml([layers] * 6)
    amp = np.sin(0.3 * np.arange(400))
    src = m.add_source_table(E.SOFT_E, [(E.Z, (h[0], h[1], 0), 1.0)], amp)
    m.add_source_table(E.HARD_E, [(E.X, (0, h[1], h[2]), 0.5)], amp[::-1].copy())
    ops = [m.add_probe(E.VOLTAGE, [(E.Z, (h[0], j, 0), 0.5 + j) for j in range(1, n[1])], interval=3),
           m.add_probe(E.CURRENT, [(E.Y, (0, j % n[1], 0), 1.0) for j in range(70)], f32_sum=True),
           m.add_probe(E.VOLTAGE, [(E.X, (0, 1, 1), 1.0)])]
    return m, src, [(op, 0) for op in ops]


def _mixed(scheme):
    m, ops = mixed_model(scheme=scheme, steps=400)
    return m, None, [(ops["pv"], 0), (ops["pi"], 0), (ops["pe"], 0), (ops["port"], 0), (ops["port"], 1),
                     (ops["port"], 2)]


def _lumped():
    m, src, s = _cavity((14, 9, 11), layers=2)
    amp = np.cos(0.2 * np.arange(300))
    a = m.add_lumped(E.Z, [4, 4, 2], [4, 6, 5], r=50.0, l=2e-9, c=1e-12, series=True, record=True, amp=amp)
    b = m.add_lumped_port_table(E.X, [6, 2, 3], [9, 2, 3], 75.0, amp)
    return m, src, s + [(a, 0), (b, 0), (b, 1), (b, 2)]


CASES = {
    "mixed_trapezoidal": lambda: _mixed(E.TRAPEZOIDAL), "mixed_leapfrog": lambda: _mixed(E.LEAPFROG),
    "tiny": lambda: _cavity((2, 2, 2)), "flat": lambda: _cavity((41, 3, 2)), "rows_33": lambda: _cavity((7, 12, 33)),
    "cpml_overlap": lambda: _cavity((9, 9, 9), layers=4), "cpml_odd": lambda: _cavity((31, 22, 45), layers=5),
    "lumped": _lumped,
}


@pytest.mark.parametrize("curl", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_resident_equals_split(name, curl):
    m, src, series = CASES[name]()
    g, s = E.Engine(m), E.Engine(m)
    s.set_schedule(4)
    for e in (g, s):
        e.set_curl_order(curl)
    rng = np.random.default_rng(5)
    before = g.launches
    for e in (g, s):
        e.run(60)
    assert g.launches - before == 1 and g.schedule == 4
    assert_fields_equal(g, s, f"{name}: 60 steps")
    for n in (1, 2, 7, 0, 31):
        if src is not None:
            v = rng.standard_normal(3)
            for e in (g, s):
                e.source_amplitude(src, e.timestep, v)
        w = [e.step_with_energy() for e in (g, s)]
        assert abs(w[0] - w[1]) <= 1e-12 * abs(w[1])
        u = rng.standard_normal(g.nodes).astype(np.float32)
        for e in (g, s):
            e.set_field(n % 2, n % 3, u)
            e.run(n)
    g.set_schedule(1)
    g.run(3)
    g.set_schedule(0)
    g.run(5)
    s.run(8)
    assert g.timestep == s.timestep
    assert_fields_equal(g, s, name)
    for op, which in series:
        x, y = g.samples(op, which), s.samples(op, which)
        assert x.size == y.size > 0
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64)), (name, op, which)


def _poles(n, sides, cpml, source, first=False):
    """Poles that keep only part of a gang busy; a source on a pole edge makes
    the saved values be captured every step; first: before the CPML."""
    m = E.Model.uniform(n, [1e-3] * 3)
    m.build(courant=0.95)
    h = [q // 2 for q in n]

    def poles():
        d = E.Dispersive()
        if sides != "magnetic":
            d.fill_cells(m, m.cells().box([h[0], h[1], 2], [n[0] - 2, n[1] - 2, n[2] - 2]), W.lorentz_poles(5))
        if sides != "electric":
            d.fill_cells(m, m.cells().box([2, 2, h[2]], [h[0], h[1], n[2] - 1]), [E.Pole.drude(2e10, 3e9)], field=1)
        m.add_dispersive(d, E.LEAPFROG)

    if first:
        poles()
    if cpml:
        m.add_cpml([4] * 6)
    if not first:
        poles()
    if source:
        m.add_source_table(E.SOFT_E, [(E.Z, (h[0] + 2, h[1] + 2, h[2]), 1.0)], np.cos(0.2 * np.arange(100)))
    return m


@pytest.mark.parametrize("sides", ["electric", "magnetic", "both"])
@pytest.mark.parametrize("cpml,source,first", [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (1, 0, 1), (1, 1, 1)])
def test_resident_poles_equal_split(sides, cpml, source, first):
    """Electric and magnetic poles over a gang of many blocks, resident against
    split and in a batch, from nonzero fields and after an upload."""
    n = (61, 45, 53)
    m = _poles(n, sides, cpml, source, first)
    g, s = E.Engine(m), E.Engine(m)
    s.set_schedule(4)
    rng = np.random.default_rng(11)
    for e in (g, s):
        before = e.launches
        e.run(1)
        assert (e.launches - before == 1) == (e is g)
    for steps in (7, 1, 12):
        u = [rng.standard_normal(g.nodes).astype(np.float32) for _ in range(2)]
        for e in (g, s):
            for f in range(2):
                e.set_field(f, 2, u[f])
            e.run(steps)
        assert_fields_equal(g, s, f"{steps} steps")
    if source:
        b = E.Batch([m, _cavity((9, 8, 7))[0], m], max_steps=100)
        s = E.Engine(m)
        s.set_schedule(4)
        for steps in (30, 11):
            b.run(steps)
            s.run(steps)
        for q in (0, 2):
            for f in range(2):
                for a in range(3):
                    assert np.array_equal(b.field(q, f, a).view(np.uint32), s.field(f, a).view(np.uint32)), (q, f, a)


def test_batch_of_more_models_than_blocks():
    """More models than resident blocks (two per SM): a block takes several,
    each for the whole run."""
    sizes = [(3 + q % 5, 4 + q % 3, 2 + q % 7) for q in range(320)]
    built = [_cavity(n)[0] for n in sizes]
    b = E.Batch(built, max_steps=200)
    b.run(20)
    for q in (0, 3, 317):
        b.set_active(q, False)
    b.run(13)
    for q in (0, 1, 3, 100, 317, 319):
        g = E.Engine(built[q])
        g.set_schedule(4)
        g.run(20 if q in (0, 3, 317) else 33)
        assert b.timestep(q) == g.timestep
        for f in range(2):
            for a in range(3):
                assert np.array_equal(b.field(q, f, a).view(np.uint32), g.field(f, a).view(np.uint32)), (q, f, a)


def test_long_runs_are_cut_into_launches():
    """A launch holds its SMs to its end: at most 128 steps each."""
    m = _cavity((12, 9, 10))[0]
    g, s = E.Engine(m), E.Engine(m)
    for n, launches in ((1, 1), (128, 1), (129, 2), (1000, 8)):
        before = g.launches
        g.run(n)
        assert g.launches - before == launches
    s.set_schedule(4)
    s.run(1258)
    assert_fields_equal(g, s, "cut into launches")


def test_large_grids_keep_the_split_kernels():
    w = W.vacuum_box(n=224, cpml=8, steps=10)
    g = E.Engine(w.model)
    before = g.launches
    g.run(4)
    assert g.launches - before > 4 * 4


@pytest.mark.parametrize("n,resident", [(138, True), (162, False)])
def test_form_without_a_cpml(n, resident):
    """96 MB of fields are the bound of PEC boxes (162^3: 100 MB)."""
    g = E.Engine(_cavity((n, n, n))[0])
    before = g.launches
    g.run(4)
    assert (g.launches - before == 1) == resident


@pytest.mark.parametrize("n,gangs", [(72, True), (150, False)])
def test_form_of_a_batch_with_poles(n, gangs):
    """Large models with poles step by graph: no gang waits. Either way the
    models equal the same ones alone."""
    m = _poles((n, n, n), "electric", 1, 1)
    b = E.Batch([m, m], max_steps=100)
    s = E.Engine(m)
    s.set_schedule(4)
    b.run(7)
    s.run(7)
    for a in range(3):
        assert np.array_equal(b.field(1, 0, a).view(np.uint32), s.field(0, a).view(np.uint32))
    b.test_wait_timeout(5_000_000)
    b.run(1)
    if gangs:
        with pytest.raises(E.EngineError):
            b.field(0, 0, 2)
    else:
        b.field(0, 0, 2)


def test_engines_on_several_threads():
    """Resident engines and a batch stepping at once from threads of their
    own (each launch fills the device): every result as when alone."""
    import threading

    m, _, series = _cavity((40, 33, 47), layers=5)
    small = [_cavity((9 + q, 11, 13))[0] for q in range(6)]
    want = E.Engine(m)
    want.run(600)
    alone = [E.Engine(x) for x in small]
    for e in alone:
        e.run(600)
    engines = [E.Engine(m) for _ in range(3)]
    b = E.Batch(small, max_steps=700)
    errors = []

    def go(x, n):
        try:
            for _ in range(600 // n):
                x.run(n)
            if isinstance(x, E.Engine):
                x.check()
        except BaseException as err:  # reported below
            errors.append(err)

    threads = [threading.Thread(target=go, args=(x, n)) for x, n in zip([*engines, b], (1, 20, 300, 5))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for e in engines:
        assert_fields_equal(e, want, "threads")
        for op, which in series:
            assert np.array_equal(e.samples(op, which), want.samples(op, which))
    for q, e in enumerate(alone):
        assert b.timestep(q) == 600 and b.samples(q, 2).size == 200
        assert np.array_equal(b.field(q, 0, 2).view(np.uint32), e.field(0, 2).view(np.uint32))


def test_autotuning_times_the_resident_form(tmp_path):
    """The candidate of the split schedule is timed in the form that will run:
    one warm-up step, then many steps per launch; the same for a batch."""
    cache = str(tmp_path / "tune.txt")
    m = _cavity((33, 20, 17), layers=4)[0]
    g, s = E.Engine(m), E.Engine(m)
    s.set_schedule(4)
    g.autotune(cache)
    for n, launches in ((1, 1), (9, 1), (7, 1)):
        before = g.launches
        g.run(n)
        assert g.launches - before == launches
    g.run(60)
    s.run(77)
    assert_fields_equal(g, s, "tuned")
    key, pick, _ = open(cache).read().strip().rsplit(" ", 2)
    assert key.startswith("engine ") and "resident=1" in key
    h = E.Engine(m)
    h.autotune(cache)
    assert h.schedule == int(pick) == g.schedule
    before = h.launches
    h.run(40)
    assert (h.launches - before == 1) == (int(pick) == 4)
    b = E.Batch([m, m], max_steps=200)
    b.autotune(cache)
    b.test_wait_timeout(5_000_000)
    b.run(1)
    with pytest.raises(E.EngineError):
        b.field(0, 0, 2)
    b = E.Batch([m, m], max_steps=200)
    b.autotune(cache)
    for n in (20, 57):
        b.run(n)
    assert b.timestep(1) == 77
    for a in range(3):
        assert np.array_equal(b.field(1, 0, a).view(np.uint32), s.field(0, a).view(np.uint32))
    line = open(cache).read().splitlines()[-1]
    assert line.startswith("batch ") and "gangs=1" in line and 0 <= int(line.split()[-2]) < 6
    c = E.Batch([m, m], max_steps=200)
    c.autotune(cache)
    c.run(77)
    assert np.array_equal(c.field(0, 1, 2).view(np.uint32), s.field(1, 2).view(np.uint32))
