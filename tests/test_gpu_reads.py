"""Field downloads through the staging buffers (2 MiB each): grids below one
buffer, ending on one, and over several, with rows that the buffers cut."""
import numpy as np
import pytest

import ems_b200 as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [(3, 3, 3), (33, 65, 31), (64, 128, 64), (65, 128, 64), (131, 113, 101)])
def test_download_returns_what_was_uploaded(nodes):
    m = E.Model.uniform([q - 1 for q in nodes], [1e-3] * 3)
    m.build()
    g = E.Engine(m)
    b = E.Batch([m], max_steps=4)
    rng = np.random.default_rng(nodes[0])
    v = [rng.standard_normal(nodes).astype(np.float32) for _ in range(6)]
    for q, x in enumerate(v):
        g.set_field(q // 3, q % 3, x)
    for _ in range(2):
        for q, x in enumerate(v):
            assert np.array_equal(g.field(q // 3, q % 3).view(np.uint32), x.view(np.uint32)), (nodes, q)
    assert not np.any(b.field(0, 0, 2)) and b.timestep(0) == 0
    b.run(3)
    assert b.timestep(0) == 3


def test_counts_and_newest_samples():
    m = E.Model.uniform([12, 11, 10], [1e-3] * 3)
    m.build()
    amp = np.sin(0.4 * np.arange(64))
    m.add_source_table(E.SOFT_E, [(E.Z, (6, 5, 5), 1.0)], amp)
    every, third = (m.add_probe(E.VOLTAGE, [(E.Z, (6, 5, 4), 1.0)], interval=q) for q in (1, 3))
    cur = m.add_probe(E.CURRENT, [(E.X, (6, 5, 5), 1.0)])
    for schedule in (0, 4, 1):
        g = E.Engine(m)
        g.set_schedule(schedule)
        with pytest.raises(E.EngineError):
            g.last_sample(every)
        assert g.samples(every).size == 0
        for n in (1, 4, 2):
            g.run(n)
            t = g.timestep
            for op, count in ((every, t), (third, (t + 2) // 3), (cur, t)):
                s = g.samples(op)
                assert s.size == count and g.last_sample(op) == s[-1]
