"""openEMS PML layers whose start values are not refreshed: a model whose layer
edges only the layer update writes, and models where a source or a port acts
on them, with fields uploaded between runs.
Fields and the layers' own state equal the oracle bit for bit."""
import numpy as np
import pytest

import ems_b200 as E
from helpers import assert_fields_equal
from oracle import OracleEngine

pytestmark = pytest.mark.gpu


def _model(where):
    n = (19, 15, 17)
    m = E.Model.uniform(n, [1e-3] * 3)
    m.fill(m.cells().box([0, 0, 0], [n[0], n[1], 8]), m.material(eps_r=2.5, kappa=0.01))
    m.build(courant=0.9)
    op = m.add_openems_pml([4] * 6)
    amp = np.sin(0.3 * np.arange(200))
    m.add_source_table(E.SOFT_E, [(E.Z, (9, 7, 8), 1.0)], amp)
    if where == "soft E in the layer":
        m.add_source_table(E.SOFT_E, [(E.Z, (2, 7, 8), 0.7)], amp)
    elif where == "hard E in the layer":
        m.add_source_table(E.HARD_E, [(E.Y, (9, 7, 1), 0.7)], amp)
    elif where == "H in the layer":
        m.add_source_table(E.SOFT_H, [(E.X, (9, 2, 8), 0.7)], amp)
    elif where == "port into the layer":
        m.add_lumped_port_table(E.Z, [9, 2, 2], [9, 2, 6], 50.0, amp)
    m.add_probe(E.VOLTAGE, [(E.Z, (8, 7, 8), 1.0)])
    return m, op


@pytest.mark.parametrize("schedule", [0, 1, 4])
@pytest.mark.parametrize("where", ["interior", "soft E in the layer", "hard E in the layer", "H in the layer",
                                   "port into the layer"])
def test_layers_equal_the_oracle(where, schedule):
    m, op = _model(where)
    g, o = E.Engine(m), OracleEngine(m, threads=2)
    g.set_schedule(schedule)
    for e in (g, o):
        e.run(12)
    assert_fields_equal(g, o, where)
    rng = np.random.default_rng(1)
    for field, axis in ((0, 2), (1, 0), (0, 0)):
        u = (1e-3 * rng.standard_normal(g.nodes)).astype(np.float32)
        for e in (g, o):
            e.set_field(field, axis, u)
            e.run(5)
    assert_fields_equal(g, o, f"{where} after uploads")
