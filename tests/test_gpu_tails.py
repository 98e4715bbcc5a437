"""States in the tail of a front: momenta and depth differences down to denormal numbers
beside larger ones, where the Riemann solvers' branch-free divisions hand over to the
operators, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fusion", [1, 2])
@pytest.mark.parametrize("order", [(1, 0), (2, 2)])
@pytest.mark.parametrize("system", ["swe", "euler"])
def test_tail_states_equal_oracle(gpu_lib, system, order, fusion):
    import forestclaw_b200 as fcb

    make = cases.radialdam_uniform if system == "swe" else cases.quadrants_uniform
    cfg = cases.replace(make(level=1, mx=16), order=order)
    o = O.OracleSolver(cfg)
    o.initialize()
    g = np.random.default_rng(3)
    q = o.all_q()
    shape = (q.shape[0],) + q.shape[2:]
    q[:, 0] = np.where(g.random(shape) < 0.5, 1.0, np.nextafter(1.0, 2.0))
    for m in (1, 2):
        size = np.ldexp(g.uniform(1.0, 2.0, shape), g.integers(-1080, -900, shape))
        q[:, m] = np.where(g.random(shape) < 0.1, 0.0, size * g.choice([-1.0, 1.0], shape))
    if system == "euler":
        q[:, 3] = 2.5
    opts = cases.to_options(cfg)
    opts.ghost_fusion = fusion
    d = fcb.Solver(opts)
    d.initialize()
    for p in range(q.shape[0]):
        o.set_q(p, q[p])
    d.set_q(q)
    dt = 0.2 / 32
    for s in (o, d):
        s.ghost_update(1, 1, 0.0, 0)
    for k in range(4):
        assert d.advance_all_levels(k * dt, dt) == o.advance(k * dt, dt)
    assert np.array_equal(d.get_q(), o.all_q())
    d.close()
