"""Scalar advection on a mesh of one level whose cell edges are not exact in double
precision: the step with the ghost exchange folded in runs (patch by patch) and equals
the unfused one bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu

INEXACT = (0.0, 0.3, -0.1, 0.6)


def _swirl(level, mx, **kw):
    return cases.replace(cases.swirl_uniform(level=level, mx=mx), extent=INEXACT, **kw), level, 0.25 / (mx << level)


def _stored(level, mx, **kw):
    kw = dict(dict(minlevel=level, maxlevel=level, regrid_interval=0, use_fixed_dt=1, mx=mx, my=mx, extent=INEXACT), **kw)
    return cases.replace(O.periodic_regression(4), **kw), level + 1, 0.1 / (mx << level + 1)


CASES = {
    "swirl_one_patch": lambda: _swirl(0, 8),
    "swirl_walls": lambda: _swirl(2, 16, mthbc=(3, 3, 3, 3)),
    "swirl_mixed_sides": lambda: _swirl(3, 32, mthbc=(3, 1, 1, 3), mthlim=(3,)),
    "swirl_v5": lambda: _swirl(3, 8, claw_version=5, mthlim=(2,)),
    "swirl_order1": lambda: _swirl(2, 16, order=(1, 0)),
    "stored_periodic": lambda: _stored(2, 16),
    "stored_periodic_y": lambda: _stored(1, 32, periodic_x=0, mthbc=(3, 1, 1, 1)),
    "stored_one_block": lambda: _stored(2, 8, periodic_x=0, periodic_y=0, claw_version=5),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fused_patches_equal_unfused(gpu_lib, name, precision):
    import forestclaw_b200 as fcb

    cfg, level, dt = CASES[name]()
    got = []
    for fusion in (1, 2):
        o = cases.to_options(cfg)
        o.ghost_fusion, o.precision = fusion, precision
        s = fcb.Solver(o)
        s.initialize()
        s.ghost_update(level, level, 0.0, 0)
        q = s.get_q()
        q += 0.1 * np.random.default_rng(7).uniform(size=q.shape)
        s.set_q(q)
        s.ghost_update(level, level, 0.0, 0)
        cfl = [s.advance_all_levels(k * dt, dt) for k in range(3)]
        _, fused = s.step_kernel_time(0.0, dt, 1)
        assert fused == (fusion == 2)
        got.append((cfl, s.get_q()))
        s.close()
    (c1, q1), (c2, q2) = got
    assert 0.0 < max(c1) <= 1.0
    if precision == 0:
        assert c1 == c2 and np.array_equal(q1, q2)
    else:  # FP32 interfaces, contracted differently by the two instantiations
        assert np.allclose(c1, c2, rtol=1e-5)
        assert np.max(np.abs(q1 - q2)) <= 3 * 64 * np.finfo(np.float32).eps * np.max(np.abs(q1))
