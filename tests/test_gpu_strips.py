"""Steps of a mesh of one level in strips (ghost_fusion 2) against patches and a
ghost fill (ghost_fusion 1), bit for bit, at the sizes where a strip can go
wrong: tall strips, a last strip narrower or lower than the others, patches of
every size, walls, periodic sides, every solver, mixed precision."""
from __future__ import annotations

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _swirl(level, mx, **kw):
    cfg = cases.replace(cases.swirl_uniform(level=level, mx=mx), **kw)
    return cfg, cases.swirl_dt(level=level, mx=mx)


def _dam(level, mx, **kw):
    return cases.replace(cases.radialdam_uniform(level=level, mx=mx), **kw), 0.3 / (mx << level)


def _euler(level, mx, **kw):
    return cases.replace(cases.quadrants_uniform(level=level, mx=mx), **kw), 0.15 / (mx << level)


WALLS = (3, 3, 3, 3)
CASES = {
    "swirl_tall": lambda: _swirl(8, 16),              # strips of 241 rows
    "swirl_one_patch": lambda: _swirl(0, 8),          # fewer columns than a warp
    "swirl_mx64": lambda: _swirl(2, 64, mthlim=(3,)),
    "swirl_v5": lambda: _swirl(5, 8, claw_version=5, mthlim=(2,)),
    "dam_walls_mx8": lambda: _dam(6, 8, mthbc=WALLS),
    "dam_mixed_sides": lambda: _dam(4, 16, mthbc=(3, 1, 1, 3), mthlim=(3, 4, 1)),
    "dam_mx64": lambda: _dam(2, 64, mthbc=(1, 3, 3, 1)),
    "dam_v5": lambda: _dam(4, 32, claw_version=5, mthbc=WALLS),
    "dam_order1": lambda: _dam(3, 16, order=(1, 0)),
    "dam_transverse1": lambda: _dam(3, 16, order=(2, 1)),
    "euler": lambda: _euler(5, 16),
    "euler_v5": lambda: _euler(4, 8, claw_version=5),
    "lake": lambda: (cases.bathy_lake(level=4, mx=16), 0.2 / 256),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", sorted(CASES))
def test_strips_equal_patches(gpu_lib, name, precision):
    import forestclaw_b200 as fcb

    cfg, dt = CASES[name]()
    if precision and (cfg.mx == 64 or cfg.order[0] == 1):
        pytest.skip("no mixed patches of this size; first order tested in FP64")
    got = []
    for fusion in (1, 2):
        o = cases.to_options(cfg)
        o.ghost_fusion, o.precision = fusion, precision
        s = fcb.Solver(o)
        s.initialize()
        s.ghost_update(cfg.minlevel, cfg.maxlevel, 0.0, 0)
        g = np.random.default_rng(5)
        q = s.get_q()
        q *= 1.0 + 0.01 * g.uniform(-1.0, 1.0, size=(q.shape[0],) + (1,) * (q.ndim - 1))
        s.set_q(q)
        s.ghost_update(cfg.minlevel, cfg.maxlevel, 0.0, 0)
        t, cfl = 0.0, []
        for _ in range(3):
            cfl.append(s.advance_all_levels(t, dt))
            t += dt
        got.append((cfl, s.get_q()))
        assert s.step_kernel_time(t, dt, 1)[1] == (fusion == 2)  # strips ran, patches ran
        s.close()
    (c1, q1), (c2, q2) = got
    if precision == 0:
        assert c1 == c2
        assert np.array_equal(q1, q2)
    else:  # FP32 interfaces, contracted differently by the two instantiations
        assert np.allclose(c1, c2, rtol=1e-5)
        assert np.max(np.abs(q1 - q2)) <= 3 * 64 * np.finfo(np.float32).eps * np.max(np.abs(q1))


@pytest.mark.parametrize("precision", [0, 1])
def test_strips_periodic_brick(gpu_lib, precision):
    """A periodic 2 x 2 brick (stored aux): the strip wraps around."""
    import forestclaw_b200 as fcb
    import oracle as O

    cfg = cases.replace(O.periodic_regression(4), minlevel=3, maxlevel=3, regrid_interval=0, use_fixed_dt=1)
    got = []
    for fusion in (1, 2):
        o = cases.to_options(cfg)
        o.ghost_fusion, o.precision = fusion, precision
        s = fcb.Solver(o)
        s.initialize()
        s.ghost_update(4, 4, 0.0, 0)  # level 3 of each block of the brick
        dt = 0.5 * 2.0 / (cfg.mx * cfg.brick * 8)
        for k in range(3):
            s.advance_all_levels(k * dt, dt)
        got.append(s.get_q())
        assert s.step_kernel_time(0.0, dt, 1)[1] == (fusion == 2)
        s.close()
    if precision == 0:
        assert np.array_equal(got[0], got[1])
    else:
        assert np.max(np.abs(got[0] - got[1])) <= 3 * 64 * np.finfo(np.float32).eps * np.max(np.abs(got[0]))
