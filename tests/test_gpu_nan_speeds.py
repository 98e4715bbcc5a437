"""A velocity that is not a number is reported, not stepped with: strips and patches,
FP64 and mixed, stream function and stored aux."""
from __future__ import annotations

import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu


def _swirl():
    return cases.swirl_uniform(level=3, mx=16), 3, float("nan")  # a NaN time


def _stored():
    cfg = cases.replace(O.periodic_regression(4), minlevel=2, maxlevel=2, regrid_interval=0, use_fixed_dt=1)
    return cases.replace(cfg, pparams=(float("nan"),) + tuple(cfg.pparams[1:])), 3, 0.0  # a NaN velocity


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("fusion", [1, 2])
@pytest.mark.parametrize("case", [_swirl, _stored])
def test_nan_speed_is_reported(gpu_lib, case, fusion, precision):
    import forestclaw_b200 as fcb

    cfg, level, t = case()
    o = cases.to_options(cfg)
    o.ghost_fusion, o.precision = fusion, precision
    s = fcb.Solver(o)
    s.initialize()
    s.ghost_update(level, level, 0.0, 0)
    with pytest.raises(fcb.FcbError, match="NaN CFL"):
        s.advance_all_levels(t, 1e-3)
    s.close()
