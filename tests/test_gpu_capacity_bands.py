"""Capacity steps in row bands (chosen by the library for launches that leave the SMs
idle) against the same solve with every patch swept whole (step_variant 1), bit for
bit: a few patches, counts around one wave of CTAs, the smallest and largest patches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mx,minlevel,maxlevel,version", [
    (8, 1, 1, 4), (8, 3, 5, 5), (16, 2, 4, 4), (32, 2, 2, 5), (32, 3, 4, 4), (32, 4, 4, 4), (64, 2, 3, 4)])
def test_banded_equals_whole(gpu_lib, mx, minlevel, maxlevel, version):
    import forestclaw_b200 as fcb
    from forestclaw_b200 import workloads

    out = []
    for variant in (0, 1):
        o = workloads.filament(minlevel=minlevel, maxlevel=maxlevel, mx=mx, claw_version=version)
        o.step_variant = variant
        o.regrid_interval = 0
        s = fcb.Solver(o)
        s.initialize()
        dt = 0.08 / (mx << minlevel)
        cfl = [s.advance_all_levels(k * dt, dt) for k in range(3)]
        out.append((cfl, s.get_q()))
    assert out[0][0] == out[1][0]
    assert np.array_equal(np.asarray(out[0][1]), np.asarray(out[1][1]))
