"""Capacity steps in row bands (chosen by the library for launches that leave the SMs
idle) against the same solve with every patch swept whole (step_variant 1), bit for
bit: a few patches, counts around one wave of CTAs, the smallest and largest patches.
Bands show in the launch count: the copy of the patches that they read is a launch more
for every level update.  Large launches are banded too where the bands' smaller aux tile
lets more CTAs share an SM (mx = 32); at mx = 8 it does not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mx,minlevel,maxlevel,version,banded", [
    (8, 1, 1, 4, True), (8, 3, 5, 5, True), (16, 2, 4, 4, True), (32, 2, 2, 5, True), (32, 3, 4, 4, True),
    (32, 4, 4, 4, True), (64, 2, 3, 4, True), (8, 7, 7, 4, False), (32, 6, 6, 5, True)])
def test_banded_equals_whole(gpu_lib, mx, minlevel, maxlevel, version, banded):
    import forestclaw_b200 as fcb
    from forestclaw_b200 import workloads

    out = []
    for variant in (0, 1):
        o = workloads.filament(minlevel=minlevel, maxlevel=maxlevel, mx=mx, claw_version=version)
        o.step_variant = variant
        o.regrid_interval = 0
        o.macro_graph = 0  # one launch per level update
        s = fcb.Solver(o)
        s.initialize()
        dt = 0.08 / (mx << minlevel)
        n0 = s.counters()
        cfl = [s.advance_all_levels(k * dt, dt) for k in range(3)]
        n1 = s.counters()
        launches = n1["count_kernel_launches"] - n0["count_kernel_launches"]
        levels = sorted({lv for lv, _, _ in s.leaves()})
        updates = 3 * sum(1 << (lv - minlevel - 1) for lv in levels)  # the brick's levels start one up
        out.append((cfl, s.get_q(), launches, updates))
        s.close()
    assert out[0][0] == out[1][0]
    assert np.array_equal(np.asarray(out[0][1]), np.asarray(out[1][1]))
    extra = out[0][2] - out[1][2]
    assert extra == (out[0][3] if banded else 0), (extra, out[0][3])
