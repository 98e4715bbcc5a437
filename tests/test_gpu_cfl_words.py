"""The CFL number a waited-for step returns is its own, whatever steps that do not
wait left on the device: asynchronous ones, and replays of a caller's graph of them,
which run no host code."""
from __future__ import annotations

import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fusion", [1, 2])
def test_waited_steps_between_asynchronous_ones_and_replays(gpu_lib, fusion):
    import torch

    import forestclaw_b200 as fcb

    cfg = cases.swirl_uniform(level=3, mx=16)
    dt = cases.swirl_dt(level=3, mx=16)
    st = torch.cuda.Stream()
    opts = cases.to_options(cfg)
    opts.ghost_fusion = fusion
    opts.macro_graph = 0  # the caller's graph takes the launches
    s = fcb.Solver(opts, stream=st.cuda_stream)
    s.initialize()
    s.ghost_update(3, 3, 0.0, 0)

    def small():  # the velocities depend on the time alone, so its number is always the same
        return s.advance_all_levels(0.0, 0.125 * dt)

    want = small()
    level = s.update_single_step(3, 0.0, 0.125 * dt)
    assert 0.0 < want == level
    s.ghost_update(3, 3, 0.0, 0)
    s.advance_all_levels_async(0.0, dt)
    assert small() == want
    big = s.read_max_cfl()
    assert big > 4.0 * want
    st.synchronize()
    macro, single = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(macro, stream=st):
        s.advance_all_levels_async(0.0, dt)  # two: the fused step swaps its arenas
        s.advance_all_levels_async(0.0, dt)
    assert small() == want and small() == want
    with torch.cuda.stream(st):
        macro.replay()
    assert small() == want
    assert s.read_max_cfl() == big
    s.ghost_update(3, 3, 0.0, 0)
    st.synchronize()
    with torch.cuda.graph(single, stream=st):
        s.update_single_step_async(3, 0.0, dt)
    s.ghost_update(3, 3, 0.0, 0)
    assert small() == want and small() == want
    s.ghost_update(3, 3, 0.0, 0)
    with torch.cuda.stream(st):
        single.replay()
    assert s.update_single_step(3, 0.0, 0.125 * dt) == want
    s.ghost_update(3, 3, 0.0, 0)
    assert small() == want and small() == want
    st.synchronize()
    s.close()
