"""Level updates that the tuner cannot time (a stream capture, with no choice made for
their kind before) run the default form, at every patch size."""
from __future__ import annotations

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mx", [8, 16, 32, 64])
def test_level_update_recorded_before_any_tuning(gpu_lib, mx):
    import torch

    import forestclaw_b200 as fcb

    # limiter 6 with 4 patches: a kind of update that nothing else tunes
    cfg = cases.replace(cases.swirl_uniform(level=1, mx=mx), mthlim=(6,))
    dt = cases.swirl_dt(level=1, mx=mx)
    got = []
    for recorded in (True, False):
        st = torch.cuda.Stream()
        o = cases.to_options(cfg)
        o.ghost_fusion = 1
        s = fcb.Solver(o, stream=st.cuda_stream)
        s.initialize()
        s.ghost_update(1, 1, 0.0, 0)
        st.synchronize()
        if recorded:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=st):
                s.update_single_step_async(1, 0.0, dt)
            with torch.cuda.stream(st):
                g.replay()
        else:
            s.update_single_step(1, 0.0, dt)
        st.synchronize()
        got.append(s.get_q())
        s.close()
    assert np.array_equal(got[0], got[1])
