"""g2p's gathers by cell, which callers that re-sort their frames get, on frames that are
not sorted (any more)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import GROUPS, perturbed_state, small_scene
from diffskill_gb300.engine import MpmEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sort", [True, False])
def test_g2p_of_a_caller_that_sorts_equals_one_that_does_not(gpu_lib, sort):
    """More particles than a wave of CTAs holds (8 x 128 per SM), a ragged last warp and one
    particle outside the grid.  One handle has sorted a frame and so fetches a cell's nodes
    once per warp, the other has not and gathers lane by lane; unsorted, most warps hold
    more cells than fit.  (The two runs' grids differ in the order of their FP32 sums: 1e-7;
    1e-6 relative in C.)"""
    n = 8 * 128 * torch.cuda.get_device_properties(0).multi_processor_count + 77
    sc = small_scene(n=64, tools=[], precision="fp32")
    rng = np.random.default_rng(1)
    aos = perturbed_state(rng.uniform(0.3, 0.5, (n, 3)), seed=1)
    aos[5, 0] = 7.0
    outs = []
    for sorts in (True, False):
        eng = MpmEngine(sc.sim, [[]], [n])
        other = MpmEngine(sc.sim, [[]], [n])
        st = eng.new_state()
        st[:, :n] = torch.as_tensor(aos.T, dtype=eng.dtype, device=eng.device)
        by_cell, perm = eng.new_state(), torch.empty(n, dtype=torch.int32, device=eng.device)
        (eng if sorts else other).sort_frame(st, by_cell, perm)
        pose = torch.zeros((1, 8), dtype=torch.float64, device=eng.device)
        st1 = eng.new_state()
        eng.substep(by_cell if sort else st, st1, pose, pose)
        torch.cuda.synchronize()
        outs.append(st1[:, :n].double())
    for sl in GROUPS.values():
        assert float((outs[0][sl] - outs[1][sl]).abs().max()) <= 1e-5 * float(outs[1][sl].abs().max())
