"""Tool kinematics with eight lanes per tool (scenes without collision pairs and rolling
pins) against the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import all_tools, more_tools, rel_err, small_scene
from diffskill_gb300.engine import MpmEngine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


# one tool, a warp's four, one more, and the most a scene may have; the shortest action,
# and one longer than a warp has lanes
@pytest.mark.parametrize("n_tools", [1, 4, 5, 8])
@pytest.mark.parametrize("n_sub", [1, 2, 33])
def test_eight_lanes_per_tool_match_oracle(gpu_lib, n_tools, n_sub):
    """Poses, velocities and both gradients; the adjoint also where the velocity
    changes within the action.  FP64: some 100 operations per substep, 33 substeps."""
    pool = [t for t in more_tools() + all_tools() if not t.shape.startswith("RollingPin")]
    tools = [pool[i % len(pool)] for i in range(n_tools)]
    sc = small_scene(n=64, tools=tools, precision="fp64", substeps=n_sub)
    eng, o = MpmEngine(sc.sim, [tools], [64]), Oracle(sc.sim, tools)
    acts, vel, pseq = o.tools_action(o.pose0(), sc.actions[0])
    dev = {"dtype": torch.float64, "device": eng.device}
    a, v = torch.zeros((o.T, 8), **dev), torch.zeros((n_sub, o.T, 8), **dev)
    p = torch.zeros((n_sub + 1, o.T, 8), **dev)
    a[:, :7] = torch.as_tensor(acts, device=eng.device)
    p[0] = eng.pose0
    eng.tools_action(a, v, p)
    assert rel_err(p.cpu().numpy(), pseq) < 1e-12
    assert rel_err(v.cpu().numpy(), vel) < 1e-12
    for change in (False, True):
        if change:
            vel = np.array(vel)
            vel[n_sub // 2:] *= 0.5
            v.copy_(torch.as_tensor(vel))
        g_ref = np.random.default_rng(n_sub).normal(size=pseq.shape)
        g = torch.as_tensor(g_ref, device=eng.device).clone()
        ga_ref, ga = np.zeros((o.T, 7)), torch.zeros((o.T, 8), **dev)
        o.tools_action_bwd(acts, vel, pseq, o.last_coll, g_ref, ga_ref)
        eng.tools_action_bwd(v, p, g, ga)
        assert rel_err(g.cpu().numpy(), g_ref) < 1e-11
        assert rel_err(ga.cpu().numpy()[:, :7], ga_ref) < 1e-11


# on both sides of where more than four tools take a lane per component
@pytest.mark.parametrize("n_sub", [12, 13])
def test_five_tools_at_the_line_between_the_two_forms(gpu_lib, n_sub):
    test_eight_lanes_per_tool_match_oracle(gpu_lib, 5, n_sub)
