"""FP64 states at sizes that FP32 cannot hold: the helpers that start from FP32 values
have no range of their own."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import GROUPS, all_tools, perturbed_state, rel_err, small_scene
from diffskill_gb300.engine import MpmEngine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


# velocities whose squares are in and above FP32.s range
@pytest.mark.parametrize("speed", [1e3, 1e25, 1e120])
def test_substep_of_very_fast_particles(gpu_lib, speed):
    """Forward substep against the oracle where the velocities meet every tool and wall:
    the contact takes the lengths of velocities up to 1e120.  (Affine fields and strains as
    usual; relative tolerance of the FP64 substep test.)"""
    tools = all_tools()
    sc = small_scene(n=1500, tools=tools, precision="fp64")
    st = perturbed_state(sc.x0, seed=2, v=1.0)
    st[:, 3:6] *= speed
    eng, o = MpmEngine(sc.sim, [tools], [sc.n_particles]), Oracle(sc.sim, tools)
    s0, s1 = eng.new_state(), eng.new_state()
    s0[:, :sc.n_particles] = torch.as_tensor(st.T, device=eng.device)
    eng.substep(s0, s1, eng.pose0, eng.pose0)
    torch.cuda.synchronize()
    assert eng.status() == 0
    ref = o.substep(o.pose0(), o.pose0(), st)
    got = s1[:, :sc.n_particles].cpu().numpy().T
    assert np.isfinite(ref).all()
    for k, sl in GROUPS.items():
        assert rel_err(got[:, sl], ref[:, sl]) < 1e-9, k
