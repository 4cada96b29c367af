"""Rounding of one sign in the adjoint of one substep adds up over a horizon."""
from __future__ import annotations

import pytest
import torch

from _util import perturbed_state, small_scene
from diffskill_gb300.engine import MpmEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strain", [5e-4, 2e-3])
def test_fp32_adjoint_of_elastic_F_keeps_its_length(gpu_lib, strain):
    """With a gradient of F alone and C = 0 an elastic particle's gradient passes a substep
    unchanged.  Its mean scale, over 20,000 particles, may be off by 1e-8 (5e-5 over 5,000
    substeps); unbiased rounding of some ten products leaves 1e-9."""
    n = 20000
    sc = small_scene(n=n, tools=[], precision="fp32")
    eng = MpmEngine(sc.sim, [[]], [n])
    st, g1, g0 = eng.new_state(), eng.new_state(), eng.new_state()
    st[:, :n] = torch.as_tensor(perturbed_state(sc.x0, seed=3, v=0.0, C=0.0, F=strain).T, dtype=eng.dtype,
                                device=eng.device)
    gen = torch.Generator(device="cuda").manual_seed(4)
    g1[15:24, :n] = torch.randn((9, n), generator=gen, device="cuda")
    pose = torch.zeros((4, 1, 8), dtype=torch.float64, device=eng.device)
    st1 = eng.new_state()
    eng.substep(st, st1, pose[0], pose[1])
    eng.substep_bwd(st, g1, g0, pose[0], pose[1], pose[2], pose[3], st1=st1)
    a, b = g0[15:24, :n].double(), g1[15:24, :n].double()
    assert float((a - b).norm() / b.norm()) < 2e-6
    assert abs(float((a * b).sum() / (b * b).sum()) - 1.0) < 1e-8
