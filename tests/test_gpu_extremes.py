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


# inside and outside the plain decompositions' ranges: strongly compressed, near the
# clamp at 0.05 and below it, inverted, stretched; no two values equal or opposite, where
# the derivative is not that of a function of F
SINGULAR = [(1.2, 0.9, 0.7), (1.1, 0.9, 0.21), (1.1, 0.9, 0.19), (1.3, 1.0, 0.08), (1.2, 1.0, -0.5), (1.3, 1.0, -0.1),
            (3.0, 1.0, 0.4), (1.05, 1.0, 0.95), (1.6, 1.1, 0.01), (1.5, 0.6, 0.3), (1.8, 1.5, 0.3), (0.4, 0.3, 0.2)]


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("fp32_svd64", 2e-4), ("fp32", 2e-4)])
def test_substep_and_adjoint_of_extreme_deformations(gpu_lib, prec, tol):
    """Against the oracle on what the device holds.  FP32: 6e-8, times up to 20 from the
    logarithm at the clamp and 10 from the closest pair, through some ten roundings."""
    sc = small_scene(n=300, tools=[], precision=prec)
    rng = np.random.default_rng(21)
    st = perturbed_state(sc.x0, seed=21, C=0.0, F=0.0)
    for p in range(sc.n_particles):
        U, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        V, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        U[:, 2] *= np.linalg.det(U)
        V[:, 2] *= np.linalg.det(V)
        st[p, 15:24] = (U @ np.diag(SINGULAR[p % len(SINGULAR)]) @ V.T).ravel()
    g1 = rng.normal(size=st.shape)
    if prec != "fp64":
        st, g1 = (a.astype(np.float32).astype(np.float64) for a in (st, g1))
    eng, o = MpmEngine(sc.sim, [[]], [sc.n_particles]), Oracle(sc.sim, [])
    s0, s1, gg1, gg0 = (eng.new_state() for _ in range(4))
    s0[:, :sc.n_particles] = torch.as_tensor(st.T, dtype=eng.dtype, device=eng.device)
    gg1[:, :sc.n_particles] = torch.as_tensor(g1.T, dtype=eng.dtype, device=eng.device)
    pose, zero = torch.zeros((4, 1, 8), dtype=torch.float64, device=eng.device), np.zeros((1, 8))
    eng.substep(s0, s1, pose[0], pose[1])
    eng.substep_bwd(s0, gg1, gg0, pose[0], pose[1], pose[2], pose[3], st1=s1)
    torch.cuda.synchronize()
    for got, ref in ((s1, o.substep(zero, zero, st)), (gg0, o.substep_bwd(zero, zero, st, g1, zero.copy(), zero.copy()))):
        aos = got[:, :sc.n_particles].double().cpu().numpy().T
        for k, sl in GROUPS.items():
            assert rel_err(aos[:, sl], ref[:, sl]) < tol, k
