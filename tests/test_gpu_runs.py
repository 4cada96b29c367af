"""Runs of substeps (mpm_substeps_fwd / mpm_substeps_bwd) against single substeps."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import all_tools, small_scene
from diffskill_gb300.engine import GridStore, MpmEngine

pytestmark = pytest.mark.gpu


# fewer particles than a warp, a ragged last warp, and more than both thresholds of
# the sorted order (12,000 in FP64, 20,000 in FP32)
@pytest.mark.parametrize("prec,n,tol", [("fp64", 7, 1e-10), ("fp64", 1001, 1e-10), ("fp64", 13001, 1e-10),
                                        ("fp32", 1001, 2e-3), ("fp32", 20011, 2e-3)])
@pytest.mark.parametrize("stored", [False, True])
def test_run_equals_single_substeps(gpu_lib, prec, n, tol, stored):
    """Six substeps and their adjoints, with and without a grid store, give the
    frames and gradients of single substeps, added to what the gradient frames
    held.  FP64 differs by its summation order (1e-16 per sum, six substeps); FP32
    gradients by 1e-7 per sum and what clamped singular values and contact make of
    it over six adjoint substeps."""
    k = 6
    sc = small_scene(n=n, substeps=k, tools=[all_tools()[0], all_tools()[1]], precision=prec)
    eng = MpmEngine(sc.sim, [sc.tools], [n])
    frames = torch.zeros((k + 1, 24, eng.ld), dtype=eng.dtype, device=eng.device)
    pose = torch.zeros((k + 1, eng.T, 8), dtype=torch.float64, device=eng.device)
    vel = torch.zeros((k, eng.T, 8), dtype=torch.float64, device=eng.device)
    frames[0].copy_(eng.init_state([sc.x0]))
    pose[0].copy_(eng.pose0)
    eng.tools_action(eng.expand_actions([sc.actions])[0], vel, pose)
    ref = frames.clone()
    for i in range(k):
        eng.substep(ref[i], ref[i + 1], pose[i], pose[i + 1])
    store = GridStore(eng, k, 4096 * k) if stored else None
    eng.substeps(frames, pose, k, store, 0)
    torch.cuda.synchronize()
    fwd_tol = 1e-12 if prec == "fp64" else 1e-5
    assert float((frames - ref).abs().max()) <= fwd_tol * float(ref.abs().max())
    if stored:
        assert store.stored_slots() == k

    gen = torch.Generator(device="cuda").manual_seed(1)
    seed = torch.randn((24, eng.ld), generator=gen, device="cuda", dtype=torch.float64).to(eng.dtype)
    held = torch.randn((24, eng.ld), generator=gen, device="cuda", dtype=torch.float64).to(eng.dtype)
    g_ref, gp_ref = torch.zeros_like(frames), torch.zeros_like(pose)
    g_ref[k], g_ref[2] = seed, held
    tmp = eng.new_state()
    for i in range(k - 1, -1, -1):
        eng.substep_bwd(frames[i], g_ref[i + 1], tmp, pose[i], pose[i + 1], gp_ref[i], gp_ref[i + 1],
                        st1=frames[i + 1])
        g_ref[i, :, :n] += tmp[:, :n]
    g, gp = torch.zeros_like(frames), torch.zeros_like(pose)
    g[k], g[2] = seed, held
    eng.substeps_bwd(frames, g, pose, gp, k, store, 0)
    torch.cuda.synchronize()
    eng.check_status()
    for got, want in ((g[0, :, :n], g_ref[0, :, :n]), (g[2, :, :n], g_ref[2, :, :n]), (gp, gp_ref)):
        assert float((got - want).double().norm()) <= tol * float(want.double().norm())


def test_run_empties_the_slot_after_it(gpu_lib):
    """A run rewrites the frame after its last substep, so that frame's own slot is
    emptied and its adjoint recomputes the grids."""
    sc = small_scene(n=500, substeps=4, precision="fp64")
    eng = MpmEngine(sc.sim, [sc.tools], [500])
    frames = torch.zeros((5, 24, eng.ld), dtype=eng.dtype, device=eng.device)
    pose = eng.pose0.expand(5, -1, -1).contiguous()
    frames[0].copy_(eng.init_state([sc.x0]))
    store = GridStore(eng, 4, 4096 * 8)
    eng.substeps(frames, pose, 4, store, 0)
    eng.substeps(frames, pose, 2, store, 0)
    torch.cuda.synchronize()
    assert (store.slot_start >= 0).tolist() == [True, True, False, True]


# the list is built from 16 flags per thread: 8 and 3 x 8 flags end inside a thread's
# share, 216 and 5 x 216 inside a warp's
@pytest.mark.parametrize("n_grid,scenes", [(8, 1), (8, 3), (24, 1), (24, 5), (64, 2)])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_substeps_leave_a_clean_grid(gpu_lib, n_grid, scenes, prec):
    """Substeps of particle sets that touch different blocks, with an adjoint in
    between, on one handle give what each gives on a handle of its own: nothing
    of an earlier substep's grid or block list is left.  The sums differ in their
    order only (1e-16 in FP64, 1e-7 in FP32, of at most a few hundred terms; the
    gradients by what clamped singular values make of that)."""
    n = 300
    sc = small_scene(n=n, tools=[all_tools()[0]], precision=prec)
    sc.sim.n_grid = n_grid
    rng = np.random.default_rng(5)

    def engine():
        return MpmEngine(sc.sim, [sc.tools] * scenes, [n] * scenes)

    sets = [[rng.uniform(lo, hi, (n, 3)) for _ in range(scenes)]
            for lo, hi in ((0.4, 0.5), (0.42, 0.75), (0.5, 0.6), (0.4, 0.5))]
    eng = engine()
    for i, x in enumerate(sets):
        one = engine()
        outs = []
        for e in (eng, one):
            st = e.init_state(x)
            st1 = e.new_state()
            e.substep(st, st1, e.pose0, e.pose0)
            if i % 2:
                g = torch.ones_like(st)
                g_in, gp = e.new_state(), torch.zeros((2,) + tuple(e.pose0.shape), dtype=torch.float64, device=e.device)
                e.substep_bwd(st, g, g_in, e.pose0, e.pose0, gp[0], gp[1], st1=st1)
                outs.append(torch.cat([st1, g_in]))
            else:
                outs.append(st1)
        torch.cuda.synchronize()
        eng.check_status()
        tol = 1e-11 if prec == "fp64" else 2e-3
        assert float((outs[0] - outs[1]).double().norm()) <= tol * float(outs[1].double().norm())
