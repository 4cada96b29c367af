"""Runs of substeps over several scenes and in FP32 with the FP64 SVD: the particle order
holds the scenes apart."""
from __future__ import annotations

import pytest
import torch

from _util import all_tools, small_scene
from diffskill_gb300.engine import MpmEngine

pytestmark = pytest.mark.gpu

K = 5


# enough particles for the order by cell, scenes that end inside a warp and an empty one;
# tolerances as between a run and single substeps of one scene
@pytest.mark.parametrize("prec,sizes,tol", [("fp64", (5003, 0, 8001), 1e-10), ("fp32", (12007, 31, 8009), 2e-3),
                                            ("fp32_svd64", (20011,), 2e-3), ("fp32_svd64", (9001, 11013), 2e-3)])
def test_run_of_several_scenes_equals_single_substeps(gpu_lib, prec, sizes, tol):
    tools = [all_tools()[0], all_tools()[1]]
    sc = small_scene(n=max(sizes), substeps=K, tools=tools, precision=prec)
    eng = MpmEngine(sc.sim, [tools] * len(sizes), list(sizes))
    one = MpmEngine(sc.sim, [tools] * len(sizes), list(sizes))
    frames = torch.zeros((K + 1, 24, eng.ld), dtype=eng.dtype, device=eng.device)
    frames[0].copy_(eng.init_state([sc.x0[:n] for n in sizes]))
    pose = eng.pose0.expand(K + 1, -1, -1).clone()
    pose[:, :, 1] -= 1e-3 * torch.arange(K + 1, device=eng.device, dtype=torch.float64)[:, None]
    gen = torch.Generator(device="cuda").manual_seed(3)
    g_last = torch.randn((24, eng.ld), generator=gen, device="cuda", dtype=torch.float64).to(eng.dtype)
    ref = frames.clone()
    for i in range(K):
        one.substep(ref[i], ref[i + 1], pose[i], pose[i + 1])
    g, g_ref = torch.zeros_like(frames), torch.zeros_like(frames)
    gp, gp_ref = torch.zeros_like(pose), torch.zeros_like(pose)
    g[K], g_ref[K] = g_last, g_last
    for i in range(K - 1, -1, -1):
        one.substep_bwd(ref[i], g_ref[i + 1], g_ref[i], pose[i], pose[i + 1], gp_ref[i], gp_ref[i + 1], st1=ref[i + 1])
    eng.substeps(frames, pose, K)
    eng.substeps_bwd(ref, g, pose, gp, K)
    torch.cuda.synchronize()
    eng.check_status()
    P = sum(sizes)
    for a, b, t in ((frames[K], ref[K], 1e-12 if prec == "fp64" else 1e-5), (g[0], g_ref[0], tol)):
        assert float((a - b)[:, :P].double().norm()) <= t * float(b[:, :P].double().norm())
    assert float((gp - gp_ref).norm()) <= tol * float(gp_ref.norm())
