"""Sizes at which the kernels' splits end unevenly, and deformation gradients that take
the decompositions' fallbacks, against the oracle or the same call scene by scene."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import GROUPS, all_tools, perturbed_state, rel_err, small_scene
from diffskill_gb300.engine import MpmEngine
from diffskill_gb300.render import ParticleSDFRenderer, RenderConfig
from oracle import oracle as O
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _batch(sizes, prec="fp64"):
    """A scene batch and one engine per scene, with the same particles."""
    tools = all_tools()
    sc = small_scene(n=max(sizes), tools=tools, precision=prec)
    states = [perturbed_state(sc.x0[:n], seed=i) for i, n in enumerate(sizes)]
    eng = MpmEngine(sc.sim, [tools] * len(sizes), list(sizes))
    return sc, tools, states, eng


def _soa(eng, aos):
    st = eng.new_state()
    st[:, :aos.shape[0]] = torch.as_tensor(aos.T, dtype=eng.dtype, device=eng.device)
    return st


# scenes that end inside a warp, fill it exactly, and are smaller than it
@pytest.mark.parametrize("sizes", [(5, 40, 33), (32, 64, 1), (700, 3, 131)])
def test_tool_terms_where_warps_hold_several_scenes(gpu_lib, sizes):
    """Soft contact, per-particle tool distances and their adjoints of a batch are those
    of its scenes alone; FP64, the sums differ in their order only."""
    sc, tools, states, eng = _batch(sizes)
    T, rng = len(tools), np.random.default_rng(3)
    g_md = rng.normal(size=T * len(sizes))

    def terms(e, aos, gm, gd):
        st, pose = _soa(e, aos), e.pose0
        md, sums = e.soft_contact(st, pose)
        gs, gp = e.new_state(), torch.zeros((e.T, 8), dtype=torch.float64, device=e.device)
        e.soft_contact_bwd(st, pose, sums, torch.as_tensor(gm, device=e.device), gs, gp)
        d = e.tool_distance(st, pose)
        gs2, gp2 = e.new_state(), torch.zeros_like(gp)
        g_out = torch.zeros_like(d)
        g_out[:, :aos.shape[0]] = torch.as_tensor(gd, dtype=e.dtype, device=e.device)
        e.tool_distance_bwd(st, pose, g_out, gs2, gp2)
        n = aos.shape[0]
        return [t.cpu().numpy() for t in (md, gs[:3, :n], gp, d[:, :n], gs2[:3, :n], gp2)]

    gd = rng.normal(size=(eng.n_dist_cols, sum(sizes)))
    cols = eng.n_dist_cols  # one column set per tool of a scene, shared by the batch's columns
    one = MpmEngine(sc.sim, [tools], [sizes[0]]).n_dist_cols
    got = terms(eng, np.concatenate(states), g_md, gd)
    first = 0
    for i, n in enumerate(sizes):
        e = MpmEngine(sc.sim, [tools], [n])
        rows = slice(0, one) if cols == one else slice(i * one, (i + 1) * one)
        ref = terms(e, states[i], g_md[i * T:(i + 1) * T], gd[rows, first:first + n])
        part, tool = slice(first, first + n), slice(i * T, (i + 1) * T)
        for a, b in zip((got[0][tool], got[1][:, part], got[2][tool], got[3][rows, part]), ref[:4]):
            assert rel_err(a, b) < 1e-11
        if cols == one:
            for a, b in zip((got[4][:, part], got[5][tool]), ref[4:]):
                assert rel_err(a, b) < 1e-11
        first += n


# eight scenes take 16 CTAs each, more take 8
@pytest.mark.parametrize("scenes", [1, 8, 9, 17])
def test_grid_reductions_over_many_scenes(gpu_lib, scenes):
    sc = small_scene(n=50, precision="fp64")
    eng = MpmEngine(sc.sim, [[] for _ in range(scenes)], [50] * scenes)
    rng = np.random.default_rng(scenes)
    gm, tgt, sdf = (rng.uniform(0, 1, size=(scenes, eng.G)) for _ in range(3))
    dev = [torch.as_tensor(a, device=eng.device) for a in (gm, tgt, sdf)]
    iou, loss = eng.iou(dev[0], dev[1]), eng.sdf_loss(dev[0], dev[2], 1.5)
    for s in range(scenes):
        ref = O.iou(gm[s], tgt[s])
        assert abs(float(iou[s]) - ref) <= 1e-11 * abs(ref)
        ref = 1.5 * O.sdf_loss(gm[s], sdf[s])[0]
        assert abs(float(loss[s]) - ref) <= 1e-11 * abs(ref)


# a volume whose last extent is not a multiple of 4, images that end inside a 16x8 tile
@pytest.mark.parametrize("res,image", [((61, 66, 63), 33), ((64, 65, 70), 50)])
def test_render_of_ragged_sizes(gpu_lib, res, image):
    cfg = RenderConfig(voxel_res=res, bake_size=6, tina_img_res=image)
    sc = small_scene(n=2000, precision="fp32")
    eng = MpmEngine(sc.sim, [[]], [sc.n_particles])
    st = eng.init_state([sc.x0])
    r = ParticleSDFRenderer(eng, cfg=cfg)
    r.set_particles(st)
    out = r.trace()
    torch.cuda.synchronize()
    assert eng.status() == 0
    x = st[0:3, :sc.n_particles].double().cpu().numpy().T
    sdf, color, bbox, over = O.render_bake(x, res, cfg.bake_size, cfg.dx, None)
    assert over == 0
    assert np.array_equal(r.sdf.cpu().numpy().reshape(res), sdf)
    assert np.array_equal(r.color.cpu().numpy().reshape(res + (3,)), color)
    depth, nrm, col, img = O.render_trace(sdf, color, r.bbox.cpu().numpy(), r.v2w, r.w2v, (image, image),
                                          cfg.sdf_threshold)
    assert np.array_equal(out["depth"].cpu().numpy(), depth)
    assert np.array_equal(out["image"].cpu().numpy(), img)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-9), ("fp32_svd64", 1e-4)])
def test_forward_of_extreme_deformations(gpu_lib, prec, tol):
    """Equal singular values, one of them zero or tiny, inverted elements, strains up
    to 3 and the identity: each leaves the refined decompositions' range at another
    test.  The clamp at 0.05 keeps newF and the stress smooth in F.  (Not for the FP32
    decomposition of F - I, which has no fallback and loses digits of F where a
    singular value vanishes.)"""
    sc = small_scene(n=256, tools=[], precision=prec)
    rng = np.random.default_rng(8)
    st = perturbed_state(sc.x0, seed=8, C=0.0, F=0.0)
    sing = [(1, 1, 1), (1, 1, 0.9), (1.2, 0.8, 0.8), (1.1, 0.9, 1e-3), (1.1, 0.9, 0.0), (1.1, 0.9, 1e-9),
            (1.2, 1.0, -0.5), (1.3, 1.0, -0.04), (3.0, 1.0, 0.4), (1.0, 0.9, 0.06), (1 + 1e-7, 1, 1 - 1e-7)]
    for p in range(0, sc.n_particles):
        U, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        V, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        U[:, 2] *= np.linalg.det(U)
        V[:, 2] *= np.linalg.det(V)
        st[p, 15:24] = (U @ np.diag(sing[p % len(sing)]) @ V.T).ravel()
    if prec == "fp32_svd64":  # what the device holds
        st = st.astype(np.float32).astype(np.float64)
    eng, o = MpmEngine(sc.sim, [[]], [sc.n_particles]), Oracle(sc.sim, [])
    pose = torch.zeros((1, 8), dtype=torch.float64, device=eng.device)
    s1 = eng.new_state()
    eng.substep(_soa(eng, st), s1, pose, pose)
    torch.cuda.synchronize()
    ref = o.substep(np.zeros((1, 8)), np.zeros((1, 8)), st)
    got = s1[:, :sc.n_particles].double().cpu().numpy().T
    for k, sl in GROUPS.items():
        assert rel_err(got[:, sl], ref[:, sl]) < tol, k


# one cell per warp, as many as g2p.grad stages, one more, and a cell per lane
@pytest.mark.parametrize("cells", [1, 4, 7, 8, 32])
def test_adjoint_by_cells_per_warp(gpu_lib, cells):
    """FP32, at the tolerance of the substep's adjoint test; a ragged last warp."""
    n, sc = 101, small_scene(n=101, tools=[], precision="fp32")
    rng, dx = np.random.default_rng(cells), sc.sim.dx
    cell = np.arange(n) % cells
    corner = np.stack([cell % 4, cell // 4 % 4, cell // 16], -1) * 2 + 24
    x = (corner + 0.5 + rng.uniform(0.05, 0.95, (n, 3))) * dx
    st = perturbed_state(x.astype(np.float32).astype(np.float64), seed=4)
    eng, o = MpmEngine(sc.sim, [[]], [n]), Oracle(sc.sim, [])
    g1 = rng.normal(size=st.shape)
    zero = np.zeros((1, 8))
    ref = o.substep_bwd(zero, zero, st, g1, np.zeros((1, 8)), np.zeros((1, 8)))
    pose = torch.zeros((4, 1, 8), dtype=torch.float64, device=eng.device)
    s0, s1, gg1, gg0 = _soa(eng, st), eng.new_state(), _soa(eng, g1), eng.new_state()
    eng.substep(s0, s1, pose[0], pose[1])
    eng.substep_bwd(s0, gg1, gg0, pose[0], pose[1], pose[2], pose[3], st1=s1)
    torch.cuda.synchronize()
    got = gg0[:, :n].double().cpu().numpy().T
    for k, sl in GROUPS.items():
        assert rel_err(got[:, sl], ref[:, sl]) < 2e-4, k


@pytest.mark.parametrize("sort", [True, False])
def test_g2p_shared_gathers_equal_lane_gathers(gpu_lib, sort):
    """More particles than a wave of CTAs holds (8 x 128 per SM), a ragged last warp and one
    particle outside the grid: the default shape shares its gathers within a cell, 10 CTAs
    per SM gather lane by lane.  Unsorted, most warps hold more cells than fit.  The two
    runs' grids differ in the order of their FP32 sums (1e-7; 1e-6 relative in C)."""
    from diffskill_gb300 import autotune

    n = 8 * 128 * torch.cuda.get_device_properties(0).multi_processor_count + 77
    sc = small_scene(n=64, tools=[], precision="fp32")
    eng = MpmEngine(sc.sim, [[]], [n])
    rng = np.random.default_rng(1)
    st0 = _soa(eng, perturbed_state(rng.uniform(0.3, 0.5, (n, 3)), seed=1))
    st0[0, 5] = 7.0
    if sort:
        by_cell, perm = eng.new_state(), torch.empty(n, dtype=torch.int32, device=eng.device)
        eng.sort_frame(st0, by_cell, perm)
        st0 = by_cell
    pose = torch.zeros((1, 8), dtype=torch.float64, device=eng.device)
    outs = []
    for ctas in (8, 10):
        autotune.apply(eng, autotune.Tuning(g2p_ctas=ctas))
        st1 = eng.new_state()
        eng.substep(st0, st1, pose, pose)
        outs.append(st1[:, :n].double())
    torch.cuda.synchronize()
    for sl in GROUPS.values():
        assert float((outs[0][sl] - outs[1][sl]).abs().max()) <= 1e-5 * float(outs[1][sl].abs().max())
