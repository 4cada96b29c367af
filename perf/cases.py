"""Workloads of the differentiable MPM framework that its speed is measured on.

Each kind is something a user's program has the framework do, through its
public entry points:

* ``action``   one ``GradModel`` rollout: reset, some actions forward, the
  observation gradients back to the actions (the drop-in autograd boundary);
* ``iterate``  one iteration of a batched trajectory optimisation: forward,
  density loss, adjoint, Adam, replayed as the CUDA graph it was captured in;
* ``rollout``  the forward and the loss of such a batch alone;
* ``forward`` / ``backward``  one substep of a batch of scenes, and its adjoint;
* ``loss``     the shaping loss of one frame and its gradient, optionally with a
  new target density (whose signed distance field is propagated first);
* ``render``   one camera image of the particles and the tools.

Scene sizes and tool sets are those of ``diffskill_gb300.scenes``; inputs come
from the seed, made on the GPU where they are large.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from diffskill_gb300.config import ActionConfig, PrimitiveConfig, SimulatorConfig
from diffskill_gb300.engine import MpmEngine
from diffskill_gb300.function import GradModel, SimEnv
from diffskill_gb300.loss import Loss, LossConfig
from diffskill_gb300.render import ParticleSDFRenderer, RenderConfig
from diffskill_gb300.scenes import Scene
from diffskill_gb300.trajectory import BatchedTrajectory


def listed():
    return [
        # a control loop that differentiates through a small dough in FP64, the reference method: launches and latency
        {"name": "action-fp64-2k", "kind": "action", "n": 2000, "grid": 64, "prec": "fp64", "tools": "capsule",
         "substeps": 19, "actions": 1, "dist": False},
        # the default simulator (30k particles, 19 substeps an action) with the tool distances in the observation
        {"name": "action-fp32-30k", "kind": "action", "n": 30000, "grid": 64, "prec": "fp32", "tools": "box+capsule",
         "substeps": 19, "actions": 2, "dist": True},
        # cutting and gripping on the fine grid, with the SVD in FP64
        {"name": "action-svd64-100k", "kind": "action", "n": 100000, "grid": 128, "prec": "fp32_svd64",
         "tools": "knife+gripper", "substeps": 39, "actions": 1, "dist": False},
        # trajectory optimisation of many scenes at once, every frame kept: the flagship
        {"name": "iterate-fp32-64x", "kind": "iterate", "scenes": 64, "n_min": 5000, "n_max": 40000, "grid": 64,
         "prec": "fp32", "substeps": 50, "actions": 2, "ckpt": 1},
        # the plain FP64 single-scene optimisation with checkpoints
        {"name": "iterate-fp64-10k", "kind": "iterate", "scenes": 1, "n_min": 10000, "n_max": 10000, "grid": 64,
         "prec": "fp64", "substeps": 50, "actions": 2, "ckpt": 10},
        # large scenes on the fine grid, checkpointed, the SVD in FP64
        {"name": "iterate-svd64-4x", "kind": "iterate", "scenes": 4, "n_min": 100000, "n_max": 300000, "grid": 128,
         "prec": "fp32_svd64", "substeps": 20, "actions": 1, "ckpt": 10},
        # scoring action sequences without a gradient (sampling planners, evaluation)
        {"name": "rollout-fp32-64x", "kind": "rollout", "scenes": 64, "n_min": 5000, "n_max": 40000, "grid": 64,
         "prec": "fp32", "substeps": 50, "actions": 2, "ckpt": 1},
        # the substep by itself, for a program with a loop of its own; ragged sizes
        {"name": "forward-fp32-48x", "kind": "forward", "scenes": 48, "n_min": 4999, "n_max": 40001, "grid": 64,
         "prec": "fp32"},
        {"name": "backward-fp32-48x", "kind": "backward", "scenes": 48, "n_min": 4999, "n_max": 40001, "grid": 64,
         "prec": "fp32"},
        {"name": "backward-fp64-37k", "kind": "backward", "scenes": 1, "n_min": 37001, "n_max": 37001, "grid": 64,
         "prec": "fp64"},
        # an environment step's reward with its gradient, for a goal that was just set
        {"name": "loss-30k", "kind": "loss", "n": 30000, "grid": 64, "prec": "fp32", "soft": True, "retarget": True},
        # an image observation
        {"name": "render-30k", "kind": "render", "n": 30000, "grid": 64, "image": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["action", "action", "iterate", "rollout", "forward", "backward", "loss", "render"])
    prec = rng.choice(["fp32", "fp32", "fp32_svd64", "fp64"])
    grid = rng.choice([64, 64, 128])
    if kind == "action":
        n = _log_int(rng, 1000, 100000 if prec == "fp32" else 40000)
        return {"kind": kind, "n": n, "grid": grid, "prec": prec,
                "tools": rng.choice(["capsule", "box+capsule", "knife+gripper"]),
                "substeps": rng.choice([10, 19, 25]), "actions": rng.choice([1, 2]), "dist": rng.random() < 0.3}
    if kind in ("iterate", "rollout"):
        scenes = _log_int(rng, 1, 48)
        n_min = _log_int(rng, 2000, 12000)
        n_max = _log_int(rng, n_min, 40000)
        if prec != "fp32":  # the FP64 arithmetic makes a particle some ten times as dear
            scenes, n_max = min(scenes, 6), min(n_max, 30000)
        ckpt = rng.choice([1, 5, 10])
        return {"kind": kind, "scenes": scenes, "n_min": n_min, "n_max": n_max, "grid": grid if scenes <= 8 else 64,
                "prec": prec, "substeps": rng.choice([20, 30, 50]), "actions": rng.choice([1, 2]), "ckpt": ckpt}
    if kind in ("forward", "backward"):
        scenes = _log_int(rng, 1, 64)
        n_min = _log_int(rng, 1001, 20001)
        n_max = _log_int(rng, n_min, 60001)
        return {"kind": kind, "scenes": scenes, "n_min": n_min, "n_max": n_max, "grid": grid if scenes <= 8 else 64,
                "prec": prec}
    if kind == "loss":
        return {"kind": kind, "n": _log_int(rng, 2000, 200000), "grid": grid, "prec": rng.choice(["fp32", "fp64"]),
                "soft": rng.random() < 0.5, "retarget": grid == 64 and rng.random() < 0.5}
    return {"kind": kind, "n": _log_int(rng, 2000, 100000), "grid": grid, "image": rng.choice([256, 512, 1024])}


# ------------------------------------------------------------------ inputs
def _sim(case, n, max_steps=1024):
    substeps = case.get("substeps", 50)
    return SimulatorConfig(E=5e3, nu=0.2, yield_stress=50.0, gravity=(0.0, -9.8, 0.0), n_grid=case["grid"],
                           dt=1e-4 * 64 / case["grid"], substeps=substeps, precision=case.get("prec", "fp32"),
                           n_particles=n, max_steps=max_steps)


def _sizes(case):
    """Particles of each scene: spread over [n_min, n_max] on a log scale."""
    S, lo, hi = case["scenes"], case["n_min"], case["n_max"]
    return [int(round(lo * (hi / lo) ** ((k + 0.5) / S))) for k in range(S)]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(gen, shape, lo, hi):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _slab(gen, n, lo=0.0):
    """A box of dough on the ground; returns the points and the height of its top."""
    w = torch.tensor([0.25, 0.08, 0.25], dtype=torch.float64, device="cuda")
    c = torch.tensor([0.5, 0.09, 0.5], dtype=torch.float64, device="cuda")
    return (torch.rand((n, 3), generator=gen, device="cuda", dtype=torch.float64) - 0.5) * w + c, 0.13


def _balls(gen, n, k):
    """k balls of dough on the ground; returns the points and (centre, radius) of each ball."""
    r = _uniform(gen, (k,), 0.04, 0.08)
    c = torch.stack([_uniform(gen, (k,), 0.3, 0.6), 0.05 + r, _uniform(gen, (k,), 0.3, 0.7)], 1)
    of = torch.multinomial((r ** 3).float(), n, replacement=True, generator=gen)
    d = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    d = d / d.norm(dim=1, keepdim=True)
    u = torch.rand((n, 1), generator=gen, device="cuda", dtype=torch.float64) ** (1 / 3)
    x = c[of] + d * u * r[of].unsqueeze(1)
    return x, list(zip(c.tolist(), r.tolist()))


def _inside(x, sim):
    return x.clamp(sim.lower_bound * sim.dx + 1e-6, 1.0 - 3 * sim.dx)


MOVE = ActionConfig(dim=3, scale=(0.005, 0.005, 0.005))


def _capsule(pos, h=0.2):
    return PrimitiveConfig(shape="Capsule", init_pos=tuple(pos), init_rot=(0.707, 0.707, 0.0, 0.0), r=0.03, h=h,
                           action=MOVE)


def _tool_set(name):
    """Tools that rest on the slab of ``_slab``."""
    if name == "capsule":
        return [_capsule((0.5, 0.157, 0.5))]
    if name == "box+capsule":
        return [PrimitiveConfig(shape="Box", init_pos=(0.5, 0.1295, 0.5), size=(0.075, 0.0025, 0.075), action=MOVE),
                _capsule((0.42, 0.157, 0.5), h=0.25)]
    knife = PrimitiveConfig(shape="Knife", init_pos=(0.5, 0.2, 0.5), size=(0.125, 0.075, 0.002), prism_h=(0.15, 0.15),
                            prot=(1.0, 0.0, 0.0, 0.0), friction=0.0, action=MOVE)
    gripper = PrimitiveConfig(shape="Gripper", init_pos=(0.5, 0.12, 0.6), size=(0.01, 0.04, 0.04), init_gap=0.25,
                              minimal_gap=0.04, maximal_gap=0.3, friction=5.0,
                              action=ActionConfig(dim=7, scale=(0.005, 0.005, 0.005, 0.0, 0.0, 0.0, 0.005)))
    return [knife, gripper]


def _ball_tools(k, balls, box):
    """1 to 3 tools (spheres, capsules and, with ``box``, plates), each pressed 5 mm into a ball of dough."""
    tools = []
    for j in range(1 + k % 3):
        (cx, cy, cz), r = balls[j % len(balls)]
        top, off, turn = cy + r, 0.3 * r * (j - 0.5), (k + j) % (3 if box else 2)
        if turn == 0:
            tools.append(PrimitiveConfig(shape="Sphere", init_pos=(cx + off, top + 0.035, cz), radius=0.04,
                                         action=MOVE))
        elif turn == 1:
            tools.append(_capsule((cx, top + 0.025, cz + off), h=0.22))
        else:
            tools.append(PrimitiveConfig(shape="Box", init_pos=(cx, top - 0.0025, cz), size=(0.05, 0.0025, 0.05),
                                         action=MOVE))
    return tools


def _density(x, n, mass):
    """Quadratic B-spline density grid of the points, for a goal (flat [n^3], on the GPU)."""
    out = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    base = (x * n - 0.5).long().clamp(0, n - 3)
    f = x * n - base
    w = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2]
    for i in range(3):
        for j in range(3):
            for k in range(3):
                at = ((base[:, 0] + i) * n + base[:, 1] + j) * n + base[:, 2] + k
                out.index_add_(0, at, w[i][:, 0] * w[j][:, 1] * w[k][:, 2] * mass)
    return out


def _host(t):
    return t.cpu().numpy()


# -------------------------------------------------- single scene, GradModel
def _prepare_action(case, seed):
    gen, n = _generator(seed), case["n"]
    sim = _sim(case, n, max_steps=case["actions"] * case["substeps"] + 1)
    x = _inside(_slab(gen, n)[0], sim)
    env = SimEnv(sim, _tool_set(case["tools"]), _host(x))
    model = GradModel(env, return_dist=case["dist"])
    dims = env.primitives.action_dim
    acts = _uniform(gen, (case["actions"], dims), -1, 1).float()
    cols = 6 + (env.simulator._eng.n_dist_cols if case["dist"] else 0)
    g_x = torch.randn((n, cols), generator=gen, device="cuda") / n
    g_t = torch.randn((len(env.primitives), 8), generator=gen, device="cuda") * 1e-2
    return {"case": case, "model": model, "acts": acts, "g_x": g_x, "g_t": g_t}


def _run_action(s):
    model = s["model"]
    acts = s["acts"].clone().requires_grad_(True)
    obs = model.reset()
    for k in range(s["case"]["actions"]):
        obs = model.forward(k, acts[k], *obs)
    loss = (obs[0] * s["g_x"]).sum() + (obs[1] * s["g_t"]).sum()
    (grad,) = torch.autograd.grad(loss, acts)
    return {"particles": obs[0].detach(), "tools": obs[1].detach(), "grad": grad}


# ------------------------------------------------------- batched trajectory
def _prepare_batch(case, seed):
    gen = _generator(seed)
    scenes = []
    for k, n in enumerate(_sizes(case)):
        sim = _sim(case, n)
        x, balls = _balls(gen, n, 1 + k % 4)
        x = _inside(x, sim)
        goal = _density(_inside(x + torch.tensor([0.1, 0.0, 0.0], dtype=torch.float64, device="cuda"), sim),
                        sim.grid, sim.p_mass)
        tools = _ball_tools(k, balls, box=True)
        acts = _host(_uniform(gen, (case["actions"], 3 * len(tools)), -1, 1))
        scenes.append(Scene(sim, tools, _host(x), _host(goal), acts))
    traj = BatchedTrajectory(scenes, ckpt_every=case["ckpt"])
    start = traj.actions.clone()
    if case["kind"] == "iterate":
        traj.capture()
        return {"case": case, "traj": traj, "start": start}
    return {"case": case, "traj": traj, "graph": traj.capture_forward()}


def _run_iterate(s):
    traj = s["traj"]
    traj.reset_optimizer()
    traj.actions.copy_(s["start"])
    traj.step()
    return {"loss": traj.loss, "grad": traj.grad, "actions": traj.actions, "g_state0": traj.hz.g_state0}


def _run_rollout(s):
    s["graph"].replay()
    return {"loss": s["traj"].loss, "density": s["traj"].hz.gm}


# ------------------------------------------------------------- one substep
def _flow(x, gen, S_of):
    """Velocity, its gradient and a deformation as in dough that is being pressed and settles."""
    n = x.shape[0]
    k = 2 * math.pi * torch.tensor([3.0, 5.0, 4.0], dtype=torch.float64, device="cuda")
    amp = torch.tensor([0.25, 0.35, 0.2], dtype=torch.float64, device="cuda")
    ph = x[:, [1, 2, 0]] * k
    v = amp * torch.sin(ph)
    v[:, 1] -= 0.2
    v = v + 0.02 * torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64)
    C = 0.5 * torch.randn((n, 3, 3), generator=gen, device="cuda", dtype=torch.float64)
    dv = amp * k * torch.cos(ph)
    for i, j in enumerate((1, 2, 0)):
        C[:, i, j] += dv[:, i]
    # strains from well below to somewhat above the yield strain (about 0.012)
    size = 0.002 * (1 + 4 * (S_of % 3).double())
    F = torch.eye(3, dtype=torch.float64, device="cuda") + size[:, None, None] * torch.randn(
        (n, 3, 3), generator=gen, device="cuda", dtype=torch.float64)
    return v, C, F


def _prepare_substep(case, seed):
    gen, sizes = _generator(seed), _sizes(case)
    sims = [_sim(case, n) for n in sizes]
    xs, tools = [], []
    for k, n in enumerate(sizes):
        x, balls = _balls(gen, n, 1 + k % 4)
        xs.append(_inside(x, sims[k]))
        tools.append(_ball_tools(k, balls, box=False))
    eng = MpmEngine(sims[0], tools, sizes)
    P = eng.P
    of = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), torch.tensor(sizes, device="cuda"))
    x = torch.cat(xs)
    v, C, F = _flow(x, gen, of)
    st = eng.new_state()
    st[:, :P] = torch.cat([x, v, C.reshape(P, 9), F.reshape(P, 9)], 1).t().to(eng.dtype)
    # sorted by cell some substeps ago, as a trajectory's frames are
    st0 = eng.new_state()
    eng.sort_frame(st, st0, torch.empty(P, dtype=torch.int32, device="cuda"))
    st0[0:3, :P] += 12 * sims[0].step_dt * st0[3:6, :P]
    st0[0:3, :P].clamp_(sims[0].lower_bound * sims[0].dx + 1e-6, 1.0 - 3 * sims[0].dx)
    pose0 = eng.pose0.clone()
    pose1 = pose0.clone()
    pose1[:, :3] += 1e-4 * torch.randn((eng.T, 3), generator=gen, device="cuda", dtype=torch.float64)
    s = {"case": case, "eng": eng, "sim": sims[0], "tools": tools, "of": of, "st0": st0, "st1": eng.new_state(),
         "pose0": pose0, "pose1": pose1}
    if case["kind"] == "backward":
        eng.substep(st0, s["st1"], pose0, pose1)
        scale = torch.tensor([1.0] * 3 + [1e-2] * 3 + [1e-4] * 9 + [1e-2] * 9, dtype=torch.float64, device="cuda")
        g1 = eng.new_state()
        g1[:, :P] = (torch.randn((24, P), generator=gen, device="cuda", dtype=torch.float64)
                     * scale[:, None]).to(eng.dtype)
        s.update(g1=g1, g0=eng.new_state(), gp0=torch.zeros_like(pose0), gp1=torch.zeros_like(pose1))
    return s


def _run_forward(s):
    s["eng"].substep(s["st0"], s["st1"], s["pose0"], s["pose1"])
    return {"state": s["st1"]}


def _run_backward(s):
    s["gp0"].zero_()
    s["gp1"].zero_()
    s["eng"].substep_bwd(s["st0"], s["g1"], s["g0"], s["pose0"], s["pose1"], s["gp0"], s["gp1"], st1=s["st1"])
    return {"g_state": s["g0"], "g_pose0": s["gp0"], "g_pose1": s["gp1"]}


# ---------------------------------------------------------------- the loss
def _prepare_loss(case, seed):
    gen, n = _generator(seed), case["n"]
    sim = _sim(case, n, max_steps=2)
    x = _inside(_slab(gen, n)[0], sim)
    env = SimEnv(sim, _tool_set("box+capsule"), _host(x))
    loss = Loss(LossConfig(soft_contact=case["soft"]), env.simulator)
    goal = _inside(_balls(gen, n, 2)[0], sim)
    grids = _host(_density(goal, sim.grid, sim.p_mass)).reshape((sim.grid,) * 3)
    loss.load_target_density(grids=grids)
    loss.reset()
    return {"case": case, "env": env, "loss": loss, "grids": grids}


def _run_loss(s):
    loss, sim = s["loss"], s["env"].simulator
    if s["case"]["retarget"]:
        loss.load_target_density(grids=s["grids"])
    sim.zero_grad()
    loss.clear()
    info = loss.compute_loss(0)
    loss.compute_loss_kernel.grad(0)
    return {"density_loss": info["density_loss"], "sdf_loss": info["sdf_loss"], "contact": info["contact_loss"],
            "loss": info["loss"], "iou": info["iou"], "target_sdf": loss.target_sdf, "density": sim.grid_m_t,
            "g_state": sim._gframes[0]}


# --------------------------------------------------------------- the image
def _prepare_render(case, seed):
    gen, n = _generator(seed), case["n"]
    sim = _sim(case, n)
    x, balls = _balls(gen, n, 2)
    x = _inside(x, sim)
    eng = MpmEngine(sim, [_ball_tools(2, balls, box=True)], [n])
    st = eng.new_state()
    st[0:3, :n] = x.t().to(eng.dtype)
    colors = torch.randint(0, 1 << 24, (n,), generator=gen, device="cuda", dtype=torch.int32)
    return {"case": case, "eng": eng, "st": st, "colors": colors,
            "r": ParticleSDFRenderer(eng, 0, RenderConfig(tina_img_res=case["image"]))}


def _run_render(s):
    s["r"].set_particles(s["st"], s["colors"])
    return s["r"].trace()


PREPARE = {"action": _prepare_action, "iterate": _prepare_batch, "rollout": _prepare_batch,
           "forward": _prepare_substep, "backward": _prepare_substep, "loss": _prepare_loss, "render": _prepare_render}
RUN = {"action": _run_action, "iterate": _run_iterate, "rollout": _run_rollout, "forward": _run_forward,
       "backward": _run_backward, "loss": _run_loss, "render": _run_render}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def run(state):
    return RUN[state["case"]["kind"]](state)


def work(case):
    """A substep reads and writes the 24 values of every particle; its adjoint reads them and the 24 gradients and
    writes 24.  Arithmetic per particle: two 27-node stencils, an SVD and 3x3 products, each about 1,500 operations
    forward and 2,500 in the adjoint."""
    w = 8 if case.get("prec") == "fp64" else 4
    kind, n3 = case["kind"], case["grid"] ** 3
    fwd_b, bwd_b, fwd_f, bwd_f = 48 * w, 72 * w, 1500, 2500
    if kind == "action":
        p = case["n"] * case["substeps"] * case["actions"]
        return {"bytes": p * (fwd_b + bwd_b), "flops": p * (fwd_f + bwd_f)}
    if kind in ("iterate", "rollout", "forward", "backward"):
        P = sum(_sizes(case))
        p = P * case.get("substeps", 1) * case.get("actions", 1)
        dense = 0 if kind in ("forward", "backward") else 2 * w * n3 * case["scenes"]
        f = kind in ("iterate", "rollout", "forward")
        b = kind in ("iterate", "backward")
        return {"bytes": p * (f * fwd_b + b * bwd_b) + dense, "flops": p * (f * fwd_f + b * bwd_f)}
    if kind == "loss":
        # positions in, their gradients out, the density, target and distance grids once each; a new goal's nearest
        # points are four more grids, found over 6^3 neighbours at least once
        more = 4 * w * n3 if case["retarget"] else 0
        return {"bytes": 6 * w * case["n"] + 4 * w * n3 + more,
                "flops": 27 * 16 * case["n"] + 8 * n3 + (215 * 8 * n3 if case["retarget"] else 0)}
    # the splat of 14^3 voxels a particle, the decoded volume, one ray a pixel
    return {"bytes": 16 * case["n"] + 16 * 168 ** 3 + 40 * case["image"] ** 2,
            "flops": 14 ** 3 * 8 * case["n"] + 2 * 27 * 168 ** 3 + 500 * case["image"] ** 2}


# ------------------------------------------------- one substep in 64 bits
class _Svd(torch.autograd.Function):
    """A = U diag(s) V^T of 3x3 matrices with the reference's clamped gradient (plb/engine/mpm_simulator.py:137-156)."""

    @staticmethod
    def forward(ctx, A):
        U, s, Vh = torch.linalg.svd(A)
        V = Vh.transpose(-1, -2)
        # proper rotations; the sign goes to the smallest singular value
        du, dv = torch.linalg.det(U), torch.linalg.det(V)
        U = torch.cat([U[..., :2], U[..., 2:] * du.sign()[..., None, None]], -1)
        V = torch.cat([V[..., :2], V[..., 2:] * dv.sign()[..., None, None]], -1)
        s = torch.cat([s[..., :2], s[..., 2:] * (du * dv).sign()[..., None]], -1)
        ctx.save_for_backward(U, s, V)
        return U, s, V

    @staticmethod
    def backward(ctx, gU, gs, gV):
        U, s, V = ctx.saved_tensors
        ss = s * s
        d = ss[..., None, :] - ss[..., :, None]
        d = torch.where(d >= 0, d.clamp(min=1e-6), d.clamp(max=-1e-6))
        off = 1 - torch.eye(3, dtype=s.dtype, device=s.device)
        a, b = U.transpose(-1, -2) @ gU, V.transpose(-1, -2) @ gV
        X = (a - a.transpose(-1, -2)) / d * off * s[..., None, :] + s[..., :, None] * (
            (b - b.transpose(-1, -2)) / d * off) + torch.diag_embed(gs)
        return U @ X @ V.transpose(-1, -2)


def _qrot(q, v):
    qv = q[1:].expand_as(v)
    uv = torch.linalg.cross(qv, v)
    return v + 2 * (q[0] * uv + torch.linalg.cross(qv, uv))


def _into(p, pos, rot):
    sign = torch.tensor([1.0, -1.0, -1.0, -1.0], dtype=torch.float64, device="cuda")
    return _qrot(rot * sign / rot.norm(), p - pos)


def _length(a, eps):
    return ((a * a).sum(-1) + eps).sqrt()


def _contact(tool, P0, P1, p, dt, v, softness=666.0):
    """Primitive.collide of a sphere or capsule (plb/engine/primitive/primive_base.py:96-120) at grid points p."""
    pos, rot = P0[:3], P0[3:7]
    if tool.shape == "Sphere":
        u = p - pos
        dist = _length(u, 1e-14) - tool.radius
        D = u / _length(u, 1e-14)[:, None]
    else:
        q = _into(p, pos, rot)
        a = q[:, 1] + tool.h / 2
        u = torch.stack([q[:, 0], a - a.clamp(0, tool.h), q[:, 2]], 1)
        dist = _length(u, 1e-14) - tool.r
        D = _qrot(rot, u / _length(u, 1e-14)[:, None])
    infl = torch.exp(-dist * softness).clamp(max=1.0)
    cv = (_qrot(P1[3:7], _into(p, pos, rot)) + P1[:3] - p) / dt
    iv = v - cv
    nc = (iv * D).sum(-1, keepdim=True)
    vt = iv - nc.clamp(max=0.0) * D
    vn = _length(vt, 1e-8)[:, None]
    slip = vt / vn * (vn + nc * tool.friction).clamp(min=0.0)
    vt = torch.where((nc < 0) & ((vt * vt).sum(-1, keepdim=True) > 1e-60), slip, vt)
    out = cv + iv * (1 - infl[:, None]) + vt * infl[:, None]
    return torch.where(((infl > 0.1) | (dist <= 0))[:, None], out, v)


def _substep64(s, st, pose0, pose1):
    """One substep (plb/engine/mpm_simulator.py:307-323) in 64 bits: [24, P] -> [24, P]."""
    sim, of = s["sim"], s["of"]
    n, dx, dt = sim.grid, sim.dx, sim.step_dt
    mu, lam = sim.mu, sim.lam
    P, S = st.shape[1], len(s["tools"])
    x, v = st[0:3].t(), st[3:6].t()
    C, F = st[6:15].t().reshape(P, 3, 3), st[15:24].t().reshape(P, 3, 3)
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    A = (eye + dt * C) @ F
    U, sig, V = _Svd.apply(A)
    eps = sig.clamp(min=0.05).log()
    dev = eps - eps.mean(1, keepdim=True)
    nrm = ((dev * dev).sum(1, keepdim=True) + 1e-8).sqrt()
    dg = nrm - sim.yield_stress / (2 * mu)
    e = torch.exp(eps - dg / nrm * dev)
    newF = torch.where((dg > 0)[:, :, None], U @ torch.diag_embed(e) @ V.transpose(1, 2), A)
    J = torch.linalg.det(newF)[:, None, None]
    stress = 2 * mu * (newF - U @ V.transpose(1, 2)) @ newF.transpose(1, 2) + eye * lam * J * (J - 1)
    aff = -dt * sim.p_vol * 4 * n * n * stress + sim.p_mass * C
    base = (x.detach() * n - 0.5).long()
    f = x * n - base
    w = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2]
    grid = torch.zeros((S * n ** 3, 4), dtype=torch.float64, device="cuda")
    offs = [(i, j, k) for i in range(3) for j in range(3) for k in range(3)]

    def at(o):
        return ((of * n + base[:, 0] + o[0]) * n + base[:, 1] + o[1]) * n + base[:, 2] + o[2]

    def weight(o):
        return (w[o[0]][:, 0] * w[o[1]][:, 1] * w[o[2]][:, 2])[:, None]

    for o in offs:
        dp = (torch.tensor(o, dtype=torch.float64, device="cuda") - f) * dx
        mv = sim.p_mass * v + (aff @ dp[:, :, None])[:, :, 0]
        grid = grid.index_add(0, at(o), weight(o) * torch.cat([mv, torch.full_like(mv[:, :1], sim.p_mass)], 1))
    live = (grid[:, 3] > 1e-12).nonzero()[:, 0]
    g = grid[live]
    drop = dt * 30 * torch.tensor(list(sim.gravity), dtype=torch.float64, device="cuda")
    gv = g[:, :3] / g[:, 3:] + drop
    node = live % n ** 3
    I = torch.stack([node // (n * n), node // n % n, node % n], 1)
    parts, t = [], 0
    ends = torch.searchsorted(live, torch.arange(S + 1, device="cuda") * n ** 3).tolist()
    for k in range(S):
        u, p = gv[ends[k]:ends[k + 1]], I[ends[k]:ends[k + 1]] * dx
        for tool in s["tools"][k]:
            u = _contact(tool, pose0[t], pose1[t], p, dt, u)
            t += 1
        parts.append(u)
    gv = torch.cat(parts)
    for d in range(3):
        low = ((I[:, d] < 3) & (gv[:, d] < 0))[:, None]
        if d == 1:  # ground friction
            side = gv * torch.tensor([1.0, 0.0, 1.0], dtype=torch.float64, device="cuda")
            held = side * (1 + sim.ground_friction * gv[:, 1] / _length(side, 1e-8)).clamp(min=0.0)[:, None]
        else:
            held = gv * (1 - eye[d])
        gv = torch.where(low, held, gv)
        gv = torch.where(((I[:, d] > n - 3) & (gv[:, d] > 0))[:, None], gv * (1 - eye[d]), gv)
    out = torch.zeros((S * n ** 3, 3), dtype=torch.float64, device="cuda").index_copy(0, live, gv)
    nv, nC = 0, 0
    for o in offs:
        q = weight(o) * out[at(o)]
        nv = nv + q
        nC = nC + 4 * n * q[:, :, None] * (torch.tensor(o, dtype=torch.float64, device="cuda") - f)[:, None, :]
    nx = (x + dt * nv).clamp(sim.lower_bound * dx, 1 - 3 * dx)
    return torch.cat([nx, nv, nC.reshape(P, 9), newF.reshape(P, 9)], 1).t()


def exact(case, seed):
    if case["kind"] not in ("forward", "backward"):
        return None
    s = prepare(case, seed)
    P, ld = s["eng"].P, s["eng"].ld

    def padded(a, like):
        out = like.double()
        out[:, :P] = a
        return out

    st = s["st0"][:, :P].double()
    if case["kind"] == "forward":
        with torch.no_grad():
            return {"state": padded(_substep64(s, st, s["pose0"], s["pose1"]), torch.zeros((24, ld), device="cuda"))}
    st, p0, p1 = st.requires_grad_(True), s["pose0"].clone().requires_grad_(True), s["pose1"].clone().requires_grad_(True)
    out = _substep64(s, st, p0, p1)
    g = torch.autograd.grad(out, (st, p0, p1), s["g1"][:, :P].double())
    return {"g_state": padded(g[0], torch.zeros((24, ld), device="cuda")), "g_pose0": g[1], "g_pose1": g[2]}
