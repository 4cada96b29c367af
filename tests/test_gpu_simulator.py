"""``MPMSimulator`` keeps the grids of its forward substeps for their adjoints: whatever
changes a frame, a pose, an action or the softness in between, ``substep_grad`` is that of
the frames and poses as they are."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import all_tools, small_scene
from diffskill_gb300.engine import MpmEngine
from diffskill_gb300.function import SimEnv

pytestmark = pytest.mark.gpu

SUB, ACTIONS = 3, 3
F = SUB * ACTIONS


def _env(prec="fp64", n=400):
    sc = small_scene(n=n, substeps=SUB, n_actions=ACTIONS, tools=[all_tools()[0], all_tools()[4]], precision=prec)
    sc.sim.max_steps = F + 2
    env = SimEnv(sc.sim, sc.tools, np.asarray(sc.x0))
    acts = np.random.default_rng(7).uniform(-1, 1, (ACTIONS, env.primitives.action_dim))
    return sc, env, acts


def _forward(sim, acts):
    for k in range(ACTIONS):
        sim.primitives.set_action(k, SUB, acts[k])
        sim._substeps(k * SUB, SUB)


def _check(sc, sim, substeps):
    """``substep_grad`` of each substep against the recomputing adjoint of another handle."""
    eng = MpmEngine(sc.sim, [sc.tools], [sim.n_particles[None]], softness=sim._eng.softness)
    gen = torch.Generator(device="cuda").manual_seed(2)
    for s in substeps:
        g1 = torch.randn(tuple(sim._gframes[s].shape), generator=gen, device="cuda", dtype=torch.float64)
        sim.zero_grad()
        sim._gframes[s + 1].copy_(g1)
        sim.substep_grad(s)
        g0, gp = eng.new_state(), torch.zeros_like(sim._g_pose[:2])
        eng.substep_bwd(sim._frames[s], g1.to(eng.dtype), g0, sim._pose[s], sim._pose[s + 1], gp[0], gp[1],
                        st1=sim._frames[s + 1])
        torch.cuda.synchronize()
        for got, want in ((sim._gframes[s], g0), (sim._g_pose[s], gp[0]), (sim._g_pose[s + 1], gp[1])):
            assert float((got - want).norm()) <= 1e-10 * float(want.norm()), s


def _state(sim, f, shift):
    """A state list like frame f's, the dough and the tools moved a little."""
    st = [np.array(a, dtype=np.float64) for a in sim.get_state(f)]
    st[0] = st[0] + shift
    for i in range(4, len(st)):
        st[i][:3] += 2 * shift
    return st


# frames counted from the end are frames, and rows of poses, of their own
MUTATE_FROM_THE_END = {
    "set_state": lambda sim: sim.set_state(-6, _state(sim, -6, 0.004)),
    "set_primitive_state": lambda sim: sim.set_primitive_state(-7, _state(sim, -7, 0.004)),
    "a tool's position": lambda sim: sim.primitives[0].set_state(-5, sim._pose[-5, 0, :3].cpu().numpy() + 0.003),
}
MUTATE = {
    "set_state at 0": lambda sim, acts: sim.set_state(0, _state(sim, 0, 0.004)),
    "set_state at 4": lambda sim, acts: sim.set_state(4, _state(sim, 4, 0.004)),
    "tools of set_primitive_state at 5": lambda sim, acts: sim.set_primitive_state(5, _state(sim, 5, 0.004)),
    "a tool's whole state": lambda sim, acts: sim.primitives[1].set_state(3, sim._pose[3, 1].cpu().numpy() + 0.003),
    "a tool's position": lambda sim, acts: sim.primitives[0].set_state(7, sim._pose[7, 0, :3].cpu().numpy() + 0.003),
    "an action": lambda sim, acts: sim.primitives.set_action(1, SUB, -acts[1]),
    "an action of one tool": lambda sim, acts: sim.primitives.set_action(2, SUB, -acts[2], only=1),
    "copyframe": lambda sim, acts: sim.copyframe(7, 2),
    "softness": lambda sim, acts: sim.primitives.set_softness(50.0),
    "reset": lambda sim, acts: sim.reset(sim.get_x(0) + 0.004),
    "a substep again": lambda sim, acts: (sim.set_state(4, _state(sim, 4, 0.004)), sim.substep(4)),
}


@pytest.mark.parametrize("what", MUTATE)
def test_gradients_after_a_change_without_a_new_forward(gpu_lib, what):
    """FP64, the sums' order differs (1e-16 a sum)."""
    sc, env, acts = _env()
    sim = env.simulator
    _forward(sim, acts)
    _check(sc, sim, (0, F - 1))
    assert sim._store.stored_slots() == F
    MUTATE[what](sim, acts)
    _check(sc, sim, range(F))


@pytest.mark.parametrize("what", MUTATE_FROM_THE_END)
def test_gradients_after_a_change_counted_from_the_end(gpu_lib, what):
    sc, env, acts = _env()
    _forward(env.simulator, acts)
    MUTATE_FROM_THE_END[what](env.simulator)
    _check(sc, env.simulator, range(F))


def test_running_from_a_later_frame_again_keeps_the_store(gpu_lib):
    """A loop that plans again from a later frame gives the space of earlier runs back: the
    store, whose size is bounded, does not fill up, and the gradients are right."""
    sc, env, acts = _env()
    sim = env.simulator
    _forward(sim, acts)
    torch.cuda.synchronize()
    used = int(sim._store.bump)
    for i in range(12):
        for k in range(1, ACTIONS):
            sim.primitives.set_action(k, SUB, acts[k] * (0.9 - 0.1 * i))
            sim._substeps(k * SUB, SUB)
        for s in range(F - 2, F):  # and substep by substep
            sim.substep(s)
        torch.cuda.synchronize()
        assert sim._store.stored_slots() >= F - SUB
        # the frames once, as many substeps again as there are before space is given back,
        # and a loop's; another action touches a few blocks more
        assert int(sim._store.bump) <= 1.3 * used * (F + sim.max_steps + 2 * SUB + 2) / F
    _check(sc, sim, range(F))


# shapes of a state's parts that would only fit after a reshape or a broadcast, another
# number of particles, a tool's state that is too long
REFUSED = {
    "x [n, 1, 3]": (0, lambda a: a[:, None, :]),
    "v [3, n]": (1, lambda a: a.T),
    "v flat": (1, lambda a: a.reshape(-1)),
    "F [n, 1]": (2, lambda a: a[:, 0, :1]),
    "C [n, 1]": (3, lambda a: a[:, 0, :1]),
    "F of fewer particles": (2, lambda a: a[1:]),
    "a tool of nine entries": (4, lambda a: np.zeros(9)),
}


@pytest.mark.parametrize("what", REFUSED)
def test_a_state_of_the_wrong_shape_is_refused_and_changes_nothing(gpu_lib, what):
    sc, env, acts = _env()
    sim = env.simulator
    _forward(sim, acts)
    frames, pose = sim._frames.clone(), sim._pose.clone()
    part, change = REFUSED[what]
    st = _state(sim, 4, 0.004)
    st[part] = change(st[part])
    with pytest.raises((RuntimeError, ValueError)):
        sim.set_state(4, st)
    assert torch.equal(sim._frames, frames) and torch.equal(sim._pose, pose)
    _check(sc, sim, range(F))
