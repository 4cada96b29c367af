"""``MPMSimulator`` with the reference's API (plb/engine/mpm_simulator.py),
running on the GB300 kernels.

Frame semantics are the reference's: ``substep(s)`` reads frame ``s`` and
writes frame ``s+1`` of ``max_steps`` stored frames (fields x, v, C, F of
shape ``(max_steps, N)``, mpm_simulator.py:38-43); ``substep_grad(s)``
accumulates the adjoint of frame ``s`` from that of frame ``s+1``, as the
taichi ``.grad`` fields do.  For horizons longer than ``max_steps`` use
``diffskill_gb300.engine.Horizon`` (checkpointed recompute) instead.
"""
from __future__ import annotations

from typing import List, Optional

import numpy as np
import torch

from .config import PREC_FP64, SimulatorConfig
from .engine import GridStore, MpmEngine
from .primitives import Primitives


class _Scalar:
    """Stand-in for a taichi 0-d field: ``n_particles[None]``."""

    def __init__(self, v=0):
        self.v = v

    def __getitem__(self, k):
        return self.v

    def __setitem__(self, k, v):
        self.v = int(v)


class _GridMassKernel:
    """``compute_grid_m_kernel(f)`` and its ``.grad(f)`` (mpm_simulator.py:456-466)."""

    def __init__(self, sim: "MPMSimulator"):
        self.sim = sim

    def __call__(self, f: int) -> None:
        sim = self.sim
        sim._eng.grid_mass(sim._frames[f], sim.grid_m_t)

    def grad(self, f: int) -> None:
        sim = self.sim
        sim._eng.grid_mass_bwd(sim._frames[f], sim.grid_m_grad_t, sim._gframes[f])


class MPMSimulator:
    def __init__(self, cfg: SimulatorConfig, primitives: Primitives = None, device=None):
        self.cfg = cfg
        self.dim = 3
        self.primitives = primitives if primitives is not None else Primitives([])
        self.primitives.sim = self
        for p in self.primitives:
            p.sim = self
        self.n_primitive = len(self.primitives)
        self.n_grid = cfg.grid
        self.dx, self.inv_dx = cfg.dx, cfg.inv_dx
        self.dt = cfg.step_dt
        self.p_vol, self.p_rho = cfg.p_vol, 1
        self.p_mass = cfg.p_mass
        self.substeps = cfg.n_substeps
        self.max_steps = int(cfg.max_steps)
        self.lower_bound = cfg.lower_bound
        self.n_particles = _Scalar(0)
        self.dtype = "float64" if cfg.precision_code == PREC_FP64 else "float32"
        self.device = torch.device(device) if device is not None else torch.device("cuda", torch.cuda.current_device())
        self._eng: Optional[MpmEngine] = None
        self.compute_grid_m_kernel = _GridMassKernel(self)
        self.cur = 0
        self._fk_bwd_done = set()

    # ------------------------------------------------------------ lifetime
    def initialize(self, n_particles: int) -> None:
        """``initialize`` (mpm_simulator.py:82-97): allocate for ``n_particles``."""
        n = int(n_particles)
        self.n_particles[None] = n
        self._eng = MpmEngine(self.cfg, [self.primitives.cfgs], [n], softness=self.primitives.get_softness(),
                              device=self.device)
        eng = self._eng
        T = max(eng.T, 1)
        M = self.max_steps
        self._frames = torch.zeros((M, 24, eng.ld), dtype=eng.dtype, device=eng.device)
        self._gframes = torch.zeros_like(self._frames)
        self._pose = torch.zeros((M + 1, T, 8), dtype=torch.float64, device=eng.device)
        self._pose[0, :eng.T] = eng.pose0
        self._vel = torch.zeros((M, T, 8), dtype=torch.float64, device=eng.device)
        self._g_pose = torch.zeros_like(self._pose)
        n_act = M // self.substeps + 1
        self._act = torch.zeros((n_act, T, 8), dtype=torch.float64, device=eng.device)
        self._g_act = torch.zeros_like(self._act)
        self._coll = eng.new_coll(n_act)  # tool-tool collision records per action
        self.grid_m_t = torch.zeros((1, eng.G), dtype=eng.dtype, device=eng.device)
        self.grid_m_grad_t = torch.zeros_like(self.grid_m_t)
        # which entries of a tool's pose are its state, and where the flat action's
        # entries sit in an action's [T, 8] row (one copy to the device for both)
        dims = self.primitives.action_dims
        state = [0] * (8 * T)
        for i, p in enumerate(self.primitives):
            state[8 * i:8 * i + p.state_dim] = [1] * p.state_dim
        index = [8 * i + k for i in range(eng.T) for k in range(dims[i + 1] - dims[i])]
        both = torch.tensor(state + index, dtype=torch.long).to(eng.device)
        self._state_mask = both[:8 * T].reshape(T, 8) != 0
        self._act_index = both[8 * T:]
        # the grids of each substep, for its adjoint: slot s belongs to substep(s) as it
        # last ran, and is emptied whenever frame s or the poses of frames s, s + 1 change
        block = 2 * 64 * 4 * (8 if eng.dtype == torch.float64 else 4) + 4
        # a particle touches at most 8 of the grid's blocks; 512 and one per 64 particles
        # hold a dough several times over (30,000 particles in a 64^3 grid touch 108,
        # 100,000 in a 128^3 grid 400).  All blocks of a 64^3 grid, 436 MB for 25 FP64
        # substeps, took 0.4 ms to allocate; a substep that does not fit is recomputed
        worst = M * min((eng.n_grid // 4) ** 3, 8 * max(eng.P, 1), 512 + eng.P // 64)
        most = 1 << 28
        if worst * block > most:  # (asking for the free memory takes 18 us)
            most = max(most, min(1 << 30, torch.cuda.mem_get_info(eng.device)[0] // 16))
        try:
            self._store = GridStore(eng, M, min(worst, most // block))
        except torch.cuda.OutOfMemoryError:
            self._store = GridStore(eng, M, 0)  # every adjoint substep recomputes its grids
        self._booked = self._again = 0  # slots from _booked up are empty; substeps run again
        self.cur = 0

    def _t64(self, a) -> torch.Tensor:
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.device)

    def _set_softness(self, softness: float) -> None:
        if self._eng is not None and softness != self._eng.softness:
            # tool tables carry the softness; rebuild them on change
            eng = self._eng
            for i in range(eng.T):
                eng._descs[i].softness = softness
            eng.softness = softness
            from . import _lib
            _lib.check(eng.lib.mpm_set_tools(eng.h, eng._descs, eng.T), eng.h, "mpm_set_tools")
            self._forget_all()

    # ------------------------------------------------------------- tools
    def _set_action(self, s: int, action: np.ndarray, only: Optional[int] = None) -> None:
        eng, n = self._eng, self.substeps
        if (s + 1) * n > self.max_steps - 1:
            raise IndexError(f"action {s} runs past max_steps={self.max_steps}")
        index, dims = self._act_index, self.primitives.action_dims
        action = torch.as_tensor(action, dtype=torch.float64, device=self.device)
        if only is not None:
            part = slice(dims[only], dims[only + 1])
            index, action = index[part], action[part]
        self._act[s].view(-1).index_copy_(0, index, action)
        self._store.forget(s * n, (s + 1) * n)
        if eng.T:
            eng.tools_action(self._act[s], self._vel[s * n], self._pose[s * n],
                             None if self._coll is None else self._coll[s])

    def _tools_action_bwd(self, s: int) -> None:
        if s in self._fk_bwd_done or not self._eng.T:
            return
        n = self.substeps
        self._eng.tools_action_bwd(self._vel[s * n], self._pose[s * n], self._g_pose[s * n], self._g_act[s],
                                   None if self._coll is None else self._coll[s])
        self._fk_bwd_done.add(s)

    def tool_sdf(self, t: int, f: int, points: np.ndarray) -> np.ndarray:
        raise NotImplementedError("per-point tool SDFs are exposed through GradModel(return_dist=True)")

    # ------------------------------------------------------------ substeps
    def substep(self, s: int) -> None:
        """``substep`` (mpm_simulator.py:307-323)."""
        self._substeps(s, 1)

    def _substeps(self, first: int, n: int) -> None:
        """Substeps first .. first + n - 1 in order."""
        if not 0 <= first <= first + n < self.max_steps:
            raise IndexError(f"substeps {first} .. {first + n - 1} run past max_steps={self.max_steps}")
        if first < self._booked:
            # run again: its grids take new space.  Once that is as many substeps as there
            # are, what the later slots hold is given back (30 us; the store has room for
            # several times as many)
            self._again += n
            if self._again >= self.max_steps:
                self._again = 0
                self._store.drop(first)
        self._booked = max(self._booked, first + n)
        self._eng.substeps(self._frames[first], self._pose[first], n, self._store, first)

    def _forget_all(self) -> None:
        self._store.reset()
        self._booked = self._again = 0

    def substep_grad(self, s: int) -> None:
        """``substep_grad`` (mpm_simulator.py:325-345): frame-(s+1) adjoint -> frame s (accumulated)."""
        self._substeps_grad(s, 1)

    def _substeps_grad(self, first: int, n: int) -> None:
        """Adjoints of substeps first + n - 1 .. first, last to first."""
        if not 0 <= first <= first + n < self.max_steps:
            raise IndexError(f"substeps {first} .. {first + n - 1} run past max_steps={self.max_steps}")
        self._eng.substeps_bwd(self._frames[first], self._gframes[first], self._pose[first], self._g_pose[first], n,
                               self._store, first)

    def step(self, is_copy: bool, action=None) -> None:
        """``step`` (mpm_simulator.py:440-451)."""
        start = 0 if is_copy else self.cur
        self.cur = start + self.substeps
        if action is not None:
            self.primitives.set_action(start // self.substeps, self.substeps, action)
        self._substeps(start, self.substeps)
        if is_copy:
            self.copyframe(self.cur, 0)
            self.cur = 0

    def copyframe(self, source: int, target: int) -> None:
        self._frames[target].copy_(self._frames[source])
        self._pose[target].copy_(self._pose[source])
        self._forget_all()

    # ----------------------------------------------------------------- io
    def _rows(self, f: int, r0: int, r1: int) -> np.ndarray:
        n = self.n_particles[None]
        return self._frames[f, r0:r1, :n].double().cpu().numpy().T.copy()

    def get_x(self, f: int) -> np.ndarray:
        return self._rows(f, 0, 3)

    def get_v(self, f: int) -> np.ndarray:
        return self._rows(f, 3, 6)

    def get_torch_x(self, f: int, device) -> torch.Tensor:
        n = self.n_particles[None]
        return self._frames[f, 0:3, :n].t().float().to(device).contiguous()

    def get_state(self, f: int) -> List[np.ndarray]:
        """``get_state`` (380-390): [x, v, F(N,3,3), C(N,3,3), tool states...]."""
        n = self.n_particles[None]
        st = self._frames[f, :, :n].double().cpu().numpy()
        out = [st[0:3].T.copy(), st[3:6].T.copy(), st[15:24].T.reshape(n, 3, 3).copy(),
               st[6:15].T.reshape(n, 3, 3).copy()]
        for p in self.primitives:
            out.append(p.get_state(f))
        return out

    def set_state(self, f: int, state) -> None:
        """``set_state`` (392-396)."""
        n = len(state[0])
        if self._eng is None or n != self.n_particles[None]:
            self.initialize(n)
        # everything is checked before the first write: a state that is refused changes no
        # frame.  The rows are transposed and rounded to the frame's type on the device.
        def rows(a):  # [n, 3], or what broadcasts to it
            t = self._t64(np.asarray(a, dtype=np.float64).T)
            while t.dim() > 2 and t.shape[0] == 1:
                t = t[0]
            return t.expand(3, n)

        frame = self._frames[f, :, :n]
        parts = [(frame[0:3], rows(state[0])), (frame[3:6], rows(state[1])),
                 (frame[15:24], self._t64(state[2]).reshape(n, 9).t()),
                 (frame[6:15], self._t64(state[3]).reshape(n, 9).t())]
        poses = self._pose_rows(dict(enumerate(state[4:4 + self.n_primitive])))
        for part, a in parts:
            part.copy_(a)
        self._write_poses(f, *poses)

    def set_primitive_state(self, f: int, state) -> None:
        self._set_poses(f, dict(enumerate(state[4:4 + self.n_primitive])))

    def _set_poses(self, f: int, states: dict) -> None:
        """Leading pose entries of the tools ``states`` at frame ``f``."""
        self._write_poses(f, *self._pose_rows(states))

    def _pose_rows(self, states: dict):
        """The tools' poses with the entries of ``states``, and which entries these are."""
        new = np.full((max(self.n_primitive, 1), 8), np.nan)
        given = np.zeros(new.shape, dtype=bool)
        for i, s in states.items():
            s = np.asarray(s, dtype=np.float64).reshape(-1)
            new[i, :len(s)] = s
            given[i, :len(s)] = True
        return new, given

    def _write_poses(self, f: int, new: np.ndarray, given: np.ndarray) -> None:
        if given.all():
            self._pose[f].copy_(torch.from_numpy(new))
        else:
            both = self._t64(np.stack([new, given]))
            self._pose[f].copy_(torch.where(both[1] != 0, both[0], self._pose[f]))
        # (counted from the end, f is another frame and another row of poses: forget all)
        self._forget_all() if f <= 0 else self._store.forget(f - 1, f)

    def reset(self, x) -> None:
        """``reset`` (402-413): x given, v = 0, F = I, C = 0 at frame 0."""
        x = np.asarray(x, dtype=np.float64)
        if self._eng is None or x.shape[0] != self.n_particles[None]:
            self.initialize(x.shape[0])
        self._frames[0].copy_(self._eng.init_state([x]))
        self._forget_all()
        self.cur = 0

    def get_m(self) -> np.ndarray:
        return self.grid_m_t[0].double().cpu().numpy().reshape(self.n_grid, self.n_grid, self.n_grid)

    def clear_and_compute_grid_m(self, f: int) -> None:
        self.compute_grid_m_kernel(f)

    # ------------------------------------------------------------- grads
    def zero_grad(self) -> None:
        """The ``.grad.fill(0)`` calls of GradModel.reset (function.py:45-61)."""
        self._gframes.zero_()
        self._g_pose.zero_()
        self._g_act.zero_()
        self._fk_bwd_done.clear()

    def check_status(self) -> None:
        self._eng.check_status()
