"""Calls whose handle keeps something from one call to the next, recorded in CUDA graphs
that run late, twice or never."""
from __future__ import annotations

import pytest
import torch

from _util import all_tools, small_scene
from diffskill_gb300.engine import MpmEngine

pytestmark = pytest.mark.gpu

K = 6


class _Run:
    """A scene of n particles with the frames, poses and a frame gradient of K substeps."""

    def __init__(self, prec, n):
        sc = small_scene(n=n, substeps=K, tools=[all_tools()[0], all_tools()[1]], precision=prec)
        self.sc, self.n, self.eng = sc, n, self.engine(sc, n)
        eng = self.eng
        self.frames = torch.zeros((K + 1, 24, eng.ld), dtype=eng.dtype, device=eng.device)
        self.pose = torch.zeros((K + 1, eng.T, 8), dtype=torch.float64, device=eng.device)
        vel = torch.zeros((K, eng.T, 8), dtype=torch.float64, device=eng.device)
        self.frames[0].copy_(eng.init_state([sc.x0]))
        self.pose[0].copy_(eng.pose0)
        eng.tools_action(eng.expand_actions([sc.actions])[0], vel, self.pose)
        gen = torch.Generator(device="cuda").manual_seed(1)
        self.g = torch.randn((24, eng.ld), generator=gen, device="cuda", dtype=torch.float64).to(eng.dtype)

    @staticmethod
    def engine(sc, n):
        return MpmEngine(sc.sim, [sc.tools], [n])

    def adjoint(self, eng, g, gp):
        """The K adjoint substeps on the frames, one call; their gradients."""
        g.zero_()
        gp.zero_()
        g[K].copy_(self.g)
        eng.substeps_bwd(self.frames, g, self.pose, gp, K)

    def buffers(self):
        return torch.zeros_like(self.frames), torch.zeros_like(self.pose)

    def single(self):
        """Frames and gradients by single substeps of a handle of its own."""
        eng, frames = self.engine(self.sc, self.n), self.frames.clone()
        for i in range(K):
            eng.substep(frames[i], frames[i + 1], self.pose[i], self.pose[i + 1])
        g, gp = self.buffers()
        g[K] = self.g
        for i in range(K - 1, -1, -1):
            eng.substep_bwd(frames[i], g[i + 1], g[i], self.pose[i], self.pose[i + 1], gp[i], gp[i + 1],
                            st1=frames[i + 1])
        return frames, g, gp


def _same(a, b, tol):
    assert float((a - b).double().norm()) <= tol * float(b.double().norm())


# enough particles for the order by cell; tolerances as between a run and single substeps
@pytest.mark.parametrize("prec,n,tol", [("fp64", 13001, 1e-10), ("fp32", 20011, 2e-3)])
def test_adjoint_after_a_forward_capture_that_never_ran(gpu_lib, prec, n, tol):
    """A forward run that was only recorded has sorted nothing: the adjoint run after it
    takes no order that it did not get, on a handle that has never run anything."""
    r = _Run(prec, n)
    frames, g_ref, gp_ref = r.single()
    fresh, scratch = r.engine(r.sc, n), r.frames.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        fresh.substeps(scratch, r.pose, K)
    del graph
    r.frames.copy_(frames)
    g, gp = r.buffers()
    r.adjoint(fresh, g, gp)
    torch.cuda.synchronize()
    fresh.check_status()
    _same(g[0, :, :n], g_ref[0, :, :n], tol)
    _same(gp, gp_ref, tol)


@pytest.mark.parametrize("prec,n,tol", [("fp64", 1001, 1e-10), ("fp64", 13001, 1e-10), ("fp32", 20011, 2e-3)])
def test_captured_runs_equal_single_substeps(gpu_lib, prec, n, tol):
    """Forward and adjoint run in one graph, and an adjoint run in a graph of its own,
    each replayed twice, on a handle that has run nothing before."""
    r = _Run(prec, n)
    frames, g_ref, gp_ref = r.single()
    eng = r.engine(r.sc, n)
    g, gp = r.buffers()
    for forward in (True, False):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            if forward:
                eng.substeps(r.frames, r.pose, K)
            r.adjoint(eng, g, gp)
        for _ in range(2):
            g.fill_(7.0)
            graph.replay()
            torch.cuda.synchronize()
            eng.check_status()
            _same(r.frames, frames, 1e-12 if prec == "fp64" else 1e-5)
            _same(g[0, :, :n], g_ref[0, :, :n], tol)
            _same(gp, gp_ref, tol)
