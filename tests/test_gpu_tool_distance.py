"""Adjoint of the per-particle tool distances of a batch against those of its scenes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import all_tools, perturbed_state, rel_err, small_scene
from diffskill_gb300.engine import MpmEngine

pytestmark = pytest.mark.gpu


def _adjoint(eng, aos, g_dist):
    n = aos.shape[0]
    st, g_out = eng.new_state(), eng.tool_distance(eng.new_state(), eng.pose0).zero_()
    st[:, :n] = torch.as_tensor(aos.T, device=eng.device)
    g_out[:, :n] = torch.as_tensor(g_dist, device=eng.device)
    gs, gp = eng.new_state(), torch.zeros((eng.T, 8), dtype=torch.float64, device=eng.device)
    eng.tool_distance_bwd(st, eng.pose0, g_out, gs, gp)
    return gs[:, :n].cpu().numpy(), gp.cpu().numpy()


# scenes that end inside a warp, fill it exactly, are smaller than it, and are empty
@pytest.mark.parametrize("sizes", [(5, 40, 33), (32, 64, 1), (700, 3, 131), (31, 0, 65)])
def test_adjoint_of_a_batch_is_that_of_its_scenes(gpu_lib, sizes):
    """FP64; the tools' sums differ in their order only (1e-16 each, 1e3 particles)."""
    tools = all_tools()
    sc, T = small_scene(n=max(sizes), tools=tools, precision="fp64"), len(all_tools())
    states = [perturbed_state(sc.x0[:n], seed=i) for i, n in enumerate(sizes)]
    eng = MpmEngine(sc.sim, [tools] * len(sizes), list(sizes))
    cols = eng.n_dist_cols // len(sizes)  # columns of one scene's tools
    gd = np.random.default_rng(3).normal(size=(eng.n_dist_cols, sum(sizes)))
    gs, gp = _adjoint(eng, np.concatenate(states), gd)
    first = 0
    for i, n in enumerate(sizes):
        part = slice(first, first + n)
        first += n
        if n == 0:
            assert not gp[i * T:(i + 1) * T].any()
            continue
        rs, rp = _adjoint(MpmEngine(sc.sim, [tools], [n]), states[i], gd[i * cols:(i + 1) * cols, part])
        assert np.abs(rs[:3]).max() > 0 and np.abs(rp).max() > 0
        assert rel_err(gs[:3, part], rs[:3]) < 1e-11 and rel_err(gp[i * T:(i + 1) * T], rp) < 1e-11
        assert not gs[3:, part].any()
