"""Render calls beside one another: a trace reads its volume and writes its outputs alone."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from _util import small_scene
from diffskill_gb300.engine import MpmEngine
from diffskill_gb300.render import ParticleSDFRenderer, RenderConfig

pytestmark = pytest.mark.gpu

KEYS = ("depth", "normal", "color", "image")


def _two_renderers():
    """Two volumes of one handle that share the bake's scratch, with different dough."""
    sc = small_scene(n=2000, precision="fp32")
    eng = MpmEngine(sc.sim, [[]], [sc.n_particles])
    cfg = RenderConfig(voxel_res=(70, 64, 66), bake_size=4, tina_img_res=128)
    a, b = (ParticleSDFRenderer(eng, cfg=cfg) for _ in range(2))
    b.packed = a.packed
    b.vol.packed = a.packed.data_ptr()
    x = np.asarray(sc.x0)
    return a, b, eng.init_state([x]), eng.init_state([x * [1.0, 0.5, 1.0] + [0.02, 0.0, 0.05]])


def test_trace_leaves_the_volume_alone(gpu_lib):
    """Every buffer of the volume, its bake's scratch among them, is as it was."""
    a, _, st, _ = _two_renderers()
    a.set_particles(st)
    names = ("packed", "sdf", "sdf_copy", "color", "bbox", "kbox")
    before = {k: getattr(a, k).clone() for k in names}
    a.trace()
    torch.cuda.synchronize()
    for k in names:
        assert torch.equal(getattr(a, k), before[k]), k


def test_traces_of_two_volumes_on_two_streams(gpu_lib):
    """Volumes that share the bake's scratch, traced at the same time on streams of their
    own, and one baked again while the other is traced: the images of each alone."""
    a, b, sa, sb = _two_renderers()
    a.set_particles(sa)
    b.set_particles(sb)
    ref = [{k: v.clone() for k, v in r.trace().items()} for r in (a, b)]
    torch.cuda.synchronize()
    assert not torch.equal(ref[0]["depth"], ref[1]["depth"])
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = [[], []]
    for _ in range(8):
        for i, r in enumerate((a, b)):
            with torch.cuda.stream(streams[i]):
                if i == 0:
                    r.set_particles(sa)
                outs[i].append(r.trace())
    torch.cuda.synchronize()
    for i in range(2):
        for o in outs[i]:
            for k in KEYS:
                assert torch.equal(o[k], ref[i][k]), k


def test_traces_beside_the_stream_that_traced_first(gpu_lib):
    """The handle's own scratch belongs to the stream of its first trace: traces on another
    stream at the same time, and on a third after it, have theirs."""
    a, b, sa, sb = _two_renderers()
    first, second, third = (torch.cuda.Stream() for _ in range(3))
    a.set_particles(sa)
    b.set_particles(sb)
    torch.cuda.synchronize()
    outs = {id(a): [], id(b): []}
    for _ in range(8):
        for r, stream in ((a, first), (b, second), (b, first), (a, third)):
            with torch.cuda.stream(stream):
                outs[id(r)].append(r.trace())
    torch.cuda.synchronize()
    for r in (a, b):
        ref = r.trace()
        torch.cuda.synchronize()
        for o in outs[id(r)]:
            for k in KEYS:
                assert torch.equal(o[k], ref[k]), k
    assert not torch.equal(outs[id(a)][0]["depth"], outs[id(b)][0]["depth"])


def test_captured_trace(gpu_lib):
    """The first trace of a handle, recorded in a graph and replayed twice."""
    a, _, st, _ = _two_renderers()
    a.set_particles(st)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = a.trace()
    for _ in range(2):
        for k in KEYS:
            out[k].fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        got = {k: out[k].clone() for k in KEYS}
        ref = a.trace()
        torch.cuda.synchronize()
        for k in KEYS:
            assert torch.equal(got[k], ref[k]), k
