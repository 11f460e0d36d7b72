"""Calls on one handle from several streams and from CUDA graphs: the staged
renderers share a handle's lists and sums between its calls, which therefore
take turns on the device (csrc/staged.h: StagedTurn)."""
from __future__ import annotations

import numpy as np
import pytest

from zillumgl_gb300.scene import DiffRenderer, LightIntegrator, PathIntegrator, Scene
from zillumgl_gb300.synthetic import cornell_scene, diff_scene

from tests.test_light_gpu import _check

pytestmark = pytest.mark.gpu

PARAMS = dict(max_depth=5, blocks_per_pass=64)  # 98,304 light paths a pass: staged


def _film(it):
    return it.get_frame()[0][..., :3].astype(np.float64)


def test_light_passes_on_two_streams(zgl_lib, cuda):
    import torch

    sc = Scene(cornell_scene(seed=41, width=96, height=80))
    one, two = LightIntegrator(sc, **PARAMS), LightIntegrator(sc, **PARAMS)
    one.render_passes(8)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for k in range(8):
        two.render_one_pass(stream=streams[k % 2])
    torch.cuda.synchronize()
    _check(_film(two), _film(one))
    for x in (one, two, sc):
        x.close()


def test_captured_light_pass_beside_eager_ones(zgl_lib, cuda):
    """A captured pass repeats its sample; the film is a sum, whatever the order."""
    import torch

    sc = Scene(cornell_scene(seed=42, width=96, height=80))
    first, five, it = (LightIntegrator(sc, **PARAMS) for _ in range(3))
    first.render_passes(1)
    five.render_passes(5)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a):
        it.render_one_pass(stream=a)
    for _ in range(4):  # samples 1 to 4, between replays of sample 0
        with torch.cuda.stream(a):
            graph.replay()
        it.render_one_pass(stream=b)
    torch.cuda.synchronize()
    _check(_film(it), _film(five) + 3.0 * _film(first))
    for x in (first, five, it, sc):
        x.close()


def test_gradients_of_two_adjoints_on_two_streams(zgl_lib, cuda):
    import torch

    sc = Scene(diff_scene(seed=43, width=193, height=171))
    r = DiffRenderer(sc, 3, max_depth=6)  # 99,009 paths: staged, replay too
    r.forward()
    gen = torch.Generator(cuda).manual_seed(3)
    adj = [torch.rand((171, 193, 3), device=cuda, generator=gen) - 0.5 for _ in range(2)]
    want = [r.backward(a).double() for a in adj]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[torch.empty(r.n_params, device=cuda) for _ in range(4)] for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(4):
        for s in range(2):
            r.backward(adj[s], out=got[s][k], stream=streams[s])
    torch.cuda.synchronize()
    for s in range(2):
        for g in got[s]:  # float sums of one block's window in atomic order: 1e-5, as between the two replays
            assert float((g.double() - want[s]).abs().max()) <= 1e-5 * float(want[s].abs().max())
    r.close()
    sc.close()


def test_captured_pass_outlives_a_larger_call(zgl_lib, cuda):
    """Several passes at once need larger buffers; a pass captured before that
    still runs on its own."""
    import torch

    sc = Scene(cornell_scene(seed=44, width=401, height=397))  # one pass runs staged
    ten, it = PathIntegrator(sc, max_depth=4), PathIntegrator(sc, max_depth=4)
    ten.render_passes(10)
    it.render_one_pass()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        it.render_one_pass(stream=stream)  # sample 1, in the frame when the graph runs
    it.render_passes(8)
    fill = [torch.full((1 << 24,), 7.0, device=cuda) for _ in range(8)]  # takes what was given back
    graph.replay()
    torch.cuda.synchronize()
    assert all(bool((f == 7.0).all()) for f in fill)
    got, want = it.get_frame()[0][..., :3], ten.get_frame()[0][..., :3]
    # ten positive float32 terms in another order: nine roundings of 2^-24 each way
    assert np.all(np.abs(got - want) <= 18 * 2.0 ** -24 * np.abs(want))
    for x in (ten, it, sc):
        x.close()
