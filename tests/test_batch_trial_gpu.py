"""The autotuner's trials (zgl_batch_autotune): a request renders as many
samples as it takes for the flat schedule to take the route of the whole
render (csrc/staged.h: staged_pays_in_batch), and two otherwise."""
from __future__ import annotations

import numpy as np
import pytest

from zillumgl_gb300.scene import BatchRenderer, PathIntegrator, Scene
from zillumgl_gb300.synthetic import cornell_scene

pytestmark = pytest.mark.gpu


def test_trials_take_the_renders_route(zgl_lib, cuda):
    import torch

    # width, height, samples, samples of a trial: 98,304 paths run staged
    table = [(64, 64, 40, 24), (64, 64, 20, 2), (256, 256, 5, 2), (31, 33, 1, 1)]
    scenes = [Scene(cornell_scene(seed=50 + k, width=w, height=h)) for k, (w, h, _, _) in enumerate(table)]
    frames = [torch.zeros((h, w, 4), device=cuda) for w, h, _, _ in table]
    batch = BatchRenderer([(s, n, dict(max_depth=3), f) for s, (_, _, n, _), f in zip(scenes, table, frames)])
    batch.autotune()
    torch.cuda.synchronize()
    for s, (_, _, _, trial), f in zip(scenes, table, frames):
        it = PathIntegrator(s, max_depth=3)
        it.render_passes(trial)
        assert np.array_equal(f.cpu().numpy().view(np.uint32), it.get_frame()[0].view(np.uint32))
        it.close()
    batch.render()
    torch.cuda.synchronize()
    for s, (_, _, n, _), f in zip(scenes, table, frames):
        it = PathIntegrator(s, max_depth=3)
        it.render_passes(n)
        assert np.array_equal(f.cpu().numpy().view(np.uint32), it.get_frame()[0].view(np.uint32))
        it.close()
    batch.close()
