"""The staged path tracer (csrc/staged.cu: ray casts and shading in separate
kernels), which the integrators, the batched renderer and the differentiable
forward pass run for calls of enough paths (staged.h: staged_pays): frames bit
for bit the oracle's, whatever the film size, depth, sampler and materials."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from zillumgl_gb300.scene import BatchRenderer, DiffRenderer, LightIntegrator, PathIntegrator, Scene, TripleIntegrator
from zillumgl_gb300.synthetic import (city_scene, cornell_scene, diff_scene, material_zoo_scene, sky_environment,
                                      sphere_box_scene, textured_scene)

from tests.test_light_gpu import _check

pytestmark = pytest.mark.gpu

W, H = 331, 301  # 99,631 pixels, no multiple of the 8x4 tile


def _env(d, **kw):
    d.env_rgb = sky_environment(64, 32, seed=6)
    return d.normalized()


CASES = {
    "cornell": (lambda: cornell_scene(seed=3, width=W, height=H), dict(max_depth=5), 2),
    "independent": (lambda: cornell_scene(seed=4, width=W, height=H, sampler=0), dict(max_depth=3), 2),
    "roulette": (lambda: cornell_scene(seed=5, width=W, height=H),
                 dict(max_depth=9, russian_roulette=1, rr_start_depth=3), 2),
    "no_light_samples": (lambda: cornell_scene(seed=6, width=W, height=H), dict(max_depth=3, sample_light=0), 1),
    "depth_0": (lambda: cornell_scene(seed=7, width=W, height=H), dict(max_depth=0), 1),
    "depth_24": (lambda: cornell_scene(seed=7, width=W, height=H), dict(max_depth=24), 1),
    "depth_25": (lambda: cornell_scene(seed=7, width=W, height=H), dict(max_depth=25), 1),
    "environment": (lambda: _env(cornell_scene(seed=8, width=W, height=H)),
                    dict(max_depth=4, light_env_uniform_sample=1, light_portion=0.4), 2),
    "zoo": (lambda: material_zoo_scene(seed=9, width=W, height=H), dict(max_depth=6), 6),  # both block sizes
    "textured": (lambda: textured_scene(seed=10, width=W, height=H, base="zoo"), dict(max_depth=4), 1),
    "city": (lambda: city_scene(seed=11, width=W, height=H, grid=12, n_spheres=40, env_size=(64, 32)),
             dict(max_depth=6, russian_roulette=1, rr_start_depth=2), 2),
    "spheres": (lambda: sphere_box_scene(12, 30000, 181, 183), dict(max_depth=6), 2),  # 33k paths, large tree
}


@pytest.mark.parametrize("name", list(CASES))
def test_passes_equal_the_oracle(zgl_lib, cuda, name):
    make, params, n = CASES[name]
    data = make()
    sc = Scene(data)
    w, h = data.film
    orc = oracle.OracleScene(data, sc.export("sobol"), params)
    pix = np.random.default_rng(1).choice(w * h, 1500, replace=False).astype(np.int32)
    ref = orc.render_pt(pix, n)
    one = PathIntegrator(sc, **params)
    for _ in range(n):
        one.render_one_pass()
    several = PathIntegrator(sc, **params)
    several.render_passes(n)
    f1, f2 = one.get_frame()[0], several.get_frame()[0]
    assert np.array_equal(f1.view(np.uint32), f2.view(np.uint32))
    got = f1[..., :3].reshape(-1, 3)[pix]
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    for x in (one, several, sc):
        x.close()


def test_paths_beyond_the_pool(zgl_lib, cuda):
    """More paths than the pool holds, in one call: chunks that end inside a sample."""
    sc = Scene(cornell_scene(seed=13, width=640, height=520))
    a, b = PathIntegrator(sc, max_depth=3), PathIntegrator(sc, max_depth=3)
    a.render_passes(9)  # 3.0M paths
    for _ in range(9):
        b.render_one_pass()
    assert np.array_equal(a.get_frame()[0].view(np.uint32), b.get_frame()[0].view(np.uint32))
    for x in (a, b, sc):
        x.close()


def test_batch_of_staged_and_shared_requests(zgl_lib, cuda):
    import torch

    specs = [(cornell_scene(seed=21, width=W, height=H), 2, dict(max_depth=5)),
             (material_zoo_scene(seed=22, width=40, height=30), 3, dict(max_depth=4)),
             (sphere_box_scene(23, 30000, 200, 170), 1, dict(max_depth=6, russian_roulette=1)),
             (cornell_scene(seed=24, width=64, height=64), 2, dict(max_depth=30))]
    scenes = [Scene(d) for d, _, _ in specs]
    frames = [torch.full((s.film[1], s.film[0], 4), 3.0, device=cuda) for s in scenes]
    batch = BatchRenderer([(s, n, p, f) for s, (_, n, p), f in zip(scenes, specs, frames)])
    for _ in range(2):
        batch.render()
    torch.cuda.synchronize()
    for s, (_, n, p), f in zip(scenes, specs, frames):
        one = PathIntegrator(s, **p)
        for _ in range(n):
            one.render_one_pass()
        assert np.array_equal(f.cpu().numpy().view(np.uint32), one.get_frame()[0].view(np.uint32))
        one.close()
    batch.close()


@pytest.mark.parametrize("make, params", [
    (lambda: diff_scene(seed=14, width=W, height=H), dict(max_depth=1)),
    (lambda: diff_scene(seed=15, width=W, height=H), dict(max_depth=8, russian_roulette=1, rr_start_depth=2)),
    (lambda: diff_scene(seed=14, width=W, height=H), dict(max_depth=11)),  # beyond the kept casts
    (lambda: _env(diff_scene(seed=16, width=W, height=H, sampler=0)), dict(max_depth=4, light_portion=0.3,
                                                                          light_env_uniform_sample=1)),
    (lambda: textured_scene(seed=17, width=W, height=H, base="zoo"), dict(max_depth=6)),
], ids=["depth_1", "depth_8", "depth_11", "environment", "textured_zoo"])
def test_adjoint_of_the_staged_forward(zgl_lib, cuda, make, params):
    """The replay of the kept casts, staged where they hold the whole path: the
    gradient is the one of the one-kernel replay that traces again (float
    atomics: 1e-5 of the largest), and the image the integrator's mean."""
    import torch

    n = 2
    sc = Scene(make())
    r = DiffRenderer(sc, n, **params)
    img = r.forward()
    integ = PathIntegrator(sc, **params)
    integ.render_passes(n)
    mean = integ.get_frame()[0][..., :3] / np.float32(n)
    assert np.array_equal(img.cpu().numpy().view(np.uint32), mean.view(np.uint32))
    d_image = torch.rand((H, W, 3), device=cuda, generator=torch.Generator(cuda).manual_seed(2)) - 0.5
    d_image[: H // 3] = 0.0  # pixels that need no replay
    kept = r.backward(d_image).cpu().numpy().astype(np.float64)
    r.set_params(r.params())  # drops the casts
    traced = r.backward(d_image).cpu().numpy().astype(np.float64)
    assert np.abs(traced).max() > 0
    assert np.abs(kept - traced).max() <= 1e-5 * np.abs(traced).max()
    for x in (r, integ, sc):
        x.close()


@pytest.mark.parametrize("make", [
    lambda: cornell_scene(seed=31, width=96, height=80),
    lambda: textured_scene(seed=32, width=90, height=70, base="zoo"),
    lambda: city_scene(seed=33, width=96, height=54, grid=12, n_spheres=40, env_size=(16, 8)),
], ids=["cornell", "textured_zoo", "city"])
@pytest.mark.parametrize("triple", [False, True])
@pytest.mark.parametrize("params", [dict(max_depth=1), dict(max_depth=6, russian_roulette=1, rr_start_depth=2)],
                         ids=["depth_1", "roulette"])
def test_light_paths_equal_the_oracle(zgl_lib, cuda, make, triple, params):
    """98,304 light paths a pass run staged; film sums within the 1e-4 that
    float atomics are held to."""
    data = make()
    sc = Scene(data)
    params = dict(params, blocks_per_pass=64)
    integ = (TripleIntegrator if triple else LightIntegrator)(sc, **params)
    integ.render_passes(2)
    got = integ.get_frame()[0][..., :3]
    orc = oracle.OracleScene(data, sc.export("sobol"), params)
    ref = orc.render_triple(2, blocks=64) if triple else orc.render_lt(2, blocks=64)
    assert ref.sum() > 0
    _check(got, ref)
    integ.close()
    sc.close()


# Calls near the smallest that run staged, and on both sides of the small shading blocks' line (77,824 paths).
SMALL = {
    "spheres_one_pass": (lambda: sphere_box_scene(31, 30000, 47, 45), dict(max_depth=5), 1),
    "cornell_three_passes": (lambda: cornell_scene(seed=32, width=57, height=49), dict(max_depth=5), 3),
    "cornell_below": (lambda: cornell_scene(seed=33, width=192, height=200), dict(max_depth=3), 2),
    "cornell_above": (lambda: cornell_scene(seed=33, width=197, height=199), dict(max_depth=3), 2),
    "zoo_one_pass": (lambda: material_zoo_scene(seed=34, width=391, height=373), dict(max_depth=4), 1),
    "textured_two_passes": (lambda: textured_scene(seed=35, width=67, height=63, base="zoo"), dict(max_depth=4), 2),
}


# One pass of the one-kernel tracer with 4, 8, 16 and 32 paths a warp (render_kernels.cuh: path_lanes).
SMALL.update({
    "thin_%dx%d_%s" % (w, h, m.__name__): ((lambda m=m, w=w, h=h: m(seed=36, width=w, height=h)), dict(max_depth=4), 1)
    for m, w, h in ((cornell_scene, 1, 1), (cornell_scene, 37, 31), (cornell_scene, 67, 63), (cornell_scene, 89, 91),
                    (cornell_scene, 131, 123), (cornell_scene, 133, 131), (material_zoo_scene, 49, 47),
                    (material_zoo_scene, 71, 67), (material_zoo_scene, 99, 98))
})
SMALL["spheres_staged"] = (lambda: sphere_box_scene(37, 30000, 191, 181), dict(max_depth=5), 1)


@pytest.mark.parametrize("name", list(SMALL))
def test_small_calls_equal_the_oracle(zgl_lib, cuda, name):
    make, params, n = SMALL[name]
    data = make()
    sc = Scene(data)
    w, h = data.film
    orc = oracle.OracleScene(data, sc.export("sobol"), params)
    pix = np.random.default_rng(2).choice(w * h, min(w * h, 1500), replace=False).astype(np.int32)
    ref = orc.render_pt(pix, n)
    it = PathIntegrator(sc, **params)
    if n == 1:
        it.render_one_pass()
    else:
        it.render_passes(n)
    got = it.get_frame()[0][..., :3].reshape(-1, 3)[pix]
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    for x in (it, sc):
        x.close()
