"""Which kernels a call runs (csrc/staged.h: staged_pays and its like), and the
frames of the staged ones: depth 0, the largest staged depth and the next, no
light samples, textures, and every size of shading block."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from zillumgl_gb300 import BVH
from zillumgl_gb300.scene import DiffRenderer, LightIntegrator, PathIntegrator, Scene
from zillumgl_gb300.synthetic import (cornell_scene, diff_scene, material_zoo_scene, sphere_box_scene, textured_scene,
                                      triangle_soup)

from tests.test_diff_gpu import GRAD_ABS, GRAD_REL

pytestmark = pytest.mark.gpu

W, H = 331, 301


def _profile(call):
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return " ".join(e.key for e in p.key_averages())


@pytest.fixture(scope="module", autouse=True)
def profiler(cuda):
    """The first profile of a process may come back empty."""
    import torch

    for _ in range(5):
        if _profile(lambda: torch.zeros(1 << 20, device=cuda).add_(1)):
            return
    pytest.skip("no kernel records from the profiler")


def _kernels(call):
    """Names of the kernels that `call` launches."""
    names = _profile(call)
    assert names, "the profiler saw no kernel"
    return names.replace("(int)", "").replace("(bool)1", "true").replace("(bool)0", "false")


STAGED = "staged_trace_kernel"
CASES = {  # scene, parameters, passes, a kernel that has to run
    "no_light_samples": (lambda: cornell_scene(seed=61, width=W, height=H), dict(max_depth=3, sample_light=0), 2, STAGED),
    "depth_0": (lambda: cornell_scene(seed=62, width=W, height=H), dict(max_depth=0), 2, STAGED),
    "depth_24": (lambda: cornell_scene(seed=63, width=W, height=H), dict(max_depth=24), 2, STAGED),
    "depth_25": (lambda: cornell_scene(seed=63, width=W, height=H), dict(max_depth=25), 2, "path_passes_kernel"),
    "textured": (lambda: textured_scene(seed=64, width=W, height=H, base="zoo"), dict(max_depth=4), 2, STAGED),
    "shade_128": (lambda: cornell_scene(seed=65, width=91, height=93), dict(max_depth=4), 2, "staged_shade_kernel<false, 128>"),
    "shade_128_full": (lambda: material_zoo_scene(seed=65, width=91, height=93), dict(max_depth=4), 2,
                       "staged_shade_kernel<true, 128>"),
    "shade_512": (lambda: cornell_scene(seed=66, width=W, height=H), dict(max_depth=4), 2, "staged_shade_kernel<false, 512>"),
    "shade_512_full": (lambda: material_zoo_scene(seed=66, width=W, height=H), dict(max_depth=4), 2,
                       "staged_shade_kernel<true, 512>"),
    "shade_1024_full": (lambda: material_zoo_scene(seed=67, width=W, height=H), dict(max_depth=4), 6,
                        "staged_shade_kernel<true, 1024>"),
    "one_pass": (lambda: cornell_scene(seed=68, width=401, height=397), dict(max_depth=4), 1, STAGED),
    "one_pass_full": (lambda: material_zoo_scene(seed=68, width=391, height=373), dict(max_depth=4), 1, STAGED),
    "one_pass_below": (lambda: cornell_scene(seed=69, width=W, height=H), dict(max_depth=4), 1, "path_kernel<"),
    "one_pass_large_tree": (lambda: sphere_box_scene(70, 30000, 191, 181), dict(max_depth=4), 1, STAGED),
}


@pytest.mark.parametrize("name", list(CASES))
def test_route_and_frame(zgl_lib, cuda, name):
    make, params, n, kernel = CASES[name]
    data = make()
    sc = Scene(data)
    it = PathIntegrator(sc, **params)
    call = it.render_one_pass if n == 1 else lambda: it.render_passes(n)
    names = _kernels(call)
    assert kernel in names, names
    w, h = data.film
    pix = np.random.default_rng(3).choice(w * h, 700, replace=False).astype(np.int32)
    ref = oracle.OracleScene(data, sc.export("sobol"), params).render_pt(pix, n)
    got = it.get_frame()[0][..., :3].reshape(-1, 3)[pix]
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
    it.close()
    sc.close()


def test_light_passes_run_staged(zgl_lib, cuda):
    sc = Scene(cornell_scene(seed=71, width=96, height=80))
    many, few = LightIntegrator(sc, max_depth=4, blocks_per_pass=64), LightIntegrator(sc, max_depth=4, blocks_per_pass=8)
    assert "light_trace_kernel" in _kernels(many.render_one_pass)
    assert "light_trace_kernel" not in _kernels(few.render_one_pass)
    for x in (many, few, sc):
        x.close()


@pytest.mark.parametrize("case", ["principled", "cornell_rr", "env_two_lights"])
def test_staged_adjoint_against_64_bits(zgl_lib, cuda, case):
    """test_diff_gpu.py's comparison with the FP64 adjoint, with paths enough
    (33,282 and more) for the staged replay."""
    import torch

    if case == "principled":
        d, spp, params = diff_scene(seed=72, width=129, height=129), 2, dict(max_depth=6)
    elif case == "cornell_rr":
        d, spp, params = (cornell_scene(seed=73, width=131, height=127), 2,
                          dict(max_depth=6, russian_roulette=1, rr_start_depth=2))
    else:
        from tests.test_tables import _multi_light_scene

        d, spp, params = _multi_light_scene(env=True, w=133, h=127), 2, dict(max_depth=4)
    sc = Scene(d)
    r = DiffRenderer(sc, spp, **params)
    w, h = d.film
    adj = np.random.default_rng(5).uniform(-1.0, 1.0, (h, w, 3)).astype(np.float32)
    dev = torch.from_numpy(adj).to(cuda)
    r.forward()
    grad = []
    assert "replay_step_kernel" in _kernels(lambda: grad.append(r.backward(dev)))
    g = grad[0].cpu().numpy().astype(np.float64)
    ref = oracle.OracleScene(d, sc.export("sobol"), params).diff_grad(d, spp, adj)
    assert np.abs(ref).max() > 0
    assert np.all(np.abs(g - ref) <= GRAD_ABS * np.abs(ref).max() + GRAD_REL * np.abs(ref))
    r.close()
    sc.close()


def test_axis_plane_rays_over_a_ground_quad(zgl_lib, cuda):
    """One large triangle ends the pad's culling at the root: rays with a zero
    component get the short budget there and finish on the face table."""
    import torch

    v, idx = triangle_soup(1 << 16, 74)
    ground = np.array([[-1, -1, -0.1], [2, -1, -0.1], [2, 2, -0.1], [-1, 2, -0.1]], np.float32)
    idx = np.concatenate([idx, np.array([0, 1, 2, 0, 2, 3], np.uint32) + v.shape[0]]).astype(np.uint32)
    v = np.concatenate([v, ground]).astype(np.float32)
    acc = BVH(v, idx).build_device()
    n = 1024
    rng = np.random.default_rng(9)
    o = rng.random((n, 3)).astype(np.float32)
    d = rng.standard_normal((n, 3))
    d[np.arange(n), np.arange(n) % 3] = rng.choice([0.0, 1e-9, -5e-7], n)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    tm = torch.from_numpy(rng.random(n).astype(np.float32)).to(cuda)
    to, td = torch.from_numpy(o).to(cuda), torch.from_numpy(d.astype(np.float32)).to(cuda)
    ids, t = acc.trace_closest(to, td)
    occ = acc.trace_any(to, td, tm)
    acc.set_trace_schedule("thread_per_ray")
    rid, rt = acc.trace_closest(to, td)
    assert torch.equal(ids, rid) and torch.equal(t.view(torch.int32), rt.view(torch.int32))
    assert torch.equal(occ, acc.trace_any(to, td, tm))
    assert int((ids >= 0).sum()) > n // 4
    acc.close()
