"""The default trace schedule's 4-wide tree (csrc/wide.cuh) against the
reference's threaded loop: ids, distances and flags bit for bit, for every ray
mode, tree shape and ray count where the two paths differ in code."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from zillumgl_gb300 import BVH
from zillumgl_gb300.synthetic import city_scene, triangle_soup

pytestmark = pytest.mark.gpu


def _rays(rng, n, lo, hi):
    """Random rays; of every 16 one each: a near-zero component (one or two
    axes, zero among them), an axis-dominant direction, an unnormalised one, an
    origin far away, NaN."""
    o = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k, ax = np.arange(n), rng.integers(0, 3, n)
    one = k % 16 == 1
    d[one, ax[one]] = rng.choice([0.0, 3e-7, -9e-7], one.sum())
    two = k % 16 == 2
    d[two] = 0.6 * rng.choice([-1.0, 1.0], (two.sum(), 3))
    d[two, ax[two]] = 1e-7
    d[two, (ax[two] + 1) % 3] = -4e-7
    dom = k % 16 == 3
    d[dom] = rng.uniform(-1e-4, 1e-4, (dom.sum(), 3))
    d[dom, ax[dom]] = rng.choice([-1.0, 1.0], dom.sum())
    d[k % 16 == 4] *= 37.0
    d[k % 16 == 5] *= 1e-3
    o[k % 16 == 6] *= np.float32(1e5)
    o[k % 256 == 7] = np.float32(2e13)
    o[k % 256 == 23, 1] = np.nan
    d[k % 256 == 39, 0] = np.nan
    return o, d.astype(np.float32)


def _chain(n):
    """Identical centroids: quickBuild peels one triangle per level, deeper
    than the traversal's stack."""
    s = np.linspace(0.1, 1.0, n, dtype=np.float32)
    t = np.array([[-1, -1, 0], [1, -1, 0.5], [0, 2, -0.5]], np.float32)
    return (s[:, None, None] * t[None]).reshape(-1, 3), np.arange(3 * n, dtype=np.uint32)


def _mesh(name):
    if name == "city":
        d = city_scene(seed=4, grid=10, n_spheres=12, env_size=(8, 4))
        return d.obj_vertices, d.obj_indices, -1.0, 8.0
    if name == "doubled":  # every hit is a tie
        v, i = triangle_soup(3000, 9)
        return np.concatenate([v, v]), np.arange(18000, dtype=np.uint32), 0.0, 1.0
    if name == "far":  # coordinates far from the origin: coarse grids
        v, i = triangle_soup(4000, 12)
        return (v * 50 + 30000).astype(np.float32), i, 30000.0, 30050.0
    if name == "chain":
        return *_chain(600), -1.0, 1.0
    n = int(name)
    v, i = triangle_soup(n, 10 + n)
    return (v * 4 if n < 100 else v), i, 0.0, 1.0


@pytest.mark.parametrize("name", ["1", "2", "3", "5", "20000", "doubled", "far", "chain", "city"])
@pytest.mark.parametrize("device", [False, True])
def test_default_schedule_equals_the_reference_loop(zgl_lib, cuda, name, device):
    import torch

    v, idx, lo, hi = _mesh(name)
    v = np.ascontiguousarray(v, np.float32)
    idx = np.ascontiguousarray(idx, np.uint32)
    acc = BVH(v, idx).build_device() if device else BVH(v, idx).build()
    p = acc.export()
    for n in (1, 31, 33, 4099):
        rng = np.random.default_rng(n)
        o, d = _rays(rng, n, lo, hi)
        tmax = rng.uniform(0.0, 2.0 * (hi - lo), n).astype(np.float32)
        tmax[::7] = (np.inf, 0.0, -1.0, np.nan)[n % 4]
        to, td, tm = (torch.from_numpy(x).to(cuda) for x in (o, d, tmax))
        ids, t = acc.trace_closest(to, td)
        occ = acc.trace_any(to, td, tm)
        rid, rt, _, _ = oracle.trace(p.bounds, p.hitTable, v, idx, o, d)
        ro = oracle.trace(p.bounds, p.hitTable, v, idx, o, d, tmax=tmax, any_hit=True)[0]
        assert np.array_equal(ids.cpu().numpy(), rid)
        assert np.array_equal(t.cpu().numpy().view(np.uint32), rt.view(np.uint32))
        assert np.array_equal(occ.cpu().numpy().astype(np.int32), ro.astype(np.int32))
    acc.close()


def test_rays_in_an_axis_plane_of_a_large_mesh(zgl_lib, cuda):
    """A symmetric camera's middle column: one direction component is zero."""
    import torch

    v, idx = triangle_soup(1 << 17, 3)
    acc = BVH(v, idx).build_device()
    n = 2048
    rng = np.random.default_rng(8)
    o = rng.random((n, 3)).astype(np.float32)
    d = rng.standard_normal((n, 3))
    d[np.arange(n), np.arange(n) % 3] = rng.choice([0.0, 1e-9, -5e-7], n)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    to, td = torch.from_numpy(o).to(cuda), torch.from_numpy(d.astype(np.float32)).to(cuda)
    ids, t = acc.trace_closest(to, td)
    acc.set_trace_schedule("thread_per_ray")
    rid, rt = acc.trace_closest(to, td)
    assert torch.equal(ids, rid) and torch.equal(t.view(torch.int32), rt.view(torch.int32))
    assert int((ids >= 0).sum()) > n // 4
    acc.close()
