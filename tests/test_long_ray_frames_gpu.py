"""Long rays in the integrators' 16x8 blocks (csrc/traverse.cuh:
traverse_group, finish_long_rays_group): a warp is two rows of a tile, so its
lanes are not threadIdx.x."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from zillumgl_gb300.scene import BatchRenderer, PathIntegrator, Scene
from zillumgl_gb300.synthetic import city_scene, triangle_soup

from tests import test_group_walk_gpu as walk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("any_hit", [False, True])
def test_group_walks_in_tiles(zgl_lib, cuda, any_hit):
    import torch

    f = walk._library().group_walk_tile
    f.restype, f.argtypes = walk._library().group_walk.restype, walk._library().group_walk.argtypes
    va, ia = triangle_soup(60000, 5)
    vb, ib = triangle_soup(30000, 7)
    na, ta, ma, pa = walk._device_tables(va, ia, cuda)
    nb, tb, mb, pb = walk._device_tables(vb, ib, cuda)
    n = 8192 + 77
    o, d = walk._rays(np.random.default_rng(61), n)
    tmax = (np.random.default_rng(62).random(n) * 2.0).astype(np.float32)
    even, odd = np.arange(0, n, 2), np.arange(1, n, 2)
    refs = [oracle.trace(p.bounds, p.hitTable, v, i, o[k], d[k], tmax=tmax[k] if any_hit else None, any_hit=any_hit)
            for p, v, i, k in ((pa, va, ia, even), (pb, vb, ib, odd))]
    assert all(int((r[2] > 256).sum()) >= 20 for r in refs), "too few rays past the budget"
    to, td, tm = (torch.from_numpy(x).to(cuda) for x in (o, d, tmax))
    ids = torch.full((n,), -7, dtype=torch.int32, device=cuda)
    ts = torch.zeros(n, dtype=torch.float32, device=cuda)
    assert f(na.data_ptr(), ta.data_ptr(), ma, nb.data_ptr(), tb.data_ptr(), mb, to.data_ptr(), td.data_ptr(),
             tm.data_ptr(), n, int(any_hit), ids.data_ptr(), ts.data_ptr()) == 0
    ids, ts = ids.cpu().numpy(), ts.cpu().numpy()
    for k, r in ((even, refs[0]), (odd, refs[1])):
        assert np.array_equal(ids[k], r[0].astype(np.int32))
        if not any_hit:
            assert np.array_equal(ts[k].view(np.uint32), r[1].view(np.uint32))


@pytest.mark.parametrize("seed", [2, 3])
def test_integrator_and_batch_agree_on_a_large_tree(zgl_lib, cuda, seed):
    """One 1080p pass of a city of 3.9M triangles: the integrator traces in
    16x8 blocks, the batched renderer on ray lists; every pixel is the same, and
    a sample of them the oracle's."""
    import torch

    data = city_scene(seed=seed, width=1920, height=1080, grid=64, n_spheres=2000, env_size=(1024, 512))
    params = dict(max_depth=8, russian_roulette=1, rr_start_depth=3)
    sc = Scene(data)
    it = PathIntegrator(sc, **params)
    it.render_one_pass()
    got = it.get_frame()[0]
    frame = torch.zeros((1080, 1920, 4), device=cuda)
    batch = BatchRenderer([(sc, 1, params, frame)])
    batch.render()
    torch.cuda.synchronize()
    want = frame.cpu().numpy()
    differ = np.nonzero((got.view(np.uint32) != want.view(np.uint32)).any(-1).reshape(-1))[0]
    pix = np.concatenate([differ[:50], np.random.default_rng(1).choice(1920 * 1080, 200)]).astype(np.int32)
    ref = oracle.OracleScene(data, sc.export("sobol"), params).render_pt(pix, 1)
    assert np.array_equal(want.reshape(-1, 4)[pix, :3].view(np.uint32), ref.view(np.uint32))
    assert differ.size == 0, f"pixels {differ[:8].tolist()}"
    batch.close()
    it.close()
    sc.close()
