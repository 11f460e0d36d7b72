"""Axis-dominant rays whose origin lies next to a box plane (csrc/wide.cuh):
boxHit asks `lo < o < hi` on the two other axes, however small the difference."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from zillumgl_gb300 import BVH

pytestmark = pytest.mark.gpu


def _walls(n, axis, side):
    """n triangles across `axis`, one edge of each in the plane 0 of the next
    axis, the rest on its negative (side -1) or positive side; small enough
    (squared box diagonal 0.125) for the tree to cull beside them."""
    b, c = (axis + 1) % 3, (axis + 2) % 3
    v = np.zeros((n, 3, 3), np.float32)
    v[:, :, axis] = np.arange(1, n + 1, dtype=np.float32)[:, None]
    v[:, 1, c] = 0.25
    v[:, 2, b] = 0.25 * side
    v[:, 2, c] = 0.125
    return v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", [-1.0, 1.0])
def test_origins_next_to_a_box_plane(zgl_lib, cuda, axis, side):
    import torch

    v, idx = _walls(64, axis, side)
    acc = BVH(v, idx).build()
    p = acc.export()
    b, c = (axis + 1) % 3, (axis + 2) % 3
    gap = np.concatenate([[0.0, 1e-45, 3e-39], np.float32(3.7) * 10.0 ** np.arange(-37, 0)])
    gap = np.concatenate([gap, -gap]).astype(np.float32)
    n = gap.size
    o = np.zeros((2 * n, 3), np.float32)
    o[:, axis] = np.repeat([0.25, 70.0], n)
    o[:, b] = np.tile(gap, 2)
    o[:, c] = 0.125
    d = np.zeros((2 * n, 3), np.float32)
    d[:, axis] = np.repeat([1.0, -1.0], n)
    tmax = np.full(2 * n, 100.0, np.float32)
    to, td, tm = (torch.from_numpy(x).to(cuda) for x in (o, d, tmax))
    ids, t = acc.trace_closest(to, td)
    occ = acc.trace_any(to, td, tm)
    rid, rt, _, _ = oracle.trace(p.bounds, p.hitTable, v, idx, o, d)
    ro = oracle.trace(p.bounds, p.hitTable, v, idx, o, d, tmax=tmax, any_hit=True)[0]
    assert int((rid >= 0).sum()) >= n // 2
    assert np.array_equal(ids.cpu().numpy(), rid)
    assert np.array_equal(t.cpu().numpy().view(np.uint32), rt.view(np.uint32))
    assert np.array_equal(occ.cpu().numpy().astype(np.int32), ro.astype(np.int32))
    acc.close()
