"""zgl_trace_closest_noalloc under every schedule: after a call with one ray,
calls of any size leave the device's free memory as it is (the kernels' stacks
come with the first launch).  Runs last, as test_zz_no_alloc.py does."""
from __future__ import annotations

import numpy as np
import pytest

from zillumgl_gb300 import BVH
from zillumgl_gb300._lib import ZGL_OK
from zillumgl_gb300.synthetic import triangle_soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", ["auto", "thread_per_ray", "prefetch"])
def test_free_memory_stays(zgl_lib, cuda, schedule):
    import torch

    v, idx = triangle_soup(20000, 37)
    acc = BVH(v, idx).build()
    acc.set_trace_schedule(schedule)
    rng = np.random.default_rng(6)
    n = 1 << 17
    o = rng.random((n, 3)).astype(np.float32)
    d = rng.standard_normal((n, 3)).astype(np.float32)
    d[::64, 0] = 0.0  # rays that the default schedule sets aside
    hid, ht = np.zeros(n, np.int32), np.zeros(n, np.float32)

    def call(k):
        assert zgl_lib.zgl_trace_closest_noalloc(acc.handle, o.ctypes.data, d.ctypes.data, k, hid.ctypes.data,
                                                 ht.ctypes.data, None) == ZGL_OK, zgl_lib.zgl_last_error()

    call(1)
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    for _ in range(10):
        call(n)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    acc.close()
