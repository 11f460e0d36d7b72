"""Exports of device-built trees on both sides of the size up to which the
records are rearranged on the host (csrc/wide_build.cu: kHostExportNodes)."""
from __future__ import annotations

import numpy as np
import pytest

from zillumgl_gb300 import BVH
from zillumgl_gb300.synthetic import triangle_soup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 7, 128, 129, 4096])
def test_export_equals_the_host_build(zgl_lib, cuda, n):
    v, idx = triangle_soup(n, 300 + n)
    want = BVH(v, idx).build_host()
    acc = BVH(v, idx).build_device()
    got = acc.export()
    acc.close()
    assert np.array_equal(got.bounds.view(np.uint32), want.bounds.view(np.uint32))
    assert np.array_equal(got.hitTable, want.hitTable)
