"""IVF routing at the edges of the device kernels: one or four queries per
thread, dimensions that do not fill a load batch, and both sort kernels (one
key per thread up to 1024 lists), against the host probe_route."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_route import empty_ivf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlist,d,B,nprobe", [(64, 1, 1, 64), (65, 31, 3, 65), (640, 33, 64, 8), (1024, 64, 41, 1024),
                                              (1025, 97, 37, 7), (2400, 5, 17, 2400), (33, 768, 130, 32)])
def test_route_sizes_match_host(ctx, nlist, d, B, nprobe):
    from bn_b200 import capi as c

    rng = np.random.default_rng(nlist * 7 + d)
    # few distinct values: equal distances are common, and the lower list ranks first
    cen = rng.integers(-2, 3, size=(nlist, d)).astype(np.float32)
    q = rng.integers(-2, 3, size=(B, d)).astype(np.float32)
    v = empty_ivf(ctx, nlist)
    v.set_centroids(cen)
    got = v.route(q, nprobe)
    assert np.array_equal(got, c.host_probe_route(cen, q, nprobe))
    v.close()
