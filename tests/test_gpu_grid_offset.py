"""A grid whose offset is large against its extent: the index stays within a few
hundred bytes a triangle (a budget of 32 MB holds it), and the FP64
interpolation is the oracle's, bit for bit."""
import numpy as np
import pytest

from jetshow_gb300.runtime import Context, triangulate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1e2, 1e4, 1e5, 1e7])
def test_offset_grid(lib, oracle, offset):
    rng = np.random.default_rng(4)
    xy = rng.random((20_000, 2)) + [offset, 0.0]
    vals = rng.random((20_000, 1)).astype(np.float32)
    tri = triangulate(xy)
    c = Context(0, 32 << 20)
    gid = c.grid_upload(xy, vals, tri)
    oracle.grid_register(gid, xy, vals, tri)
    q = np.vstack([rng.uniform(-0.1, 1.1, (2000, 2)) + [offset, 0.0], xy[:500]])
    g = c.grid_interpolate(gid, 0, q, nan_value=-7.0)
    r = np.array([oracle.grid_value(gid, 0, z, rr, -7.0) for z, rr in q])
    assert np.array_equal(g, r)
    assert (r != -7.0).sum() > 1500
    c.close()
