"""A grid under an HBM budget that holds its points, fields, triangles and lists
but not the full index (2 249 KiB at 20 000 points of four fields): the FP64
lookups are the oracle's and its renders those of the full grid, bit for bit;
the mixed renders are the same in every form, and each grid's within the
contract's tau and I gates of the converged image, so within twice these of
the other's."""
import numpy as np
import pytest

from helpers import I_RTOL, QUV_ATOL_FRAC, TAU_RTOL, compare_images, flat
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W
from jetshow_gb300.runtime import Context, triangulate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid():
    xy, vals = W.simulation_grid_c3(n_points=20_000)
    return xy, vals, triangulate(xy)


def test_fits_its_budget(lib, oracle, grid):
    xy, vals, tri = grid
    c = Context(0, 2249 << 10)
    gid = c.grid_upload(xy, vals, tri)
    oracle.grid_register(gid, xy, vals, tri)
    rng = np.random.default_rng(5)
    q = np.vstack([np.column_stack([rng.uniform(-1.0, 21.0, 3000), rng.uniform(-0.05, 0.55, 3000)]), xy[:500]])
    c.close()
    c = Context(0, (2249 + 1024) << 10)  # and the smallest workspace
    gid = c.grid_upload(xy, vals, tri)
    for field in range(vals.shape[1]):
        g = c.grid_interpolate(gid, field, q[:2000], nan_value=-7.0)
        r = np.array([oracle.grid_value(gid, field, z, rr, -7.0) for z, rr in q[:2000]])
        assert np.array_equal(g, r)
    c.close()


@pytest.mark.parametrize("fields", [4, 5])
def test_renders(ctx, grid, fields):
    xy, vals, tri = grid
    if fields == 5:  # rows of five floats, the jet's fields the last four
        vals = np.concatenate([np.zeros((len(xy), 1), np.float32), vals], 1)
    lean = Context(0, 64 << 20)  # the full index is above a thirty-second of it
    images = []
    for c in (ctx, lean):
        gid = c.grid_upload(xy, vals, tri)
        jet, plane, nu, _ = W.simulation_c3(gid, scale=16)
        d = fields - 4
        jet.vfield, jet.nfield = J.SimulationVField(gid, 3 + d), J.SimulationNField(gid, 2 + d, True)
        jet.bfield = J.SimulationBField(gid, d, 1 + d, True)
        f64, _ = c.render(jet.desc(), plane.desc(), nu, J.make_params(precision="fp64", schedule="static", **dict(
            W.ACCURATE_KW, tau_rtol=1e-4, rtol=1e-4)))
        kw = dict(W.GRID_MIXED_KW)
        a, sa = c.render(jet.desc(), plane.desc(), nu, J.make_params(precision="mixed", schedule="static", **kw))
        b, sb = c.render(jet.desc(), plane.desc(), nu, J.make_params(precision="mixed", schedule="persistent", **kw))
        assert sa["rhs_evals"] == sb["rhs_evals"]
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=True), k
        images.append((f64, a))
    for k in images[0][0]:
        assert np.array_equal(images[0][0][k], images[1][0][k], equal_nan=True), k
    compare_images(flat(images[0][1]), flat(images[1][1]), full=True, tau_max=1e4, tau_rtol=2 * TAU_RTOL,
                   i_rtol=2 * I_RTOL, quv_frac=2 * QUV_ATOL_FRAC)
    lean.close()
