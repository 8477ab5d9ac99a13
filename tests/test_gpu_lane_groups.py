"""The forms that spread one ray over several lanes, at the sizes where their
maps can go wrong.

* FP64 transfer, five lanes an item, six items a warp, 24 a CTA: item counts
  around those edges, one and two segments a ray, random directions drawn at
  every evaluation (a sixth evaluation per step); the static and the queue
  schedule bitwise the same, and the oracle at the same tolerances within the
  contract gates.
* Mixed precision, an item on one lane (static schedule) or on a group of five
  (persistent schedule, up to a number of items): every plane and counter
  bitwise the same, for the fused family and the general build, with a random
  direction per evaluation, and on a gridded field, whose point location
  tries the triangle of the point before.
* The stripe pass, 32 steps of a pixel at a time: step counts around 32 and a
  stop inside a group of steps, against the oracle to the last bits of pow
  over n steps (1e-10, as the stripe test).
"""
import math

import numpy as np
import pytest

from jetshow_gb300 import _capi as A
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W
from helpers import compare_images, flat

pytestmark = pytest.mark.gpu


def conical(points=False, half=0.05):
    jet = W.conical_model(half_angle=half)
    if points:
        jet.bfield = J.PointsRandomVectorBField(jet.bfield, 0.3, seed=11)
    return jet


@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("along,n_nu,half", [(2, 1, 0.05), (3, 1, 0.05), (4, 2, 0.05), (13, 1, 0.05), (5, 1, 0.15)])
def test_fp64_groups(ctx, oracle, output, along, n_nu, half):
    lg = math.log10(0.4 * 1.8443 * J.pc)
    plane = J.ImagePlane((2, along), lg, lg, 0.1)
    nu = np.array([8e9, 15.4e9][:n_nu]) * 1.1
    jet = conical(half=half)
    kw = dict(W.ACCURATE_KW, output=output)
    g, st = ctx.render(jet.desc(), plane.desc(), nu, J.make_params(precision="fp64", schedule="static", **kw))
    q, sq = ctx.render(jet.desc(), plane.desc(), nu, J.make_params(precision="fp64", schedule="persistent", **kw))
    assert st["n_work_items"] > 0
    for k in g:
        assert np.array_equal(g[k], q[k]), k
    assert (st["rhs_evals"], st["steps_accepted"], st["steps_rejected"]) == (
        sq["rhs_evals"], sq["steps_accepted"], sq["steps_rejected"])
    r = oracle.render(jet.desc(), plane.desc(), nu, J.make_params(precision="fp64", schedule="static", **kw))
    compare_images(flat(g), r, full=output == "full", tau_max=1e4)


def test_fp64_group_random_directions(ctx, oracle):
    """The sixth evaluation of a step has a direction of its own: the image
    follows the oracle's draws (evaluation by evaluation) and differs from
    the unperturbed field's."""
    plane = W.conical_c0(scale=16)[1]
    nu = np.array([16.94e9])
    p = J.make_params(precision="fp64", schedule="static", **dict(W.ACCURATE_KW, tau_rtol=1e-3, rtol=1e-3, dt_max=0.0))
    g, _ = ctx.render(conical(True).desc(), plane.desc(), nu, p)
    r = oracle.render(conical(True).desc(), plane.desc(), nu, p)
    assert np.array_equal(g["status"].reshape(1, -1) & 1, r["status"] & 1)
    hit = (r["status"] & 1) != 0
    # the draws never converge: only the same directions at the same
    # evaluations give the same image, up to the last bits of pow
    np.testing.assert_allclose(g["I"].reshape(1, -1)[hit], r["I"][hit], rtol=1e-6)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("tau_max", [1e4, 0.5])
def test_stripe_step_groups(ctx, oracle, n, tau_max):
    jet, plane, nu, _ = W.conical_c1(scale=8)
    g = ctx.stripe(jet.desc(), plane.desc(), nu[0], n=n, tau_max=tau_max)
    r = oracle.stripe(jet.desc(), plane.desc(), nu[0], n=n, tau_max=tau_max)
    assert np.array_equal(g == 0, r == 0) and (g > 0).any()
    np.testing.assert_allclose(g, r, rtol=1e-10, atol=0)


@pytest.fixture(scope="module")
def grid_id(ctx):
    from jetshow_gb300.runtime import triangulate
    xy, vals = W.simulation_grid_c3(n_points=20_000)
    return ctx.grid_upload(xy, vals, triangulate(xy))


def mixed_jet(kind, grid_id):
    jet = conical(points=kind == "points")
    if kind == "sheath":
        jet.vfield = J.SheathFlatVField(10.0, 3.0, 0.5 * J.pc)
    elif kind == "tangled":
        jet.bfield = J.RandomScalarBFieldZ(0.1, 1.0)
    elif kind == "grid":
        jet.vfield, jet.nfield = J.SimulationVField(grid_id, 3), J.SimulationNField(grid_id, 2, True)
        jet.bfield = J.SimulationBField(grid_id, 0, 1, True)
    return jet


@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("kind", ["fused", "general", "sheath", "tangled", "points", "grid"])
@pytest.mark.parametrize("shape,n_nu", [((2, 2), 1), ((2, 7), 1), ((6, 13), 3), ((64, 66), 1)])
def test_mixed_groups_match_lanes(ctx, grid_id, output, kind, shape, n_nu):
    mas = (0.01 if kind == "grid" else 6.4) / shape[1]
    lg = math.log10(mas * 1.8443 * J.pc)
    plane = J.ImagePlane(shape, lg, lg, 0.1)
    nu = np.array([8e9, 15.4e9, 22e9][:n_nu]) * 1.1
    kw = dict(W.ACCURATE_KW, output=output)
    if kind == "points":  # the draws never converge: the step limits must
        kw.update(tau_rtol=1e-3, rtol=1e-3)
    flags = A.FLAG_GENERAL_KERNELS if kind == "general" else 0
    jet = mixed_jet(kind, grid_id).desc()
    a, sa = ctx.render(jet, plane.desc(), nu, J.make_params(precision="mixed", schedule="static", **kw))
    b, sb = ctx.render(jet, plane.desc(), nu, J.make_params(precision="mixed", schedule="persistent", flags=flags, **kw))
    assert sa["n_work_items"] > 0
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
    for k in ("rhs_evals", "steps_accepted", "steps_rejected", "status_or"):
        assert sa[k] == sb[k], k


@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("flags", [0, A.FLAG_FARADAY_THICK])
@pytest.mark.parametrize("shape,refill", [((80, 120), 1), ((80, 120), 0), ((128, 140), 32)])
def test_mixed_lanes_handed_to_groups(ctx, output, flags, shape, refill):
    """More items than the grid's groups take (one warp an SM): they begin on
    single lanes and the last of each warp end on its groups, bitwise as on
    one lane throughout."""
    lg = math.log10(6.4 / shape[1] * 1.8443 * J.pc)
    plane = J.ImagePlane(shape, lg, lg, 0.1)
    jet, nu = conical().desc(), np.array([8e9 * 1.1])
    kw = dict(W.ACCURATE_KW, output=output, flags=flags)
    a, sa = ctx.render(jet, plane.desc(), nu, J.make_params(precision="mixed", schedule="static", **kw))
    b, sb = ctx.render(jet, plane.desc(), nu, J.make_params(precision="mixed", schedule="persistent", block_size=32,
                                                           ctas_per_sm=1, refill_threshold=refill, **kw))
    assert sa["n_work_items"] > 4 * 6 * 152
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
    for k in ("rhs_evals", "steps_accepted", "steps_rejected", "status_or"):
        assert sa[k] == sb[k], k
