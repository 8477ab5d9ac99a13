"""FP64 renders of densities below zero: the plasma frequency is the square
root of the density, so an item whose k_I meets a negative one (or whose
Faraday rotation meets a negative thermal fraction) ends with JSH_ST_NAN, as
in the oracle, whatever the field law, the frame and the schedule.  A density
of zero, of either sign, is none of these."""
import math

import numpy as np
import pytest

from jetshow_gb300 import _capi as A
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("n0,frame,thermal,tangled", [(-500.0, True, 0.0, False), (-500.0, False, 0.0, False),
                                                      (-500.0, True, 0.0, True), (500.0, True, -0.1, False),
                                                      (0.0, True, 0.0, False), (-0.0, True, 0.1, False)])
def test_density_below_zero_is_an_error(ctx, oracle, output, n0, frame, thermal, tangled):
    jet = W.conical_model(thermal_fraction=thermal)
    jet.nfield = J.BKNField(n0, 2.0, frame)
    if tangled:
        jet.bfield = J.RandomScalarBFieldZ(0.1, 1.0)
    lg = math.log10(12.8 / 12 * 1.8443 * J.pc)
    plane, nu = J.ImagePlane((6, 12), lg, lg, 0.1), np.array([15.4e9 * 1.1])
    kw = dict(W.ACCURATE_KW, output=output)
    r = oracle.render(jet.desc(), plane.desc(), nu, J.make_params(precision="fp64", schedule="static", **kw))
    failed = n0 < 0 or (thermal < 0 and output == "full")
    for schedule in ("static", "persistent"):
        g, st = ctx.render(jet.desc(), plane.desc(), nu, J.make_params(precision="fp64", schedule=schedule, **kw))
        assert np.array_equal(g["status"].reshape(1, -1), r["status"])
        hit = (r["status"] & A.ST_HIT) != 0
        assert hit.any() and np.all(((r["status"][hit] & A.ST_NAN) != 0) == failed)
        assert bool(st["status_or"] & A.ST_NAN) == failed
        if failed:  # the state before the failing step
            for k in ("I", "Q", "U", "V"):
                assert np.array_equal(g[k].reshape(1, -1), r[k], equal_nan=True), k
