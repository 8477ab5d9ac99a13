"""The forms that spread one ray over several lanes, at the sizes where their
maps can go wrong.

* The stripe pass, 32 steps of a pixel at a time: step counts around 32 and a
  stop inside a group of steps, against the oracle to the last bits of pow
  over n steps (1e-10, as the stripe test).
"""
import numpy as np
import pytest

from jetshow_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("tau_max", [1e4, 0.5])
def test_stripe_step_groups(ctx, oracle, n, tau_max):
    jet, plane, nu, _ = W.conical_c1(scale=8)
    g = ctx.stripe(jet.desc(), plane.desc(), nu[0], n=n, tau_max=tau_max)
    r = oracle.stripe(jet.desc(), plane.desc(), nu[0], n=n, tau_max=tau_max)
    assert np.array_equal(g == 0, r == 0) and (g > 0).any()
    np.testing.assert_allclose(g, r, rtol=1e-10, atol=0)
