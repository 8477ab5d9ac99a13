"""Jets of the log-domain family whose coefficients pass through FP32 numbers
below 2^-126 (powers of weak fields, thin far densities): the mixed render
follows FP64, in every form, as far as a subnormal factor resolves it -- one of
2^-126 2^-k has 23 - k bits.  At the weakest cases here k is 8 or less over the
jet, so a relative 2^-14 of tau and I; and renders in the normal range are the
same bits in the fused and in the every-law kernels."""
import math

import numpy as np
import pytest

from jetshow_gb300 import _capi as A
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W

pytestmark = pytest.mark.gpu

NU = np.array([15.4e9 * 1.1])
KW = dict(W.ACCURATE_KW, tau_min=0.0, tau_atol=1e-60, atol=1e-70)
KW_I = dict(KW, output="I")  # at these densities full Stokes is a question of Faraday rotations


def plane():
    lg = math.log10(0.5 * 1.8443 * J.pc)
    return J.ImagePlane((4, 6), lg, lg, 0.1).desc()


@pytest.mark.parametrize("s,b0,n0", [(6.0, 2e-9, 1e25), (6.0, 1e-9, 1e25), (5.0, 5e-11, 1e25), (4.0, 1e-12, 1e28)])
def test_weak_fields(ctx, s, b0, n0):
    jet = W.conical_model(b0=b0, n0=n0, s=s).desc()
    f, _ = ctx.render(jet, plane(), NU, J.make_params(precision="fp64", schedule="static", **KW_I))
    assert (f["tau"] > 0).any()
    for schedule, flags in (("persistent", 0), ("persistent", A.FLAG_SINGLE_KERNEL), ("static", 0)):
        g, _ = ctx.render(jet, plane(), NU, J.make_params(precision="mixed", schedule=schedule, flags=flags, **KW_I))
        hit = f["tau"] > 0
        np.testing.assert_allclose(g["tau"][hit], f["tau"][hit], rtol=2.0 ** -14)
        np.testing.assert_allclose(g["I"][hit], f["I"][hit], rtol=2.0 ** -14)


@pytest.mark.parametrize("s,b0,n0", [(2.5, 0.1, 500.0), (6.0, 1e-3, 500.0), (3.0, 1e-7, 1e-6)])
def test_normal_range_same_bits(ctx, s, b0, n0):
    jet = W.conical_model(b0=b0, n0=n0, s=s).desc()
    a, _ = ctx.render(jet, plane(), NU, J.make_params(precision="mixed", schedule="persistent", **KW))
    b, _ = ctx.render(jet, plane(), NU, J.make_params(precision="mixed", schedule="persistent",
                                                     flags=A.FLAG_GENERAL_KERNELS, **KW))
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
