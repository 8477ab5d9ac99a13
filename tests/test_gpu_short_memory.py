"""Requests under an HBM budget that holds their hits, ranking and planes but not
the 128 bytes a pixel of the hits' segments in FP32 (nor the partial sums of
the visibilities' finest split): they run without them, image by image the
bits of an unlimited context.  The budgets are the bytes of the request's
buffers, each rounded up to 256, and the 4 KiB that the records may take."""
import math

import numpy as np
import pytest

from jetshow_gb300 import _capi as A
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W
from jetshow_gb300.runtime import Context, JetshowError

pytestmark = pytest.mark.gpu

ACROSS, ALONG = 96, 128
NU = np.array([15.4e9 * 1.1])


def up(n):
    return (n + 255) // 256 * 256


def arena_bytes(n_nu):
    """Tables, hits, ranking and planes of a request."""
    npix = ACROSS * ALONG
    return (2 * up(8 * ALONG) + up(8 * ACROSS // 2 * ALONG) + up(112 * npix) + up(4 * npix) + up(npix)
            + up(32 * npix * n_nu) + up(4 * npix * n_nu) + 6 * up(8 * npix * n_nu) + up(4 * npix * n_nu))


def request(law="conical"):
    jet = W.conical_model(half_angle=0.15)  # one and two segments a ray
    if law == "sheath":
        jet.vfield = J.SheathFlatVField(10.0, 3.0, 0.5 * J.pc)
    lg = math.log10(0.1 * 1.8443 * J.pc)
    return jet.desc(), J.ImagePlane((ACROSS, ALONG), lg, lg, 0.1).desc()


def same(a, b):
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k


@pytest.mark.parametrize("schedule", ["static", "persistent"])
@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("law,flags", [("conical", 0), ("sheath", 0), ("conical", A.FLAG_FARADAY_THICK)])
def test_render(ctx, schedule, output, law, flags):
    model, plane = request(law)
    p = J.make_params(precision="mixed", schedule=schedule, flags=flags, **dict(W.ACCURATE_KW, output=output))
    a, sa = ctx.render(model, plane, NU, p)
    small = Context(0, arena_bytes(1) + 8192)
    for _ in range(2):
        b, sb = small.render(model, plane, NU, p)
        same(a, b)
        assert sa["rhs_evals"] == sb["rhs_evals"] and sa["n_work_items"] > 0
    small.close()
    none = Context(0, arena_bytes(1) // 2)
    with pytest.raises(JetshowError) as e:
        none.render(model, plane, NU, p)
    assert e.value.status == A.JSH_ERR_OOM
    none.close()


def test_visibilities(ctx):
    model, plane = request()
    p = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_I_KW)
    n_uv = 3000
    uv = np.random.default_rng(1).uniform(-1e8, 1e8, (n_uv, 2))
    scale = 4.84813681109536e-09 / (1.8443 * J.pc)
    a, _ = ctx.visibilities(model, plane, NU, p, uv, scale, 1.0)
    # four CTAs an SM: 26 splits of 24 groups of 128 points, one a column group of 5
    splits = -(-ALONG // -(-ALONG // -(-4 * 152 // 24)))
    extra = up(4 * ALONG * ACROSS) + 2 * up(8 * ALONG) + 3 * up(16 * n_uv) + up(16 * splits * n_uv)
    small = Context(0, arena_bytes(1) + extra + 8192)
    b, _ = small.visibilities(model, plane, NU, p, uv, scale, 1.0)
    np.testing.assert_allclose(a, b, rtol=0, atol=1e-12 * np.abs(a).max())  # another split of the FP64 sums
    small.close()


@pytest.mark.parametrize("graphs", [True, False])
def test_served(ctx, graphs):
    from jetshow_gb300.serving import Server
    model, plane = request()
    p = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_KW)
    a, _ = ctx.render(model, plane, NU, p)
    s = Server(max_inflight_batches=1, max_batch_requests=2, hbm_budget_bytes=arena_bytes(1), use_graphs=graphs)
    ids = [s.submit(model, plane, NU, p) for _ in range(2)]
    for i in ids:
        same(a, s.wait(i)[0])
    s.close()
