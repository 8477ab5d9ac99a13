"""The along tables of an image plane, uploaded with a request up to 16 384
columns and walked by the device's serial kernel above: origins and sizes bit
for bit the oracle's on both sides of the line, and a ring of uploads longer
than its stages keeps every render's own plane."""
import math

import numpy as np
import pytest

from jetshow_gb300 import jet as J
from jetshow_gb300 import runtime as R
from jetshow_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("along", [1, 2, 16384, 16385])
def test_plane_tables_bit_exact(ctx, oracle, along):
    # one column has no base (a division by zero in the reference): skip its size step
    plane = J.ImagePlane((4, along), 15.0, 15.0 if along == 1 else 15.4, 0.1)
    o, d, s = ctx.plane_rays(plane.desc())
    oo, od, os_ = oracle.plane_rays(plane.desc())
    assert np.array_equal(o, oo) and np.array_equal(d, od) and np.array_equal(s, os_)
    assert np.array_equal(ctx.plane_sizes(plane.desc()), os_)


def test_uploads_in_turn(ctx):
    """Ten renders enqueued without a wait between them, each with its own
    plane, frequency and output: as each by itself."""
    torch = pytest.importorskip("torch")
    jet = W.conical_model().desc()
    params = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_KW)
    planes = [J.ImagePlane((16, 20 + k), 17.0 + 0.05 * k, 17.4, 0.1) for k in range(10)]
    outs = []
    for k, plane in enumerate(planes):
        out = torch.zeros((1, 16, 20 + k), dtype=torch.float64, device="cuda")
        ctx.render_device(jet, plane.desc(), np.array([8e9 + 1e9 * k]), params, 0, {"I": out.data_ptr()})
        outs.append(out)
    torch.cuda.synchronize()
    for k, plane in enumerate(planes):
        ref, _ = ctx.render(jet, plane.desc(), np.array([8e9 + 1e9 * k]), params)
        assert np.array_equal(outs[k].cpu().numpy(), ref["I"]) and ref["I"].max() > 0


def test_fp64_request_fits_its_budget(ctx):
    """The FP64 path has no FP32 segments: a 128x128 request takes about 205
    bytes a pixel of a context's budget, and not the 128 more of a mixed one."""
    jet = W.conical_model()
    lg = math.log10(0.4 * 1.8443 * J.pc)
    plane = J.ImagePlane((128, 128), lg, lg, 0.1)
    nu = np.array([15.4e9])
    kw = dict(W.ACCURATE_KW, output="I", precision="fp64")
    small = R.Context(0, hbm_budget_bytes=5 << 20)
    try:
        g, _ = small.render(jet.desc(), plane.desc(), nu, J.make_params(**kw))
    finally:
        small.close()
    w, _ = ctx.render(jet.desc(), plane.desc(), nu, J.make_params(**kw))
    for k in w:
        assert np.array_equal(g[k], w[k]), k
