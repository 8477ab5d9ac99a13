"""The statistics of the last asynchronous render are its own after the other
calls that use the context's workspace (the stripe among them, which the CPU
test of the host calls does not link)."""
import numpy as np
import pytest

from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", ["plane_rays", "trace_plane", "stripe", "sizes", "grid", "cells", "directions"])
def test_last_stats_after(ctx, other):
    torch = pytest.importorskip("torch")
    jet, plane, nu, _ = W.conical_c0(scale=4)
    p = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_KW)
    _, want = ctx.render(jet.desc(), plane.desc(), nu, p)
    if other == "grid":
        from jetshow_gb300.runtime import triangulate
        xy = np.random.default_rng(0).random((50, 2))
        gid = ctx.grid_upload(xy, xy[:, 0], triangulate(xy))
    elif other == "cells":
        from jetshow_gb300.runtime import cells_generate
        cells = ctx.cells_upload(*cells_generate(100, J.pc, 10 * J.pc, 0.1, 2.0, 3))
    shape = (nu.size,) + tuple(plane.image_size)
    t = {k: torch.empty(shape, dtype=torch.float64, device="cuda") for k in ("tau", "l", "I", "Q", "U", "V")}
    t["status"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    ctx.render_device(jet.desc(), plane.desc(), nu, p, torch.cuda.current_stream().cuda_stream,
                      {k: v.data_ptr() for k, v in t.items()})
    if other == "plane_rays":
        ctx.plane_rays(plane.desc())
    elif other == "trace_plane":
        ctx.trace_plane(jet.desc(), plane.desc())
    elif other == "stripe":
        ctx.stripe(jet.desc(), plane.desc(), nu[0], n=10)
    elif other == "grid":
        ctx.grid_interpolate(gid, 0, xy)
    elif other == "cells":
        ctx.cells_nearest(cells, np.ones((50, 3)) * J.pc)
    elif other == "directions":
        ctx.random_directions(7, np.arange(150).reshape(50, 3))
    else:
        plane.getPixelSizes(ctx)
    got = ctx.last_stats()
    for k in ("n_pixels", "n_hit_pixels", "n_work_items", "rhs_evals", "steps_accepted", "steps_rejected",
              "status_or"):
        assert got[k] == want[k], k
    assert got["rhs_evals"] > 0
