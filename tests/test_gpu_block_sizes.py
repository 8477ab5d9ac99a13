"""Threads per CTA of the persistent mixed schedule, up to the largest that the
parameters take (512, run as 256): every form and build launches, its stage
storage above the 48 KB of an unasked launch included, and renders bitwise
what the static schedule does.  The every-law split form runs its lanes here
(more items an SM than it puts on groups), not its groups."""
import math

import numpy as np
import pytest

from jetshow_gb300 import _capi as A
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W

pytestmark = pytest.mark.gpu

NU = np.array([15.4e9 * 1.1])


@pytest.fixture(scope="module")
def grid_id(ctx):
    from jetshow_gb300.runtime import triangulate
    xy, vals = W.simulation_grid_c3(n_points=20_000)
    return ctx.grid_upload(xy, vals, triangulate(xy))


def model(law, grid_id):
    jet = W.conical_model()
    if law == "sheath":
        jet.vfield = J.SheathFlatVField(10.0, 3.0, 0.5 * J.pc)
    elif law == "grid":
        jet.vfield, jet.nfield = J.SimulationVField(grid_id, 3), J.SimulationNField(grid_id, 2, True)
        jet.bfield = J.SimulationBField(grid_id, 0, 1, True)
    return jet.desc()


def square(shape, mas):
    lg = math.log10(mas / shape[1] * 1.8443 * J.pc)
    return J.ImagePlane(shape, lg, lg, 0.1).desc()


def compare(ctx, jet, plane, blocks, output, flags):
    kw = dict(W.ACCURATE_KW, output=output)
    thick = flags & A.FLAG_FARADAY_THICK
    a, sa = ctx.render(jet, plane, NU, J.make_params(precision="mixed", schedule="static", flags=thick, **kw))
    for bs in blocks:
        b, sb = ctx.render(jet, plane, NU, J.make_params(precision="mixed", schedule="persistent", block_size=bs,
                                                         flags=flags, **kw))
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=True), (bs, k)
        for k in ("rhs_evals", "steps_accepted", "steps_rejected", "status_or"):
            assert sa[k] == sb[k], (bs, k)
    return sa


@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("law,flags", [("fused", 0), ("fused", A.FLAG_GENERAL_KERNELS), ("sheath", 0),
                                       ("sheath", A.FLAG_FARADAY_THICK), ("grid", 0)])
def test_split_form(ctx, grid_id, output, law, flags):
    # the gridded image is narrow about the jet: few of its rays hit
    shape, mas = ((128, 1040), 12.8 if law != "grid" else 0.04)
    st = compare(ctx, model(law, grid_id), square(shape, mas), (64, 128, 256, 512), output, flags)
    assert st["n_work_items"] > 0


@pytest.mark.parametrize("output", ["I", "full"])
@pytest.mark.parametrize("law", ["fused", "sheath"])
@pytest.mark.parametrize("flags", [0, A.FLAG_FARADAY_THICK, A.FLAG_COMPACT_REGS])
def test_single_kernel_form(ctx, grid_id, output, law, flags):
    st = compare(ctx, model(law, grid_id), square((32, 48), 6.4), (32, 96, 256, 512), output,
                 flags | A.FLAG_SINGLE_KERNEL)
    assert st["n_work_items"] > 0


def test_shape_tuned_on_another_output(ctx, grid_id):
    """The shape that a Stokes I request tunes is the default of the context's
    full-Stokes requests of every law."""
    from jetshow_gb300.runtime import Context
    c = Context(0)
    plane = square((128, 1040), 12.8)
    c.autotune(model("fused", grid_id), plane, NU, J.make_params(precision="mixed", schedule="persistent",
                                                                **W.ACCURATE_I_KW))
    p = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_KW)
    a, _ = ctx.render(model("sheath", grid_id), plane, NU, p)
    b, _ = c.render(model("sheath", grid_id), plane, NU, p)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
    c.close()
