"""The staged columns of the visibility sum at the row counts where their shared
memory changes: 48 KB of columns (1 536 rows, beside which the kernel's static
arrays have to fit), the last count with eight columns and the first with
seven, and one column alone; against the exact sum at the gate of
test_gpu_visibility.py (1e-6 in relative l2 norm, the requested precision of
the reference's transform)."""
import math

import numpy as np
import pytest

from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W
from vis_oracle import direct_sum, pixel_centres

pytestmark = pytest.mark.gpu

MAS_TO_RAD = 4.84813681109536e-09


@pytest.mark.parametrize("rows", [1504, 1506, 1536, 1538, 3072, 3074, 12290])
def test_row_counts(ctx, rows):
    mas = 4.0 / rows
    lg = math.log10(mas * 1.8443 * J.pc)
    plane, nu = J.ImagePlane((rows, 9), lg, math.log10(0.4 * 1.8443 * J.pc), 0.1), np.array([15.4e9 * 1.1])
    jet = W.conical_model()
    p = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_I_KW)
    img, _ = ctx.render(jet.desc(), plane.desc(), nu, p)
    assert (img["I"] > 0).any()
    rad_per_cm = MAS_TO_RAD / (1.8443 * J.pc)
    jy = 1e23 / (1 + W.Z) ** 3 * rad_per_cm ** 2
    uv = np.random.default_rng(rows).uniform(-3e8, 3e8, (40, 2))
    vis, _ = ctx.visibilities(jet.desc(), plane.desc(), nu, p, uv, rad_per_cm, jy)
    sizes = ctx.plane_sizes(plane.desc()).reshape(plane.image_size)[0]
    across, along = pixel_centres(sizes, rows)
    ref = direct_sum(img["I"][0] * sizes[None, :] ** 2 * jy, across, along, uv, rad_per_cm, 0.0, 0.0, 0.0)
    assert np.linalg.norm(vis[0] - ref) / np.linalg.norm(ref) < 1e-6
