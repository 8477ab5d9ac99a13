"""The autotuner does not settle on a slower shape than the context's present one:
renders of the fused family (whose kernels hold fewer registers than the
every-law ones) after the search against those before it, in turns, by the
best of twelve; 2.5 % is above the spread of such minima (below 1 %) and below
what a tuner costs that cannot reach the untuned shape (3 %).  A second search on
the same context starts from the first one's shape."""
import numpy as np
import pytest

from jetshow_gb300 import _capi as A
from jetshow_gb300 import jet as J
from jetshow_gb300 import workloads as W
from jetshow_gb300.runtime import Context

pytestmark = pytest.mark.gpu


def test_tuned_is_not_slower(ctx):
    torch = pytest.importorskip("torch")
    jet, plane, nu, _ = W.conical_c1()
    p = J.make_params(precision="mixed", schedule="persistent", **W.ACCURATE_KW)
    plain, tuned = Context(0), Context(0)
    for _ in range(2):
        t = tuned.autotune(jet.desc(), plane.desc(), nu, p)
        assert t["ctas_per_sm"] >= 1 and 1 <= t["refill_threshold"] <= 32 and t["ms"] > 0
    shape = (nu.size,) + tuple(plane.image_size)
    out = {k: torch.empty(shape, dtype=torch.float64, device="cuda") for k in ("tau", "l", "I", "Q", "U", "V")}
    out["status"] = torch.empty(shape, dtype=torch.int32, device="cuda")
    pointers = {k: v.data_ptr() for k, v in out.items()}
    stream = torch.cuda.current_stream()
    best = {plain: np.inf, tuned: np.inf}
    for k in range(13):
        for c in (plain, tuned):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            c.render_device(jet.desc(), plane.desc(), nu, p, stream.cuda_stream, pointers)
            b.record(stream)
            b.synchronize()
            if k:
                best[c] = min(best[c], a.elapsed_time(b))
    print("untuned, tuned ms:", best[plain], best[tuned], t)
    assert best[tuned] <= 1.025 * best[plain]
    plain.close()
    tuned.close()


@pytest.mark.parametrize("precision,flags", [("fp64", 0), ("mixed", A.FLAG_SINGLE_KERNEL), ("mixed", A.FLAG_FARADAY_THICK),
                                             ("mixed", A.FLAG_GENERAL_KERNELS)])
def test_every_kernel_kind(ctx, precision, flags):
    """The search asks for the occupancy of the kernels that the request runs."""
    c = Context(0)
    jet, plane, nu, _ = W.conical_c1(scale=32)
    p = J.make_params(precision=precision, schedule="persistent", flags=flags, **W.ACCURATE_KW)
    a, _ = ctx.render(jet.desc(), plane.desc(), nu, p)
    t = c.autotune(jet.desc(), plane.desc(), nu, p)
    assert t["block_size"] in (64, 96, 128, 192, 256) and 1 <= t["ctas_per_sm"] <= 32
    b, _ = c.render(jet.desc(), plane.desc(), nu, p)
    for k in a:
        assert np.array_equal(a[k], b[k], equal_nan=True), k
    c.close()
