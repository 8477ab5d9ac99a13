"""Performance cases of the renderer: the calls a user's program makes, over
the range of sizes, outputs, precisions and field laws that it makes them in.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare(case, seed)`` builds what the program holds before the call
(jet, image plane, frequencies, parameters, output planes; the context, an
uploaded grid and the serving loop are made once per process, as a program
keeps them), ``run(state)`` is one call, ``work(case)`` the bytes and flops
it cannot do without and ``exact(case, seed)`` the same outputs from plain
torch arithmetic in 64 bits.
"""
import math

import numpy as np
import torch

PC = 3.0856775814671913e18          # cm, the constant of the reference
MAS_TO_RAD = 4.84813681109536e-09
PC_PER_MAS = 1.844325               # z = 0.1, flat cosmology (H0 = 70, Om = 0.3)
Z = 0.1
PLANES = ("tau", "l", "I", "Q", "U", "V")
# the accuracy-qualified tolerances of the mixed-precision renders
TOL = dict(n=100, tau_max=1e4, tau_min=1e-10, tau_atol=1e-20, tau_rtol=5e-8, atol=1e-24)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a model-fitting loop's smallest render: one frequency, Stokes I,
        # planes left on the device; latency and launches count
        dict(name="i_64x64", call="device", jet="conical", precision="mixed", output="I", across=64, along=64,
             mas0=0.2, mas1=0.2, n_nu=1),
        # the 128 x 128 uniform image at 15.4 GHz with full Stokes
        dict(name="iquv_128x128", call="device", jet="conical", precision="mixed", output="full", across=128,
             along=128, mas0=0.1, mas1=0.1, n_nu=1),
        # an odd, ragged image of the log-spaced plane at three frequencies
        dict(name="iquv_log_102x333", call="device", jet="conical", precision="mixed", output="full", across=102,
             along=333, mas0=0.01, mas1=0.1, n_nu=3),
        # the headline render: 512 x 1024 log-spaced pixels, 4 frequencies
        dict(name="iquv_log_512x1024", call="device", jet="conical", precision="mixed", output="full", across=512,
             along=1024, mas0=0.001, mas1=0.1, n_nu=4),
        # visibilities of a Stokes I model at the points of an observation:
        # the image stays on the device, n_uv complex numbers come back
        dict(name="vis_200x300", call="visibilities", jet="conical", precision="mixed", output="I", across=200,
             along=300, mas0=0.02, mas1=0.1, n_nu=2, n_uv=5000),
        # field laws outside the log-domain family: radial outflow, radial
        # field, density on |z|
        dict(name="laws_128x192", call="device", jet="radial", precision="mixed", output="full", across=128,
             along=192, mas0=0.05, mas1=0.1, n_nu=2),
        # the parabolic-to-conical jet whose core is Faraday thick
        dict(name="parabolic_512x512", call="device", jet="parabolic", precision="mixed", output="full", across=512,
             along=512, mas0=0.04, mas1=0.04, n_nu=2),
        # a jet read from a simulation's (z, r) grid of 200 000 points
        dict(name="grid_256x256", call="device", jet="grid", precision="mixed", output="full", across=256, along=256,
             mas0=0.001, mas1=0.001, n_nu=1),
        # the same arithmetic as the reference: FP64 throughout, full Stokes
        dict(name="fp64_64x96", call="device", jet="conical", precision="fp64", output="full", across=64, along=96,
             mas0=0.15, mas1=0.15, n_nu=1),
        # the reference's Python binding: get_i_image, images on the host
        dict(name="binding_60x90", call="binding", jet="tangled", precision="fp64", output="I", across=60, along=90,
             mas0=0.05, mas1=0.2, n_nu=1),
        # the stripe pass of the reference's image-size search
        dict(name="stripe_1000", call="stripe", jet="conical", precision="fp64", output="I", across=16, along=2000,
             mas0=0.01, mas1=0.1, n_nu=1),
        # a burst of requests of mixed shapes through the serving loop
        dict(name="serve_8", call="serve", jet="mixed", precision="mixed", output="full", across=128, along=128,
             mas0=0.1, mas1=0.1, n_nu=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "iquv", "i", "visibilities", "laws", "parabolic", "grid", "fp64", "binding", "stripe",
                       "serve"])
    across = 2 * _log_int(rng, 16, 200)   # the plane takes an even number of rows
    along = _log_int(rng, 40, 700)
    mas0 = round(10 ** rng.uniform(-2, -1), 4)
    case = dict(call="device", jet="conical", precision="mixed", output="full", across=across, along=along, mas0=mas0,
                mas1=0.1, n_nu=rng.randint(1, 4))
    if kind == "small":
        case.update(output=rng.choice(["I", "full"]), across=2 * rng.randint(8, 48), along=rng.randint(16, 96),
                    mas0=0.15, mas1=0.15, n_nu=1)
    elif kind == "i":
        case.update(output="I")
    elif kind == "visibilities":
        case.update(call="visibilities", output="I", across=2 * _log_int(rng, 16, 128), along=_log_int(rng, 32, 300),
                    n_uv=_log_int(rng, 100, 8000), n_nu=rng.randint(1, 2))
    elif kind == "laws":
        case.update(jet=rng.choice(["radial", "sheath", "tangled"]), across=2 * rng.randint(20, 64),
                    along=rng.randint(40, 192), mas0=0.05, n_nu=rng.randint(1, 2))
    elif kind == "parabolic":
        case.update(jet="parabolic", across=2 * rng.randint(48, 256), along=rng.randint(96, 512), mas0=0.04,
                    mas1=0.04, n_nu=rng.randint(1, 2))
    elif kind == "grid":
        case.update(jet="grid", across=2 * rng.randint(24, 128), along=rng.randint(48, 256), mas0=0.001, mas1=0.001,
                    n_nu=1)
    elif kind == "fp64":
        case.update(precision="fp64", across=2 * rng.randint(10, 40), along=rng.randint(20, 80), mas0=0.15, mas1=0.15,
                    n_nu=1, output=rng.choice(["I", "full"]))
    elif kind == "binding":
        case.update(call="binding", jet="tangled", precision="fp64", output="I", across=2 * rng.randint(8, 36),
                    along=rng.randint(16, 100), mas0=0.05, mas1=0.2, n_nu=1)
    elif kind == "stripe":
        case.update(call="stripe", precision="fp64", output="I", across=16, along=_log_int(rng, 64, 3000), n_nu=1)
    elif kind == "serve":
        case.update(call="serve", jet="mixed", across=2 * rng.randint(24, 64), along=rng.randint(48, 128), mas0=0.1,
                    n_nu=rng.randint(1, 4))
    return case


# ------------------------------------------------------- inputs of a seed
def _parameters(case, seed):
    """What the seed draws: the jet's numbers (priors of a model fit around
    the benchmark jets), the source-frame frequencies and the (u, v) points."""
    rng = np.random.default_rng([seed, 20])
    v = dict(half=0.05 * rng.uniform(0.9, 1.1), los=0.1 * rng.uniform(0.97, 1.1), b0=0.1 * rng.uniform(0.8, 1.25),
             n0=500.0 * rng.uniform(0.8, 1.25), gamma=rng.uniform(8.0, 12.0), pitch=math.pi / 4)
    nu0 = {1: [15.4], 2: [5.0, 15.4], 3: [8.1, 12.1, 15.4], 4: [8.1, 8.4, 12.1, 15.4]}[case["n_nu"]]
    v["nu"] = np.asarray(nu0) * 1e9 * (1 + Z) * rng.uniform(0.98, 1.02)
    if case["jet"] == "grid":   # the grid covers a 0.05 rad cone up to z = 20 pc
        v["half"] = 0.05 * rng.uniform(0.97, 1.0)
    if case["jet"] == "parabolic":
        v.update(los=0.05 * rng.uniform(0.97, 1.03), b0=1.0 * rng.uniform(0.9, 1.1), r0=0.1 * rng.uniform(0.97, 1.03))
    if case["jet"] == "tangled":
        v.update(b0=0.3 * rng.uniform(0.8, 1.25))
    if case["call"] == "visibilities":
        r, t = 3e8 * np.sqrt(rng.random(case["n_uv"])), rng.uniform(0, 2 * np.pi, case["n_uv"])
        v["uv"] = np.column_stack([r * np.cos(t), r * np.sin(t)])
        v.update(dx=0.1 * MAS_TO_RAD, dy=-0.05 * MAS_TO_RAD, rot=rng.uniform(-0.5, 0.5))
    return v


_kept = {}


def _once(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _upload_grid():
    from jetshow_gb300 import workloads as W
    from jetshow_gb300.runtime import default_context, triangulate
    xy, values = W.simulation_grid_c3()
    return default_context().grid_upload(xy, values, triangulate(xy))


def _jet(case, v):
    from jetshow_gb300 import jet as J
    cone = J.Cone((0, 0, 0), (0, 0, 1), v["half"], 100.0 * PC)
    helical = J.HelicalConicalBField(v["b0"], 1.0, v["pitch"], True)
    kind = case["jet"]
    if kind == "conical":
        return J.Jet(cone, J.ConstFlatVField(v["gamma"]), helical, J.BKNField(v["n0"], 2.0, True), s=2.5,
                     gamma_min=10.0)
    if kind == "radial":
        return J.Jet(cone, J.ConstCentralVField(v["gamma"]), J.RadialConicalBField(v["b0"], 1.0, True),
                     J.BKNFieldZ(v["n0"], 2.0, True), s=2.5, gamma_min=10.0)
    if kind == "sheath":
        return J.Jet(cone, J.SheathFlatVField(v["gamma"], 3.0, 0.5 * PC),
                     J.HelicalConicalBField(v["b0"], 1.0, v["pitch"], False), J.BKNField(v["n0"], 2.0, False), s=2.5,
                     gamma_min=10.0)
    if kind == "tangled":
        return J.Jet(cone, J.ConstFlatVField(v["gamma"]), J.RandomScalarBFieldZ(v["b0"], 1.0),
                     J.BKNFieldZ(v["n0"], 2.0, True), s=3.42)
    if kind == "parabolic":
        geometry = J.ParabaloidCone((0, 0, 0), (0, 0, 1), v["r0"] * PC, 1.0 * PC, 100.0 * PC)
        return J.Jet(geometry, J.ConstFlatVField(v["gamma"]), helical, J.BKNField(v["n0"], 2.0, True), s=2.5,
                     gamma_min=10.0, thermal_fraction=0.1)
    g = _once("grid", _upload_grid)
    return J.Jet(cone, J.SimulationVField(g, 3), J.SimulationBField(g, 0, 1, True), J.SimulationNField(g, 2, True),
                 s=2.5, gamma_min=10.0)


def _lg_cm(mas):
    return math.log10(mas * PC_PER_MAS * PC)


def _burst(case, seed):
    """The requests of a burst: images from a quarter of the case's size up,
    1 .. n_nu frequencies, every other jet parabolic-to-conical."""
    from jetshow_gb300 import jet as J
    rng = np.random.default_rng([seed, 21])
    requests = []
    for k in range(8):
        f = 0.25 + 0.75 * k / 7
        across, along = 2 * max(8, int(f * case["across"] / 2)), max(16, int(f * case["along"]))
        one = dict(case, jet="parabolic" if k % 2 else "conical", n_nu=1 + k % case["n_nu"])
        v = _parameters(one, int(rng.integers(1 << 30)))
        v.update(b0=v["b0"] * (0.1 if k % 2 else 1.0), los=0.1 * rng.uniform(1.0, 2.0))
        mas = case["mas0"] * case["across"] / across
        plane = J.ImagePlane((across, along), _lg_cm(mas), _lg_cm(mas), v["los"])
        requests.append((_jet(one, v).desc(), plane.desc(), v["nu"], _params(one)))
    return requests


def _server():
    from jetshow_gb300.serving import Server
    return Server(max_inflight_batches=3, max_batch_requests=16, hbm_budget_bytes=4 << 30)


def _params(case):
    from jetshow_gb300 import _capi as A
    from jetshow_gb300 import jet as J
    mixed = case["precision"] == "mixed"
    return J.make_params(**TOL, rtol=1e-7 if mixed and case["output"] == "I" else 1e-6, precision=case["precision"],
                         schedule="persistent" if mixed else "static", output=case["output"],
                         flags=A.FLAG_FARADAY_THICK if case["jet"] == "parabolic" else 0)


def prepare(case, seed):
    from jetshow_gb300 import jet as J
    from jetshow_gb300.runtime import default_context
    v = _parameters(case, seed)
    state = {"call": case["call"], "ctx": default_context(), "v": v, "params": _params(case)}
    if case["call"] == "serve":
        return dict(state, server=_once("server", _server), requests=_burst(case, seed))
    if case["call"] == "binding":
        state["args"] = (v["los"], Z, case["along"], case["across"], case["mas0"], case["mas1"], v["half"], v["b0"],
                         1.0, v["n0"], 2.0, v["gamma"], float(v["nu"][0]) / 1e9 / (1 + Z))
        return state
    plane = J.ImagePlane((case["across"], case["along"]), _lg_cm(case["mas0"]), _lg_cm(case["mas1"]), v["los"])
    jet = _jet(case, v)
    if case["call"] == "stripe":
        return dict(state, observation=J.Observation(jet, plane, v["nu"]))
    state.update(model=jet.desc(), plane=plane.desc(), nu=v["nu"])
    if case["call"] == "device":
        shape = (case["n_nu"], case["across"], case["along"])
        out = {k: torch.empty(shape, dtype=torch.float64, device="cuda") for k in PLANES}
        out["status"] = torch.empty(shape, dtype=torch.int32, device="cuda")
        state.update(out=out, pointers={k: t.data_ptr() for k, t in out.items()})
    return state


def _jy_factor():
    return 1e23 / (1 + Z) ** 3 * (MAS_TO_RAD / (PC_PER_MAS * PC)) ** 2


def run(state):
    call, ctx = state["call"], state["ctx"]
    if call == "device":
        ctx.render_device(state["model"], state["plane"], state["nu"], state["params"],
                          torch.cuda.current_stream().cuda_stream, state["pointers"])
        return state["out"]
    if call == "visibilities":
        v = state["v"]
        vis, _ = ctx.visibilities(state["model"], state["plane"], state["nu"], state["params"], v["uv"],
                                  MAS_TO_RAD / (PC_PER_MAS * PC), _jy_factor(), v["dx"], v["dy"], v["rot"])
        return vis
    if call == "binding":
        from jetshow_gb300.pyjetshow import get_i_image
        tau, image = get_i_image(*state["args"])
        return {"tau": tau, "I": image}
    if call == "stripe":
        return state["observation"].run_stripe(100, TOL["tau_max"]).getStripe("tau")
    server = state["server"]
    ids = [server.submit(model, plane, nu, params) for model, plane, nu, params in state["requests"]]
    return [server.wait(i)[0] for i in ids]


def work(case):
    """Outputs written once (the inputs are a few hundred bytes, but for the
    (u, v) points), and the arithmetic of the pixels that hit the jet (about
    0.57 of a plane): a ray's optical depth from some 60 evaluations of the
    absorption coefficient (34 multiply-adds each) and its Stokes vector from
    some 100 evaluations of the transfer equation (116; 50 for I alone)."""
    values = case["across"] * case["along"] * case["n_nu"]
    if case["call"] == "stripe":
        n = case["along"] - case["along"] // 2
        return {"bytes": 8.0 * n, "flops": n * 201.0 * 68}
    if case["call"] == "serve":
        values = 8 * values * 0.43 * (case["n_nu"] + 1) / (2 * case["n_nu"])
    bytes_ = values * 52.0
    flops = 0.57 * values * (60 * 68 + 100 * (232 if case["output"] == "full" else 100))
    if case["call"] == "binding":
        bytes_ = values * 16.0
    if case["call"] == "visibilities":
        bytes_ = 32.0 * case["n_uv"] * case["n_nu"]
        flops += 4.0 * 0.57 * values * case["n_uv"]
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------ 64-bit references
M_E, Q_E, C = 9.10938356e-28, 4.80320467299766e-10, 29979245800.0


def _coefficients(kind, v, p, nl, nu):
    """Lab-frame k_I, k_Q, k_V, k_F, k_C [1/pc] and eta_I, eta_Q, eta_V [per
    pc] at points p [..., 3] in pc: the uniform-pitch-angle power-law
    synchrotron formulas in the plasma frame, k = k'/D, eta = eta' D^2."""
    s, g = (3.42, 100.0) if kind == "tangled" else (2.5, 10.0)
    G = math.gamma
    gamma = v["gamma"]
    b = math.sqrt(1 - 1 / gamma ** 2)
    r, z = p.norm(dim=-1), p[..., 2]
    if kind == "radial":
        beta = b * p / r[..., None]
        n = v["n0"] * z.abs() ** -2.0
    else:
        beta = torch.zeros_like(p)
        beta[..., 2] = b
        n = v["n0"] * (z.abs() if kind == "tangled" else r) ** -2.0
    D = 1 / (gamma * (1 - (beta * nl).sum(-1)))
    nlp = nl * D[..., None] - beta * ((D + 1) * (gamma / (gamma + 1)))[..., None]
    nup = nu / D
    plasma2 = n * Q_E ** 2 / (math.pi * M_E)
    per_gauss = Q_E / (2 * math.pi * M_E * C)
    ki0 = 3 ** ((s + 1) / 2) / 4 * G(s / 4 + 11 / 6) * G(s / 4 + 1 / 6)
    ei0 = 3 ** (s / 2) / (2 * (s + 1)) * G(s / 4 + 19 / 12) * G(s / 4 - 1 / 12)
    if kind == "tangled":
        bperp = v["b0"] * z.abs() ** -1.0
        ki0 *= math.sqrt(math.pi / 4) * G((6 + s) / 4) / G((8 + s) / 4)
        ei0 *= math.sqrt(math.pi / 4) * G((5 + s) / 4) / G((7 + s) / 4)
    else:
        if kind == "radial":
            field = v["b0"] * p / (r ** 2)[..., None]
        else:
            rc = (p[..., 0] ** 2 + p[..., 1] ** 2).sqrt()
            sp, cp = math.sin(v["pitch"]), math.cos(v["pitch"])
            field = (v["b0"] / r)[..., None] * torch.stack([-sp * p[..., 1] / rc, sp * p[..., 0] / rc,
                                                            torch.full_like(rc, cp)], -1)
        bperp = torch.linalg.cross(nlp, field).norm(dim=-1)
    x = per_gauss * bperp / nup
    k0, e0 = math.pi * plasma2 * per_gauss * bperp / (C * nup ** 2), math.pi * plasma2 * per_gauss * bperp * M_E / C
    kI, eI = k0 * x ** (s / 2) * ki0 / D * PC, e0 * x ** ((s - 1) / 2) * ei0 * D * D * PC
    if kind == "tangled":
        o = torch.zeros_like(kI)
        return kI, o, o, o, o, eI, o, o
    bpar = (field * nlp).sum(-1)
    kv0 = 3 ** (s / 2) * (s + 3) * (s + 2) / (4 * (s + 1)) * G(s / 4 + 11 / 12) * G(s / 4 + 7 / 12)
    ev0 = 3 ** ((s - 1) / 2) * (s + 2) / (2 * s) * G(s / 4 + 2 / 3) * G(s / 4 + 1 / 3)
    par = math.pi * plasma2 * per_gauss * bpar
    kV = -par / (C * nup ** 2) * x ** ((s + 1) / 2) * kv0 / D * PC
    eV = -par * M_E / C * x ** (s / 2) * ev0 * D * D * PC
    kF = (s + 2) * math.log(g) / ((s + 1) * g ** (s + 1)) * 2 * par / (C * nup ** 2) / D * PC
    kC = -2 / (s - 2) * (g ** (2 - s) - x ** ((s - 2) / 2)) * math.pi * plasma2 * (per_gauss * bperp) ** 2 / (
        C * nup ** 3) / D * PC
    return kI, (s + 2) / (s + 10 / 3) * kI, kV, kF, kC, eI, (s + 1) / (s + 7 / 3) * eI, eV


class _Rays:
    """The rays of an image plane that hit the cone: the chord's near point
    [pc], direction away from the observer, chord length."""

    def __init__(self, v, sizes_cm, across):
        dev = torch.device("cuda")
        size = torch.tensor(sizes_cm / PC, dtype=torch.float64, device=dev)
        along = torch.cumsum(size, 0) - 0.5 * size
        k = (across - 1) / 2 - torch.arange(across, dtype=torch.float64, device=dev)
        y = k[:, None] * size[None, :]
        o = torch.stack([torch.zeros_like(y), y, (along / math.sin(v["los"])).expand_as(y)], -1).reshape(-1, 3)
        self.d = torch.tensor([-math.sin(v["los"]), 0.0, -math.cos(v["los"])], dtype=torch.float64, device=dev)
        c2 = math.cos(v["half"]) ** 2
        a = self.d[2] ** 2 - c2
        b = o[:, 2] * self.d[2] - c2 * (o @ self.d)
        c = o[:, 2] ** 2 - c2 * (o * o).sum(-1)
        disc = b * b - a * c
        self.n, self.hit = o.shape[0], torch.nonzero(disc > 0).squeeze(1)
        b, c, disc, o = b[self.hit], c[self.hit], disc[self.hit], o[self.hit]
        q = -b - torch.where(b > 0, 1.0, -1.0) * disc.sqrt()
        t = torch.stack([q / a, c / q], -1).sort(-1).values
        self.start, self.length = o + t[:, :1] * self.d, t[:, 1] - t[:, 0]

    def part(self, a, b):
        r = object.__new__(_Rays)
        r.d, r.start, r.length = self.d, self.start[a:b], self.length[a:b]
        return r

    def point(self, t):
        return self.start[:, None, :] + t[..., None] * self.d

    def stretched(self):
        """t(u), its inverse range and dt/du of t = tc + w sinh(u): fine about
        the closest approach to the jet axis, where the fields turn."""
        tc = (-self.start[:, 0] / self.d[0]).minimum(self.length).clamp(min=0.0)
        w = self.start[:, 1].abs().maximum(1e-6 * self.length)
        return tc, w, torch.asinh(-tc / w), torch.asinh((self.length - tc) / w)


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1), 0.5 * w


def _panels(rays, kind, v, nu, n_panels=96):
    """k_I, eta_I and weights dt at Gauss nodes of panels along each chord,
    and the optical depth between the observer and each node."""
    m = 8
    x, w = _gauss(m)
    # integrals of the Lagrange basis from 0 to each node (and to 1)
    basis = [np.polynomial.Polynomial(np.polynomial.polynomial.polyfit(x, row, m - 1)).integ() for row in np.eye(m)]
    to_node = torch.tensor(np.array([[q(t) - q(0.0) for q in basis] for t in x]), device=rays.d.device)
    x, w = (torch.tensor(a, device=rays.d.device) for a in (x, w))
    tc, sc, u0, u1 = rays.stretched()
    h = ((u1 - u0) / n_panels)[:, None, None]
    u = u0[:, None, None] + h * (torch.arange(n_panels, device=x.device)[None, :, None] + x)
    t = (tc[:, None, None] + sc[:, None, None] * torch.sinh(u)).flatten(1)
    dt = h * sc[:, None, None] * torch.cosh(u)
    co = _coefficients(kind, v, rays.point(t), -rays.d, nu)
    kI, eI = co[0].view_as(dt), co[5].view_as(dt)
    panel = (kI * dt * w).sum(-1)
    before = torch.cumsum(panel, 1) - panel
    return eI * dt * w, before[..., None] + (kI * dt) @ to_node.T, panel.sum(1), (u0, u1)


def _tau_and_i(rays, kind, v, nu):
    emitted, tau, total, _ = _panels(rays, kind, v, nu)
    return total, (emitted * torch.exp(-tau)).flatten(1).sum(1)


def _stokes(rays, kind, v, nu, steps=512):
    """I, Q, U, V at the observer: fourth-order Magnus steps of the linear
    system, from the far end, on a mesh even in u and in the optical depth
    in front (up to 40)."""
    _, tau, total, (u0, u1) = _panels(rays, kind, v, nu)
    tau = torch.cat([torch.zeros_like(total)[:, None], tau.flatten(1), total[:, None]], 1).clamp(max=40.0)
    x, _ = _gauss(8)
    g = torch.tensor((np.arange(96)[:, None] + x).ravel() / 96, device=tau.device)
    g = torch.cat([g.new_zeros(1), g, g.new_ones(1)])
    m = g + tau / 4.0
    want = m[:, -1:] * torch.linspace(0, 1, steps + 1, dtype=torch.float64, device=tau.device)
    k = torch.searchsorted(m, want.contiguous()).clamp(1, m.shape[1] - 1)
    m0, m1 = m.gather(1, k - 1), m.gather(1, k)
    f = g[k - 1] + (g[k] - g[k - 1]) * ((want - m0) / (m1 - m0)).clamp(0, 1)
    tc, sc, _, _ = rays.stretched()
    t = tc[:, None] + sc[:, None] * torch.sinh(u0[:, None] + (u1 - u0)[:, None] * f)
    scale = None
    state = torch.zeros(t.shape[0], 5, 1, dtype=torch.float64, device=t.device)
    state[:, 4] = 1.0
    c = math.sqrt(3) / 6
    for i in range(steps - 1, -1, -1):
        h = (t[:, i + 1] - t[:, i])[:, None, None]
        q = t[:, i + 1:i + 2] - (t[:, i + 1:i + 2] - t[:, i:i + 1]) * torch.tensor([0.5 - c, 0.5 + c],
                                                                                  dtype=t.dtype, device=t.device)
        kI, kQ, kV, kF, kC, eI, eQ, eV = _coefficients(kind, v, rays.point(q), -rays.d, nu)
        if scale is None:
            scale = float((eI / kI).max())
        a = torch.zeros(*kI.shape, 5, 5, dtype=t.dtype, device=t.device)
        for j in range(4):
            a[..., j, j] = -kI
        a[..., 0, 1] = a[..., 1, 0] = -kQ
        a[..., 0, 3] = a[..., 3, 0] = -kV
        a[..., 1, 2], a[..., 2, 1] = -kF, kF
        a[..., 2, 3], a[..., 3, 2] = -kC, kC
        a[..., 0, 4], a[..., 1, 4], a[..., 3, 4] = eI / scale, eQ / scale, eV / scale
        a1, a2 = a[:, 0], a[:, 1]
        omega = 0.5 * h * (a1 + a2) + math.sqrt(3) / 12 * h * h * (a2 @ a1 - a1 @ a2)
        state = torch.linalg.matrix_exp(omega) @ state
    return state[:, :4, 0].T * scale


def _mas_to_pc(z):
    """Parsecs per mas in the binding's default cosmology."""
    x, w = _gauss(32)
    om, ov, gnu = 0.2865, 0.7134130719051658, 8.69280948342326e-05
    f = ((om + (1 + z * x) * gnu) * (1 + z * x) ** 3 + ov) ** -0.5
    return MAS_TO_RAD * 299792.458 / 69.32 * 1e6 * z * float(f @ w) / (1 + z)


def _sizes(case, pc_per_mas):
    return np.geomspace(case["mas0"], case["mas1"], case["along"]) * pc_per_mas * PC


def _image(case, v, pc_per_mas, stokes):
    """tau, l, I (and Q, U, V) of the whole plane, [n_nu, across, along]."""
    rays = _Rays(v, _sizes(case, pc_per_mas), case["across"])
    shape = (len(v["nu"]), case["across"], case["along"])
    out = {k: torch.zeros(shape[0], rays.n, dtype=torch.float64, device="cuda") for k in PLANES}
    for f, nu in enumerate(v["nu"]):
        for a in range(0, rays.length.numel(), 8192):
            part, at = rays.part(a, a + 8192), rays.hit[a:a + 8192]
            tau, i = _tau_and_i(part, case["jet"], v, float(nu))
            out["tau"][f, at], out["l"][f, at] = tau, part.length * PC
            seen = torch.where(tau > TOL["tau_min"], 1.0, 0.0)
            if stokes:
                for k, x in zip("IQUV", _stokes(part, case["jet"], v, float(nu))):
                    out[k][f, at] = x * seen
            else:
                out["I"][f, at] = i * seen
    if float(out["tau"].max()) >= TOL["tau_max"]:
        out["tau"] = None  # such a ray keeps its depth at the end of the step that reached tau_max
    return {k: x if x is None else x.view(shape) for k, x in out.items()}


def exact(case, seed):
    """The outputs in plain 64-bit arithmetic.  None for the parabolic and
    gridded jets, the sheath's jump and the full-Stokes images of more than
    60 000 rays, which take longer than the render is worth, and for the
    stripe, whose rule takes its last step or not by the last bit of the
    chord's length (the reference's constant-step range)."""
    v = _parameters(case, seed)
    kind = case["jet"]
    if kind not in ("conical", "radial", "tangled") or case["call"] == "stripe":
        return None
    stokes = case["output"] == "full" and kind != "tangled"
    if stokes and case["across"] * case["along"] * case["n_nu"] > 105_000:
        return None
    if case["call"] == "binding":
        pcm = _mas_to_pc(Z)
        img = _image(case, v, pcm, False)
        omega = torch.tensor((_sizes(case, pcm) / (pcm * PC)) ** 2 * MAS_TO_RAD ** 2, device="cuda")
        return {"tau": None if img["tau"] is None else img["tau"][0],
                "I": img["I"][0] * 1e23 * omega / (1 + Z) ** 3}
    img = _image(case, v, PC_PER_MAS, stokes)
    if case["call"] == "visibilities":
        return _exact_visibilities(case, v, img["I"])
    return dict(img, status=None)


def _exact_visibilities(case, v, image):
    size = torch.tensor(_sizes(case, PC_PER_MAS), device="cuda")
    rad = MAS_TO_RAD / (PC_PER_MAS * PC)
    k = (case["across"] - 1) / 2 - torch.arange(case["across"], dtype=torch.float64, device="cuda")
    x = (-k[:, None] * size * rad).flatten()
    y = ((torch.cumsum(size, 0) - 0.5 * size) * rad).expand(case["across"], -1).flatten()
    uv = torch.tensor(v["uv"], device="cuda")
    c, s = math.cos(v["rot"]), math.sin(v["rot"])
    up, vp = uv[:, 0] * c + uv[:, 1] * s, -uv[:, 0] * s + uv[:, 1] * c
    flux = (image * size ** 2 * _jy_factor()).flatten(1)
    seen = torch.nonzero(flux.amax(0) > 0).squeeze(1)
    x, y, flux = x[seen], y[seen], flux[:, seen]
    out = torch.empty(flux.shape[0], uv.shape[0], dtype=torch.complex128, device="cuda")
    for a in range(0, uv.shape[0], 512):
        ph = torch.outer(x, up[a:a + 512]) + torch.outer(y, vp[a:a + 512])
        ph = 2 * math.pi * (ph - ph.round())
        out[:, a:a + 512] = torch.complex(flux @ torch.cos(ph), -(flux @ torch.sin(ph)))
    shift = -2 * math.pi * (uv[:, 0] * v["dx"] + uv[:, 1] * v["dy"])
    return (out * torch.polar(torch.ones_like(shift), shift)).cpu().numpy()

