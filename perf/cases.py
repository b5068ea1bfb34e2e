"""The work that users of this library have it do, as cases that can be timed and compared.

Every case is one call (or the few calls a time loop repeats) of the public binding `cb200`: whole
SSP-RK3 steps, the pieces of a step that a host solver calls one by one (`rhs`, `properties`),
batched closed blocks and batched 0-D reactors.  Inputs are smooth seeded fields built on the GPU;
ghost layers are filled with the periodic images, as a solver has them after its boundary call.
`exact` restates the same results in plain torch, FP64.
"""
import functools
import math
import os
import random
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(REPO, "corefl-cpc_b200"))

import cb200  # noqa: E402
from cb200 import abi, cases as examples, mech as mechanisms  # noqa: E402
from cb200.field import DeviceBlock, array_specs, box_faces, shape_of  # noqa: E402

F = torch.float64
R_U = 8314.462618
R_AIR = R_U / 28.9647
GAMMA = 1.4
SCHEMES = {"ausm": abi.INV_AUSMP, "hllc": abi.INV_HLLC, "char5": abi.INV_WENO5_CH, "char7": abi.INV_WENO7_CH}
RECS = {"muscl": abi.REC_MUSCL, "weno5": abi.REC_WENO5, "weno7": abi.REC_WENO7}


def listed():
    return [
        # the Sod tube of the reference's example at its size: a time loop of many tiny kernels
        {"name": "tube_1000", "kind": "tube", "n": 1000, "scheme": "char5", "steps": 40},
        # one step of a small block, where launches and latency count
        {"name": "air_step_33", "kind": "air_step", "mx": 33, "my": 33, "mz": 33, "scheme": "ausm", "rec": "weno7", "visc": 8},
        # the sine-wave workload of the benchmark at its full size
        {"name": "air_step_257", "kind": "air_step", "mx": 257, "my": 257, "mz": 257, "scheme": "ausm", "rec": "weno7", "visc": 8},
        # the same scheme's residual in the mixed-precision form, on a ragged block
        {"name": "air_rhs_mixed_161", "kind": "air_rhs", "mx": 161, "my": 129, "mz": 97, "scheme": "ausm", "rec": "weno7", "visc": 8, "mixed": True},
        # the reference's own default flux (characteristic WENO7) with 8th-order viscous terms
        {"name": "air_rhs_char7_129", "kind": "air_rhs", "mx": 129, "my": 113, "mz": 97, "scheme": "char7", "rec": "weno7", "visc": 8, "mixed": False},
        # the reacting H2/air box of the benchmark at its full size
        {"name": "h2_step_192", "kind": "h2_step", "mx": 192, "my": 192, "mz": 192, "scheme": "hllc", "rec": "weno5"},
        # the residual of a small reacting block with the reference's reconstruction, as a host solver calls it
        {"name": "h2_rhs_49", "kind": "h2_rhs", "mx": 49, "my": 41, "mz": 37, "scheme": "hllc", "rec": "muscl", "mixed": False},
        # the reacting residual in the mixed-precision form
        {"name": "h2_rhs_mixed_97", "kind": "h2_rhs", "mx": 97, "my": 97, "mz": 97, "scheme": "hllc", "rec": "weno5", "mixed": True},
        # the transport and thermodynamic properties alone, called after every change of the state
        {"name": "h2_properties_97", "kind": "h2_properties", "mx": 97, "my": 89, "mz": 81, "mixed": False},
        # steps of the two-temperature Mach-10 cylinder of the benchmark (four blocks, walls, inner faces)
        {"name": "cylinder_256x512", "kind": "cylinder", "side": 256, "normal": 512, "steps": 1},
        # a batch of 0-D ignition reactors, some step attempts of each
        {"name": "reactors_1024", "kind": "reactors", "n": 1024, "attempts": 24},
        # many closed blocks of uneven size advanced together
        {"name": "blocks_96", "kind": "blocks", "count": 96, "low": 12, "high": 40, "scheme": "ausm", "rec": "weno7", "steps": 2},
    ]


def _size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["tube", "air_step", "air_step", "air_rhs", "air_rhs", "h2_step", "h2_rhs", "h2_rhs",
                       "h2_properties", "cylinder", "reactors", "blocks"])
    box = {"mx": _size(rng, 24, 192), "my": _size(rng, 24, 160), "mz": _size(rng, 24, 128)}
    if kind == "tube":
        return {"kind": kind, "n": _size(rng, 200, 4000), "scheme": rng.choice(["char5", "char7"]), "steps": rng.randint(10, 60)}
    if kind == "air_step":
        return {"kind": kind, **box, "scheme": rng.choice(["ausm", "hllc"]), "rec": rng.choice(["weno5", "weno7"]), "visc": rng.choice([0, 8])}
    if kind == "air_rhs":
        scheme = rng.choice(["ausm", "hllc", "char5", "char7"])
        mixed = scheme in ("ausm", "hllc") and rng.random() < 0.6
        return {"kind": kind, **box, "scheme": scheme, "rec": rng.choice(["weno5", "weno7"]), "visc": rng.choice([0, 8]), "mixed": mixed}
    if kind == "h2_step":
        return {"kind": kind, **box, "scheme": rng.choice(["hllc", "ausm"]), "rec": rng.choice(["muscl", "weno5"])}
    if kind == "h2_rhs":
        mixed = rng.random() < 0.5
        return {"kind": kind, **box, "scheme": rng.choice(["hllc", "ausm"]), "rec": "weno5" if mixed else rng.choice(["muscl", "weno5"]), "mixed": mixed}
    if kind == "h2_properties":
        return {"kind": kind, **box, "mixed": rng.random() < 0.3}
    if kind == "cylinder":
        return {"kind": kind, "side": _size(rng, 64, 256), "normal": _size(rng, 96, 512), "steps": rng.randint(1, 3)}
    if kind == "reactors":
        return {"kind": kind, "n": _size(rng, 16, 8192), "attempts": rng.randint(8, 40)}
    return {"kind": kind, "count": _size(rng, 8, 200), "low": rng.randint(10, 16), "high": rng.randint(20, 40),
            "scheme": rng.choice(["ausm", "hllc"]), "rec": rng.choice(["weno5", "weno7"]), "steps": rng.randint(1, 3)}


# ---- mechanisms --------------------------------------------------------------------------------
@functools.lru_cache(None)
def h2_air():
    return mechanisms.load_json(os.path.join(REPO, "tests", "golden", "h2_li2004.json"))


@functools.lru_cache(None)
def air5():
    path = os.path.join(REPO, "tests", "golden", "air5_park.json")
    import json
    with open(path) as f:
        d = json.load(f)
    return mechanisms.MechStruct(d), mechanisms.TwoTemperatureStruct(d)


# ---- states ------------------------------------------------------------------------------------
def _waves(rng, grid, n=4, kmax=2):
    """A sum of n seeded periodic modes in [-1, 1] on the unit cube coordinates `grid`."""
    out = torch.zeros(torch.broadcast_shapes(*(q.shape for q in grid)), dtype=F, device=grid[0].device)
    for _ in range(n):
        k = [rng.randint(-kmax, kmax) for _ in range(3)]
        if not any(k):
            k[rng.randrange(3)] = 1
        a = sum(2 * math.pi * kk * q for kk, q in zip(k, grid)) + rng.uniform(0, 2 * math.pi)
        out = out + torch.sin(a) / n
    return out


def _grid(mx, my, mz, g, device):
    """Computational coordinates of the padded nodes on the unit cube; node m-1 is node 0's image."""
    q = [((torch.arange(-g, m + g, device=device, dtype=torch.int64) % (m - 1)).to(F) / (m - 1)) for m in (mx, my, mz)]
    return q[0][None, None, :], q[1][None, :, None], q[2][:, None, None]


def _zeros(specs, dims, device):
    return {n: torch.zeros(shape_of(*dims, nc, g), dtype=F, device=device) for n, (nc, g) in specs.items()}


def _curved_metric(t, dims, g, device, amp=0.05):
    """Exact metrics of x = X + a sin(2 pi Y) sin(2 pi Z) (cyclic), X, Y, Z in computational coordinates."""
    X, Y, Z = _grid(*dims, g, device)
    tp = 2 * math.pi
    s, c = torch.sin, torch.cos
    one = torch.ones((Z * Y * X).shape, dtype=F, device=device)
    rows = [[one, amp * tp * c(tp * Y) * s(tp * Z), amp * tp * s(tp * Y) * c(tp * Z)],
            [amp * tp * s(tp * Z) * c(tp * X), one, amp * tp * c(tp * Z) * s(tp * X)],
            [amp * tp * c(tp * X) * s(tp * Y), amp * tp * s(tp * X) * c(tp * Y), one]]
    J = [[rows[r][d] / (dims[d] - 1) for d in range(3)] for r in range(3)]  # d(x_r)/d(index_d)
    cof = [[J[(r + 1) % 3][(d + 1) % 3] * J[(r + 2) % 3][(d + 2) % 3] - J[(r + 1) % 3][(d + 2) % 3] * J[(r + 2) % 3][(d + 1) % 3]
            for d in range(3)] for r in range(3)]
    det = J[0][0] * cof[0][0] + J[0][1] * cof[0][1] + J[0][2] * cof[0][2]
    for d in range(3):
        for r in range(3):
            t["metric"][3 * d + r] = cof[r][d] / det
    t["jac"][0] = det.expand(t["jac"][0].shape)


def _air_state(t, dims, g, rng, device):
    grid = _grid(*dims, g, device)
    bv = t["bv"]
    bv[0] = 1.0 + 0.2 * _waves(rng, grid)
    for c in range(3):
        bv[1 + c] = rng.uniform(0.5, 1.0) + 0.3 * _waves(rng, grid)
    bv[4] = 1.0 + 0.1 * _waves(rng, grid)
    bv[5] = bv[4] / (bv[0] * R_AIR)
    _air_cv(t["bv"], t["cv"])


def _air_cv(bv, cv):
    cv[0] = bv[0]
    cv[1:4] = bv[0] * bv[1:4]
    cv[4] = 0.5 * (bv[1] ** 2 + bv[2] ** 2 + bv[3] ** 2) * bv[0] + bv[4] / (GAMMA - 1)


MU = 1e-4


def _air_param(case):
    mixed = abi.PREC_MIXED if case.get("mixed") else abi.PREC_FP64
    return examples.make_param(dim=3, inviscid_scheme=SCHEMES[case["scheme"]], reconstruction=RECS[case["rec"]],
                               viscous_order=case.get("visc", 0), cfl=0.5, rho_ref=1.0, v_ref=math.sqrt(3.0),
                               mu_constant=MU, precision=mixed)


def _air_block(case, seed, device, dims=None):
    dims = dims or (case["mx"], case["my"], case["mz"])
    g = 4
    t = _zeros(array_specs(*dims, g, 5, 0, viscous_order=case.get("visc", 0)), dims, device)
    t["mul"][0] = MU
    _curved_metric(t, dims, g, device)
    _air_state(t, dims, g, random.Random(seed), device)
    return t, dims, g


def _tube_state(case, seed, device):
    dims, g = (case["n"], 1, 1), 4 if case["scheme"] == "char7" else 3
    rng = random.Random(seed)
    t = _zeros(array_specs(*dims, g, 5, 0), dims, device)
    dx = 1.0 / (dims[0] - 1)
    x = torch.arange(-g, dims[0] + g, dtype=F, device=device) * dx
    left = x <= rng.uniform(0.4, 0.6)
    bv = t["bv"]
    ripple = 1 + 0.02 * torch.sin(2 * math.pi * (3 * x + rng.random()))
    bv[0] = torch.where(left, rng.uniform(0.9, 1.1), rng.uniform(0.1, 0.15)) * ripple
    bv[4] = torch.where(left, rng.uniform(0.9, 1.1), rng.uniform(0.08, 0.12)) * ripple
    bv[5] = bv[4] / (bv[0] * R_AIR)
    _air_cv(bv, t["cv"])
    t["metric"][0] = 1.0 / dx
    t["metric"][4] = t["metric"][8] = 1.0
    t["jac"][0] = dx
    return t, dims, g, dx


def _h2_composition(rng, grid, mech):
    """Premixed H2/air some way into its ignition: every species present, smooth in space."""
    ys = mechanisms.stoich_h2_air(mech)
    burnt = 0.3 + 0.2 * _waves(rng, grid)
    frac = {"H": 0.002, "O": 0.004, "OH": 0.01, "HO2": 2e-4, "H2O2": 5e-5}
    y = [torch.zeros_like(burnt) for _ in range(mech.ns)]
    for n in ("H2", "O2"):
        y[mech.index(n)] = float(ys[mech.index(n)]) * (1 - burnt)
    y[mech.index("N2")] = float(ys[mech.index("N2")]) * torch.ones_like(burnt)
    y[mech.index("H2O")] = float(ys[mech.index("H2")] + ys[mech.index("O2")]) * burnt
    for n, f in frac.items():
        y[mech.index(n)] = f * (1 + 0.5 * _waves(rng, grid))
    total = sum(y)
    return [v / total for v in y]


H2_SIDE, H2_DT = 1e-3, 2e-9


def _h2_block(case, seed, device):
    mech = h2_air()
    dims, g = (case["mx"], case["my"], case["mz"]), 3
    rng = random.Random(seed)
    specs = array_specs(*dims, g, 5 + mech.ns, mech.ns, viscous_order=2, reaction=True)
    t = _zeros(specs, dims, device)
    grid = _grid(*dims, g, device)
    bv, sv = t["bv"], t["sv"]
    for s, y in enumerate(_h2_composition(rng, grid, mech)):
        sv[s] = y
    for c in range(3):
        bv[1 + c] = 10.0 * _waves(rng, grid)
    bv[4] = 101325.0 * (1 + 0.05 * _waves(rng, grid))
    bv[5] = 1300.0 + 250.0 * _waves(rng, grid)
    bv[0] = bv[4] / (bv[5] * sum(sv[s] * (R_U / float(mech.mw[s])) for s in range(mech.ns)))
    for d, m in enumerate(dims):
        t["metric"][4 * d] = (m - 1) / H2_SIDE
    t["jac"][0] = math.prod(H2_SIDE / (m - 1) for m in dims)
    return t, dims, g, mech


def _h2_param(case, mech):
    mixed = abi.PREC_MIXED if case.get("mixed") else abi.PREC_FP64
    p = examples.make_param(n_var=5 + mech.ns, n_spec=mech.ns, dim=3, inviscid_scheme=SCHEMES[case.get("scheme", "hllc")],
                            reconstruction=RECS[case.get("rec", "weno5")], viscous_order=2, cfl=0.5, rho_ref=0.25, v_ref=750.0,
                            mech=mech.ptr(), precision=mixed)
    p.reaction = 1
    return p


def _h2_dt(case):
    # the benchmark's step, shortened on grids finer than its own
    return H2_DT * min(1.0, 191.0 / (max(case["mx"], case["my"], case["mz"]) - 1))


def _air_dt(case):
    return 0.1 / max(case["mx"], case["my"], case["mz"])


def _view(t, dims, g):
    v = abi.ZoneView(*dims, g)
    for n in abi.ZONE_ARRAYS:
        if n in t:
            setattr(v, n, t[n].data_ptr())
    return v


def _periodic(dims):
    return box_faces(*dims, {(d, s): abi.BC_PERIODIC for d in range(3) for s in (-1, 1)})


GROUPS = {"cv": (0, 1, 4, 5), "dq": (0, 1, 4, 5), "bv": (0, 1, 4, 5)}


def _parts(out):
    """The outputs by unit (mass, momentum or velocity, energy or pressure, the rest), so that a large
    one does not hide another's differences."""
    got = {}
    for name, a in out.items():
        base = name.rstrip("0123456789")
        if a is None or base not in GROUPS or a.dim() != 4:
            got[name] = a
            continue
        cuts = [c for c in GROUPS[base] if c < a.shape[0]] + [a.shape[0]]
        for c, e in zip(cuts[:-1], cuts[1:]):
            got["%s[%d:%d]" % (name, c, e)] = a[c:e]
    return got


class _State:
    """What a program keeps: its context, its arrays and the one call it repeats."""

    def __init__(self, call, out, *keep):
        self.call, self.out, self.keep = call, _parts(out), keep


def _bound(param, t, dims, g, faces):
    torch.cuda.synchronize()
    ctx = cb200.Context(param)
    ctx.bind(0, _view(t, dims, g), faces)
    return ctx


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed, torch.device("cuda"))


def run(state):
    state.call()
    return state.out


def _prepare_tube(case, seed, device):
    t, dims, g, _ = _tube_state(case, seed, device)
    p = examples.make_param(dim=2, inviscid_scheme=SCHEMES[case["scheme"]], cfl=0.5, rho_ref=1.0, v_ref=math.sqrt(GAMMA))
    faces = box_faces(*dims, {(d, s): abi.BC_OUTFLOW for d in range(2) for s in (-1, 1)})
    ctx = _bound(p, t, dims, g, faces)
    return _State(lambda: ctx.rk3_run(case["steps"]), {"cv": t["cv"], "bv": t["bv"]}, ctx, t)


def _prepare_air_step(case, seed, device):
    t, dims, g = _air_block(case, seed, device)
    ctx = _bound(_air_param(case), t, dims, g, _periodic(dims))
    dt = _air_dt(case)
    return _State(lambda: ctx.rk3_step(dt), {"cv": t["cv"], "bv": t["bv"]}, ctx, t)


def _prepare_air_rhs(case, seed, device):
    t, dims, g = _air_block(case, seed, device)
    ctx = _bound(_air_param(case), t, dims, g, _periodic(dims))
    return _State(lambda: ctx.rhs(0), {"dq": t["dq"]}, ctx, t)


def _prepare_h2_step(case, seed, device):
    t, dims, g, mech = _h2_block(case, seed, device)
    ctx = _bound(_h2_param(case, mech), t, dims, g, _periodic(dims))
    ctx.cv_from_bv(0)
    ctx.properties(0)
    dt = _h2_dt(case)
    return _State(lambda: ctx.rk3_step(dt), {n: t[n] for n in ("cv", "bv", "sv")}, ctx, t)


def _prepare_h2_rhs(case, seed, device):
    t, dims, g, mech = _h2_block(case, seed, device)
    ctx = _bound(_h2_param(case, mech), t, dims, g, _periodic(dims))
    ctx.cv_from_bv(0)
    ctx.properties(0)
    return _State(lambda: ctx.rhs(0), {n: t[n] for n in ("dq", "reaction_timeScale")}, ctx, t)


PROPERTIES = ("mul", "thermal_conductivity", "rho_D", "acoustic_speed", "gamma", "mach")


def _prepare_h2_properties(case, seed, device):
    t, dims, g, mech = _h2_block(case, seed, device)
    ctx = _bound(_h2_param(case, mech), t, dims, g, _periodic(dims))
    return _State(lambda: ctx.properties(0), {n: t[n] for n in PROPERTIES}, ctx, t)


@functools.lru_cache(2)
def _cylinder(side, normal):
    """The grid, metrics and faces (the same for every seed) of the AIR5 cylinder on the host."""
    mech, tt = air5()
    return examples.square_cylinder_air5(mech, tt, n_side=side, n_normal=normal)


def _prepare_cylinder(case, seed, device):
    c = _cylinder(case["side"], case["normal"])
    p = c.param
    p.positive_preserving = 1
    p.limit_flow = 1
    ctx = cb200.Context(p)
    rng = random.Random(seed)
    devs = []
    nb = len(c.blocks)
    for b, hb in enumerate(c.blocks):
        dev = DeviceBlock(hb, device=device)
        # the freestream with a seeded ripple of some per cent in density and temperature
        j = torch.arange(-hb.ngg, hb.my + hb.ngg, dtype=F, device=device)[None, :, None] / hb.my
        bv = dev.t["bv"]
        r = 1 + 0.03 * torch.sin(2 * math.pi * (2 * j + rng.random()))
        bv[0] /= r
        bv[5] *= r
        dev.t["temperature_ve"][0] = bv[5]
        ctx.bind(b, dev.view(), c.faces[b])
        devs.append(dev)
    for b in range(nb):
        ctx.bind_inner_faces(b, c.meta["inner"][b])
    # the initialisation of the benchmark's program
    for b in range(nb):
        ctx.properties(b)
    for b in range(nb):
        ctx.boundary(b)
    ctx.halo()
    for b in range(nb):
        ctx.properties(b)
    for b in range(nb):
        ctx.cv_from_bv(b)
    out = {"%s%d" % (n, b): dev.t[n] for b, dev in enumerate(devs) for n in ("cv", "bv", "sv", "temperature_ve")}
    return _State(lambda: ctx.rk3_run(case["steps"]), out, ctx, devs)


def _reactor_requests(case, seed, device):
    mech = h2_air()
    rng = np.random.default_rng(seed)
    n = case["n"]
    T0 = rng.uniform(1000.0, 1500.0, n)
    p0 = rng.uniform(1.0, 10.0, n) * 101325.0
    phi = rng.uniform(0.5, 2.0, n)
    x = np.zeros((n, mech.ns))
    x[:, mech.index("H2")] = 2 * phi
    x[:, mech.index("O2")] = 1.0
    x[:, mech.index("N2")] = 3.76
    for s in ("H", "O", "OH", "H2O"):  # some way into the induction time
        x[:, mech.index(s)] = 10.0 ** rng.uniform(-6, -2, n)
    y = x * mech.mw
    y /= y.sum(axis=1, keepdims=True)
    return mech, [torch.from_numpy(np.ascontiguousarray(a)).to(device) for a in (T0, p0, y, np.full(n, 1e-3))]


REACTOR_H0, RTOL, ATOL = 1e-8, 1e-6, 1e-12


def _prepare_reactors(case, seed, device):
    import ctypes
    mech, (T0, p0, y, t_end) = _reactor_requests(case, seed, device)
    p = examples.make_param(n_var=5 + mech.ns, n_spec=mech.ns, inviscid_scheme=abi.INV_HLLC, reconstruction=abi.REC_WENO5, mech=mech.ptr())
    torch.cuda.synchronize()
    ctx = cb200.Context(p)
    n = case["n"]
    buf = torch.zeros((n, ctypes.sizeof(abi.Reactor) // 8), dtype=F, device=device)

    def call():
        ctx.reactor_setup(buf.data_ptr(), n, T0.data_ptr(), p0.data_ptr(), y.data_ptr(), t_end.data_ptr(), h0=REACTOR_H0)
        ctx.reactor_advance(buf.data_ptr(), n, case["attempts"], rtol=RTOL, atol=ATOL)

    ns = abi.REACTOR_MAX_SPEC
    out = {"rhoY": buf[:, :ns], "rho_E_T_p": buf[:, ns:ns + 4], "time_h": buf[:, ns + 4:ns + 7:2], "error": buf[:, ns + 7],
           "counts": buf[:, ns + 8:].view(torch.int32)}
    return _State(call, out, ctx, buf, T0, p0, y, t_end)


def _block_sizes(case):
    # the same sizes for every seed: the work of a case does not depend on it
    rng = random.Random(case["count"] * 1000 + case["low"] * 50 + case["high"])
    return [rng.randint(case["low"], case["high"]) for _ in range(case["count"])]


def _prepare_blocks(case, seed, device):
    sizes = _block_sizes(case)
    total = sum((n + 8) ** 3 for n in sizes)
    state = torch.zeros((2, 6 * total), dtype=F, device=device)  # cv, bv of all blocks, one after another
    arr = (abi.BlockCase * len(sizes))()
    keep, at = [], 0
    for c, (q, n) in zip(arr, enumerate(sizes)):
        t, dims, g = _air_block(case, seed * 1009 + q, device, dims=(n, n, n))
        for r, name in enumerate(("cv", "bv")):
            nc, size = t[name].shape[0], t[name].numel()
            flat = state[r, 6 * at:6 * at + size].view(t[name].shape)
            flat.copy_(t[name])
            t[name] = flat
            assert nc <= 6
        at += (n + 8) ** 3
        c.zone = _view(t, dims, g)
        c.time, c.t_end, c.dt = 0.0, 1e30, 0.0
        keep.append(t)
    torch.cuda.synchronize()
    ctx = cb200.Context(_air_param(case))
    ctx.block_batch_set_schedule(8, 4)  # the schedule the tuner picks for such batches
    return _State(lambda: ctx.block_batch_advance(arr, case["steps"]), {"cv": state[0], "bv": state[1]}, ctx, keep, arr, state)


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    """Bytes: every input field read once, every output field written once.  Operations: the
    arithmetic of the schemes per node and stage (reconstructions, fluxes, stencils, rate and
    transport exponentials counted as about 20 operations each)."""
    kind = case["kind"]
    nodes = case["mx"] * case["my"] * case["mz"] if "mx" in case else 0
    air_sweep = {"weno7": 950, "weno5": 600, "muscl": 250}
    if kind == "tube":
        n = case["n"] * case["steps"]
        return {"bytes": 8 * (5 + 6 + 10 + 11) * case["n"], "flops": n * 3 * 1500}
    if kind in ("air_step", "air_rhs"):
        flux = 2000 if case["scheme"] == "char7" else 1300 if case["scheme"] == "char5" else air_sweep[case["rec"]]
        res = 3 * flux + (450 if case["visc"] == 8 else 0)
        if kind == "air_rhs":
            return {"bytes": 8 * nodes * ((6 + 10 + 5) / (2 if case["mixed"] else 1) + 5), "flops": nodes * res}
        return {"bytes": 8 * nodes * (5 + 6 + 10 + 1 + 11), "flops": nodes * 3 * (res + 60)}
    if kind.startswith("h2"):
        chemistry, transport, viscous = 1400, 2300, 3 * 400
        flux = 3 * (14 * {"weno5": 80, "muscl": 15}[case.get("rec", "weno5")] + 600)
        if kind == "h2_properties":
            return {"bytes": 8 * nodes * (6 + 9 + 14), "flops": nodes * transport}
        if kind == "h2_rhs":
            return {"bytes": 8 * nodes * (6 + 9 + 14 + 11 + 10 + 14), "flops": nodes * (chemistry + viscous + flux)}
        return {"bytes": 8 * nodes * (14 + 6 + 9 + 10 + 29 + 13), "flops": nodes * 3 * (chemistry + transport + viscous + flux + 300)}
    if kind == "cylinder":
        nodes = 4 * case["side"] * case["normal"]
        return {"bytes": 8 * nodes * (11 + 13 + 10 + 30), "flops": nodes * case["steps"] * 3 * 9000}
    if kind == "reactors":
        return {"bytes": 8 * case["n"] * 40, "flops": case["n"] * case["attempts"] * 6000}
    nodes = sum(n ** 3 for n in _block_sizes(case))
    return {"bytes": 8 * nodes * (5 + 6 + 10 + 1 + 11), "flops": nodes * case["steps"] * 3 * (3 * air_sweep[case["rec"]] + 60)}


def tolerance(case):
    """About four times the differences from `exact`, which sums in another order, measured over the
    listed sizes and the range that `draw` covers.  In FP64 a step differs by rounding, a residual by the rounding of
    the large fluxes whose difference it is, and the reactors by their step control, which raises an
    error norm (itself a small difference) to powers.  A temperature inversion that ends one step
    earlier or later moves single nodes by about 1e-10.  The mixed form's residuals are FP32."""
    kind = case["kind"]
    if case.get("mixed"):
        return {"rel": 1e-4, "max": 1e-2} if kind == "air_rhs" else {"rel": 6e-4, "max": 5e-2} if kind == "h2_rhs" else {"rel": 4e-6, "max": 4e-5}
    return {"tube": {"rel": 5e-14, "max": 1e-11}, "air_step": {"rel": 2e-15, "max": 1e-13}, "blocks": {"rel": 2e-15, "max": 1e-13},
            "air_rhs": {"rel": 4e-13, "max": 1e-10}, "h2_step": {"rel": 1e-13, "max": 1e-9}, "h2_rhs": {"rel": 2e-12, "max": 1e-10},
            "h2_properties": {"rel": 2e-15, "max": 2e-14}, "cylinder": {"rel": 1e-9, "max": 1e-6},
            "reactors": {"rel": 1e-8, "max": 1e-5, "differ": 0.005}}[kind]


# ---- the same results in plain torch, 64 bits --------------------------------------------------
def exact(case, seed):
    """None for the two-temperature cylinder: its model (two energy equations inverted per node,
    four blocks with inner faces) takes a plain torch statement minutes per step."""
    if case["kind"] == "cylinder":
        return None
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    got = globals()["_exact_" + case["kind"]](case, seed, device)
    return None if got is None else _parts(got)


def _sq(x):
    return x * x


def _weno_left(v, order, eps):
    """Left-biased value at the right face of the middle node of the stencil v (a list of shifts)."""
    if order == 5:
        q = [(2 * v[0] - 7 * v[1] + 11 * v[2]) / 6, (-v[1] + 5 * v[2] + 2 * v[3]) / 6, (2 * v[2] + 5 * v[3] - v[4]) / 6]
        b = [13 / 12 * _sq(v[0] - 2 * v[1] + v[2]) + 0.25 * _sq(v[0] - 4 * v[1] + 3 * v[2]),
             13 / 12 * _sq(v[1] - 2 * v[2] + v[3]) + 0.25 * _sq(v[1] - v[3]),
             13 / 12 * _sq(v[2] - 2 * v[3] + v[4]) + 0.25 * _sq(3 * v[2] - 4 * v[3] + v[4])]
        w = [0.1 / _sq(eps + b[0]), 0.6 / _sq(eps + b[1]), 0.3 / _sq(eps + b[2])]
    else:
        q = [(-3 * v[0] + 13 * v[1] - 23 * v[2] + 25 * v[3]) / 12, (v[1] - 5 * v[2] + 13 * v[3] + 3 * v[4]) / 12,
             (-v[2] + 7 * v[3] + 7 * v[4] - v[5]) / 12, (3 * v[3] + 13 * v[4] - 5 * v[5] + v[6]) / 12]
        d1 = [(-2 * v[0] + 9 * v[1] - 18 * v[2] + 11 * v[3]) / 6, (v[1] - 6 * v[2] + 3 * v[3] + 2 * v[4]) / 6,
              (-2 * v[2] - 3 * v[3] + 6 * v[4] - v[5]) / 6, (-11 * v[3] + 18 * v[4] - 9 * v[5] + 2 * v[6]) / 6]
        mid = v[2] - 2 * v[3] + v[4]
        d2 = [-v[0] + 4 * v[1] - 5 * v[2] + 2 * v[3], mid, mid, 2 * v[3] - 5 * v[4] + 4 * v[5] - v[6]]
        d3 = [-v[r] + 3 * v[r + 1] - 3 * v[r + 2] + v[r + 3] for r in range(4)]
        b = [a * a + 13 / 12 * c * c + 1043 / 960 * e * e + a * e / 12 for a, c, e in zip(d1, d2, d3)]
        tau = _sq(b[0] + 3 * b[1] - 3 * b[2] - b[3])
        w = [c * (1 + tau / _sq(eps + x)) for c, x in zip((1 / 35, 12 / 35, 18 / 35, 4 / 35), b)]
    return sum(a * c for a, c in zip(w, q)) / sum(w)


def _pair(v, rec, eps):
    """(left state at n+1/2, right state at n-1/2) from the stencil around node n."""
    if rec == "muscl":
        a, b = v[1] - v[0], v[2] - v[1]
        d = 0.25 * (torch.sign(a) + torch.sign(b)) * torch.minimum(a.abs(), b.abs())
        return v[1] + d, v[1] - d
    order = 5 if rec == "weno5" else 7
    return _weno_left(v, order, eps), _weno_left(v[::-1], order, eps)


def _lines(a, d, dims, g):
    """The padded array a [..., k, j, i] on the interior's cross-section, the sweep direction last."""
    axis = 2 - d
    sl = [slice(g, g + dims[2]), slice(g, g + dims[1]), slice(g, g + dims[0])]
    sl[axis] = slice(None)
    return a[(Ellipsis, *sl)].movedim(a.dim() - 3 + axis, -1)


def _back(a, d):
    return a.movedim(-1, a.dim() - 3 + 2 - d)


def _ausm(l, r, ml, mr, jl, jr):
    k = [0.5 * (jl * a + jr * b) for a, b in zip(ml, mr)]
    gk = torch.sqrt(sum(a * a for a in k))
    ul, ur = (sum(a * b for a, b in zip(k, s["q"][1:4])) / gk for s in (l, r))
    c = 0.5 * (torch.sqrt(l["gam"] * l["q"][4] / l["q"][0]) + torch.sqrt(r["gam"] * r["q"][4] / r["q"][0]))
    Ml, Mr = ul / c, ur / c
    al = 3 / 16
    sup_l, sup_r = Ml.abs() > 1, Mr.abs() > 1
    a, b = 0.25 * _sq(Ml + 1), _sq(Ml * Ml - 1)
    mlp = torch.where(sup_l, 0.5 * (Ml + Ml.abs()), a + 0.125 * b)
    plp = torch.where(sup_l, (Ml > 0).to(F), a * (2 - Ml) + al * Ml * b)
    a, b = 0.25 * _sq(Mr - 1), _sq(Mr * Mr - 1)
    mrn = torch.where(sup_r, 0.5 * (Mr - Mr.abs()), -a - 0.125 * b)
    prn = torch.where(sup_r, (Mr < 0).to(F), a * (2 + Mr) - al * Mr * b)
    pc = plp * l["q"][4] + prn * r["q"][4]
    mh = mlp + mrn
    flux = c * (l["q"][0] * 0.5 * (mh + mh.abs()) + r["q"][0] * 0.5 * (mh - mh.abs()))
    up = flux >= 0
    pick = lambda x, y: torch.where(up, x, y)  # noqa: E731
    co = flux * gk
    rho, p, E = pick(l["q"][0], r["q"][0]), pick(l["q"][4], r["q"][4]), pick(l["E"], r["E"])
    return [co] + [co * pick(l["q"][1 + a], r["q"][1 + a]) + pc * k[a] for a in range(3)] + [co * (E + p) / rho] + \
           [co * pick(x, y) for x, y in zip(l["q"][5:], r["q"][5:])]


def _hllc(l, r, ml, mr, jl, jr, gas):
    sl0, sr0 = torch.sqrt(l["q"][0]), torch.sqrt(r["q"][0])
    a, b = sl0 / (sl0 + sr0), sr0 / (sl0 + sr0)
    roe = [a * x + b * y for x, y in zip(l["q"], r["q"])]
    if gas is None:
        ht = a * (l["E"] + l["q"][4]) / l["q"][0] + b * (r["E"] + r["q"][4]) / r["q"][0]
        ct = torch.sqrt((GAMMA - 1) * (ht - 0.5 * (roe[1] ** 2 + roe[2] ** 2 + roe[3] ** 2)))
    else:
        rm = sum(y * float(c) for y, c in zip(roe[5:], gas.r))
        t = (a * l["q"][4] / l["q"][0] + b * r["q"][4] / r["q"][0]) / rm
        ct = gas.sound(t, roe[5:])[1]
    k = [0.5 * (x + y) for x, y in zip(ml, mr)]
    gk = torch.sqrt(sum(x * x for x in k))
    Ut = sum(x * y for x, y in zip(k, roe[1:4])) / gk
    ja = 0.5 * (jl + jr)
    U = [sum(x * y for x, y in zip(k, s["q"][1:4])) for s in (l, r)]
    cs = [torch.sqrt(s["gam"] * s["q"][4] / s["q"][0]) for s in (l, r)]
    sL = torch.minimum(U[0] / gk - cs[0], Ut - ct)
    sR = torch.maximum(U[1] / gk + cs[1], Ut + ct)
    (rl, pl), (rr, pr) = ((s["q"][0], s["q"][4]) for s in (l, r))
    ul, ur = U[0] / gk, U[1] / gk
    sm = (rr * ur * (sR - ur) - rl * ul * (sL - ul) + pl - pr) / (rr * (sR - ur) - rl * (sL - ul))
    pm = rl * (sL - ul) * (sm - ul) + pl

    def plain(s, Uk):
        rU = s["q"][0] * Uk
        return [ja * rU] + [ja * (rU * s["q"][1 + x] + s["q"][4] * k[x]) for x in range(3)] + \
               [ja * (s["E"] + s["q"][4]) * Uk] + [ja * rU * y for y in s["q"][5:]]

    def star(s, ss, Us):
        co = ja / (ss - sm)
        q = co * sm * (ss * gk - Us) * s["q"][0]
        dP = (ss * pm - sm * s["q"][4]) * co
        return [q] + [q * s["q"][1 + x] + dP * k[x] for x in range(3)] + \
               [q * s["E"] / s["q"][0] + co * (ss * pm * sm * gk - sm * s["q"][4] * Us)] + [q * y for y in s["q"][5:]]

    out = []
    for fl, fsl, fsr, fr in zip(plain(l, U[0]), star(l, sL, U[0]), star(r, sR, U[1]), plain(r, U[1])):
        out.append(torch.where(sL >= 0, fl, torch.where(sR < 0, fr, torch.where(sm >= 0, fsl, fsr))))
    return out


def _scales(case, nv):
    rho, v = (0.25, 750.0) if case["kind"].startswith("h2") else (1.0, math.sqrt(3.0))
    return [1e-40 * s * s for s in [rho, v, v, v, rho * v * v] + [1.0] * (nv - 5)]


def _primitive_flux(case, t, dims, g, dq, gas=None):
    """dq -= the differences of the primitive-reconstruction fluxes along the three directions."""
    names = 5 + (0 if gas is None else gas.ns)
    eps = _scales(case, names)
    h = {"muscl": 1, "weno5": 2, "weno7": 3}[case["rec"]]
    for d in range(3):
        m = dims[d]
        left, right = [], []
        for v in range(names):
            a = _lines(t["bv"][v] if v < 5 else t["sv"][v - 5], d, dims, g)
            st = [a[..., g - 1 + o:g - 1 + o + m + 2] for o in range(-h, h + 1)]  # nodes -1 .. m
            lp, rm = _pair(st, case["rec"], eps[v])
            left.append(lp[..., :-1])  # faces -1/2 .. m-1/2
            right.append(rm[..., 1:])
        states = []
        for q in (left, right):
            ek = 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
            if gas is None:
                states.append({"q": q, "E": ek * q[0] + q[4] / (GAMMA - 1), "gam": torch.tensor(GAMMA, dtype=F, device=ek.device)})
            else:
                tt = q[4] / (q[0] * sum(y * float(c) for y, c in zip(q[5:], gas.r)))
                gam, _, e = gas.sound(tt, q[5:])
                states.append({"q": q, "E": q[0] * (ek + e), "gam": gam})
        met = [_lines(t["metric"][3 * d + c], d, dims, g)[..., g - 1:g + m + 1] for c in range(3)]
        jac = _lines(t["jac"][0], d, dims, g)[..., g - 1:g + m + 1]
        args = (*states, [a[..., :-1] for a in met], [a[..., 1:] for a in met], jac[..., :-1], jac[..., 1:])
        flux = _ausm(*args) if case["scheme"] == "ausm" else _hllc(*args, gas)
        for v in range(names):
            dq[v] -= _back(flux[v][..., 1:] - flux[v][..., :-1], d)


def _characteristic_flux(order, t, dims, g, dq, eps, ndir=3):
    """dq -= the differences of the characteristic WENO fluxes of air (local Lax-Friedrichs splitting)."""
    R = order // 2 + 1
    for d in range(ndir):
        m = dims[d]
        met = [_lines(t["metric"][3 * d + c], d, dims, g) for c in range(3)]
        Q = [_lines(t["cv"][v], d, dims, g) for v in range(5)]
        p, T = _lines(t["bv"][4], d, dims, g), _lines(t["bv"][5], d, dims, g)
        J = _lines(t["jac"][0], d, dims, g)
        Uk = (Q[1] * met[0] + Q[2] * met[1] + Q[3] * met[2]) / Q[0]
        Fl = [Q[0] * Uk] + [Q[1 + c] * Uk + p * met[c] for c in range(3)] + [(Q[4] + p) * Uk]
        cg = torch.sqrt(sum(a * a for a in met)) * torch.sqrt(GAMMA * R_AIR * T)
        at = lambda a, o: a[..., g - 1 + o:g - 1 + o + m + 1]  # noqa: E731  (interfaces -1/2 .. m-1/2, offset o from the left node)
        # the face metric: averaged along the sweep for x, with the i+1 neighbour for y and z
        if d == 0:
            k = [0.5 * (at(a, 0) + at(a, 1)) for a in met]
        else:
            k = []
            for c in range(3):
                a = t["metric"][3 * d + c]
                k.append(0.5 * (at(_lines(a, d, dims, g), 0) + at(_lines(torch.roll(a, -1, -1), d, dims, g), 0)))
        rl, rr = at(Q[0], 0), at(Q[0], 1)
        s = torch.sqrt(rl * rr)
        a, b = 1 / (rl + s), 1 / (s + rr)
        u = [a * at(Q[1 + c], 0) + b * at(Q[1 + c], 1) for c in range(3)]
        c2 = GAMMA * (a * at(p, 0) + b * at(p, 1))
        cm = torch.sqrt(c2)
        gm1 = GAMMA - 1
        n = torch.sqrt(sum(x * x for x in k))
        k = [x / n for x in k]
        big = k[0].abs() > 0.8
        zero = torch.zeros_like(n)
        e = [torch.where(big, -k[2], zero), torch.where(big, zero, k[2]), torch.where(big, k[0], -k[1])]
        n = torch.sqrt(sum(x * x for x in e))
        e = [x / n for x in e]
        q = [k[1] * e[2] - k[2] * e[1], k[2] * e[0] - k[0] * e[2], k[0] * e[1] - k[1] * e[0]]
        dot = lambda x, y: sum(i * j for i, j in zip(x, y))  # noqa: E731
        Ub, Un, Uq, alf = dot(k, u), dot(e, u), dot(q, u), 0.5 * gm1 * dot(u, u)
        lam = functools.reduce(torch.maximum, [at(Uk, o).abs() + at(cg, o) for o in range(-R + 1, R + 1)])
        rows = []
        for sg in (1.0, -1.0):
            rows.append([0.5 * (alf + sg * Ub * cm) / c2] + [-0.5 * (gm1 * u[c] + sg * k[c] * cm) / c2 for c in range(3)] + [0.5 * gm1 / c2])
        L = [rows[0], [-Un, *e, zero], [-Uq, *q, zero], [1 - alf / c2] + [gm1 * u[c] / c2 for c in range(3)] + [-gm1 / c2], rows[1]]
        f = []
        for row in L:
            plus, minus = [], []
            for o in range(-R + 1, R + 1):
                LQ, LF = (sum(w * at(x, o) for w, x in zip(row, arr)) for arr in (Q, Fl))
                hj = 0.5 * at(J, o)
                plus.append(hj * (LF + lam * LQ))
                minus.append(hj * (LF - lam * LQ))
            f.append(_weno_left(plus[:-1], order, eps) + _weno_left(minus[:0:-1], order, eps))
        f034, f04 = f[0] + f[3] + f[4], f[0] - f[4]
        h = a * (at(Q[4], 0) + at(p, 0)) + b * (at(Q[4], 1) + at(p, 1))
        out = [f034] + [u[c] * f034 - k[c] * cm * f04 + e[c] * f[1] + q[c] * f[2] for c in range(3)] + \
              [h * f034 - Ub * cm * f04 + Un * f[1] + Uq * f[2] - c2 / gm1 * f[3]]
        for v in range(5):
            dq[v] -= _back(out[v][..., 1:] - out[v][..., :-1], d)


def _d8(a, d, dims, g):
    """8th-order central derivative along direction d on the interior nodes."""
    a = _lines(a, d, dims, g)
    m = dims[d]
    s = lambda o: a[..., g + o:g + o + m]  # noqa: E731
    return _back(0.8 * (s(1) - s(-1)) - 0.2 * (s(2) - s(-2)) + 4 / 105 * (s(3) - s(-3)) - 1 / 280 * (s(4) - s(-4)), d)


def _inner(a, dims, g):
    return a[..., g:g + dims[2], g:g + dims[1], g:g + dims[0]]


def _wrap(a, d, dims, g, ext):
    """Periodic faces of direction d: the end nodes averaged, then the ghosts copied, over the
    interior's cross-section (ext = 0) or with its ghosts (ext = g)."""
    axis, m = 2 - d, dims[d]
    sl = [slice(g - ext, g + dims[2 - x] + ext) for x in range(3)]

    def at(n):
        s = list(sl)
        s[axis] = g + n
        return (Ellipsis, *s)

    ave = 0.5 * (a[at(0)] + a[at(m - 1)])
    a[at(0)] = ave
    a[at(m - 1)] = ave
    for q in range(1, g + 1):
        a[at(-q)] = a[at(m - 1 - q)]
        a[at(m - 1 + q)] = a[at(q)]


def _stress(G, mu):
    (ux, uy, uz), (vx, vy, vz), (wx, wy, wz) = G
    xx, yy, zz = (mu * (4 * a - 2 * b - 2 * c) / 3 for a, b, c in ((ux, vy, wz), (vy, ux, wz), (wz, ux, vy)))
    xy, xz, yz = mu * (uy + vx), mu * (uz + wx), mu * (vz + wy)
    return [[xx, xy, xz], [xy, yy, yz], [xz, yz, zz]]


def _viscous8(t, dims, g, dq):
    met = [_inner(t["metric"][c], dims, g) for c in range(9)]
    grad = []
    for v in (1, 2, 3, 5):
        dd = [_d8(t["bv"][v], d, dims, g) for d in range(3)]
        grad.append([sum(dd[d] * met[3 * d + x] for d in range(3)) for x in range(3)])
    tau = _stress(grad[:3], MU)
    kap = MU / 0.72 * GAMMA * R_AIR / (GAMMA - 1)
    vel = [_inner(t["bv"][1 + c], dims, g) for c in range(3)]
    E = [sum(vel[c] * tau[c][x] for c in range(3)) + kap * grad[3][x] for x in range(3)]
    vec = [tau[0], tau[1], tau[2], E]
    jac = _inner(t["jac"][0], dims, g)
    # the exchange runs over x, then y, then z faces, averaging the end nodes of every flux array
    for v in range(4):
        full = []
        for d in range(3):
            f = torch.zeros_like(t["jac"][0])
            _inner(f, dims, g)[...] = sum(met[3 * d + x] * vec[v][x] for x in range(3))
            for a in range(3):
                _wrap(f, a, dims, g, 0)
            full.append(f)
        dq[1 + v] += jac * sum(_d8(full[d], d, dims, g) for d in range(3))


def _air_residual(case, t, dims, g):
    dq = torch.zeros((5, dims[2], dims[1], dims[0]), dtype=F, device=t["bv"].device)
    if case["visc"] == 8:
        _viscous8(t, dims, g, dq)
    if case["scheme"] in ("ausm", "hllc"):
        _primitive_flux(case, t, dims, g, dq)
    else:
        # (rho_ref v_ref)^2 scales the reference's eps
        _characteristic_flux(5 if case["scheme"] == "char5" else 7, t, dims, g, dq, 1e-40 * 3.0)
    return dq


def _exact_air_rhs(case, seed, device):
    t, dims, g = _air_block(case, seed, device)
    return {"dq": _air_residual(case, t, dims, g)}


STAGES = ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (1 / 3, 2 / 3, 2 / 3))


def _air_update(t, dims, g, qn, dq, dt, stage):
    a, b, c = stage
    q = a * qn + b * _inner(t["cv"], dims, g) + c * dt / _inner(t["jac"][0], dims, g) * dq
    bv = _inner(t["bv"], dims, g)
    _inner(t["cv"], dims, g)[...] = q
    bv[0] = q[0]
    bv[1:4] = q[1:4] / q[0]
    bv[4] = (GAMMA - 1) * (q[4] - 0.5 * q[0] * (bv[1] ** 2 + bv[2] ** 2 + bv[3] ** 2))
    bv[5] = bv[4] / (q[0] * R_AIR)


def _air_wrap(t, dims, g):
    for d in range(3):
        _wrap(t["bv"], d, dims, g, 0)
    # cv is rebuilt wherever the faces wrote
    cv = torch.empty_like(t["cv"])
    _air_cv(t["bv"], cv)
    touched = torch.zeros_like(cv[0], dtype=torch.bool)
    for axis, m in ((2, dims[0]), (1, dims[1]), (0, dims[2])):
        sl = [slice(g, g + dims[2]), slice(g, g + dims[1]), slice(g, g + dims[0])]
        for part in (slice(0, g + 1), slice(g + m - 1, None)):
            s = list(sl)
            s[axis] = part
            touched[tuple(s)] = True
    t["cv"][:] = torch.where(touched, cv, t["cv"])


def _air_rk3(case, t, dims, g, dt):
    qn = _inner(t["cv"], dims, g).clone()
    for stage in STAGES:
        _air_update(t, dims, g, qn, _air_residual(case, t, dims, g), dt, stage)
        _air_wrap(t, dims, g)


def _exact_air_step(case, seed, device):
    t, dims, g = _air_block(case, seed, device)
    _air_rk3(case, t, dims, g, _air_dt(case))
    return {"cv": t["cv"], "bv": t["bv"]}


def _cfl(t, dims, g, cfl, ndir=3):
    m, bv = _inner(t["metric"], dims, g), _inner(t["bv"], dims, g)
    a = torch.sqrt(GAMMA * R_AIR * bv[5])
    lam = [(bv[1] * m[3 * d] + bv[2] * m[3 * d + 1] + bv[3] * m[3 * d + 2]).abs() +
           a * torch.sqrt(m[3 * d] ** 2 + m[3 * d + 1] ** 2 + m[3 * d + 2] ** 2) for d in range(ndir)]
    return cfl / functools.reduce(torch.maximum, lam).max()


def _exact_blocks(case, seed, device):
    sizes = _block_sizes(case)
    if sum(n ** 3 for n in sizes) * case["steps"] > 12e6:
        return None  # thousands of small torch operations per block: minutes
    total = sum((n + 8) ** 3 for n in sizes)
    state, at = torch.zeros((2, 6 * total), dtype=F, device=device), 0
    inviscid = dict(case, visc=0)
    for q, n in enumerate(sizes):
        t, dims, g = _air_block(inviscid, seed * 1009 + q, device, dims=(n, n, n))
        for _ in range(case["steps"]):
            _air_rk3(inviscid, t, dims, g, _cfl(t, dims, g, 0.5))
        for r, name in enumerate(("cv", "bv")):
            state[r, 6 * at:6 * at + t[name].numel()] = t[name].reshape(-1)
        at += (n + 8) ** 3
    return {"cv": state[0], "bv": state[1]}


def _exact_tube(case, seed, device):
    device = torch.device("cpu")  # a thousand nodes
    t, dims, g, dx = _tube_state(case, seed, device)
    order = 5 if case["scheme"] == "char5" else 7

    def spread():
        """Ghosts of the outflow faces, then every k plane a copy of plane 0."""
        for name in ("bv", "cv"):
            a = t[name]
            row = a[:, g:g + 1, g:g + 1, :].clone()
            row[..., :g] = row[..., g:g + 1]
            row[..., -g:] = row[..., -g - 1:-g]
            mid = slice(g, -g)
            a[:, g, g, :] = row[:, 0, 0, :]  # x faces at j = 0
            a[:, g, :, mid] = row[:, 0, :, mid].expand(-1, a.shape[2], -1)  # y faces over the interior i
            a[:] = a[:, g:g + 1].clone().expand(a.shape)

    for _ in range(case["steps"]):
        dt = _cfl(t, dims, g, 0.5, 2)
        qn = _inner(t["cv"], dims, g).clone()
        for stage in STAGES:
            dq = torch.zeros((5, 1, 1, dims[0]), dtype=F, device=device)
            _characteristic_flux(order, t, dims, g, dq, 1e-40 * GAMMA, 1)
            _air_update(t, dims, g, qn, dq, dt, stage)
            _inner(t["cv"], dims, g)[3] = 0
            _inner(t["bv"], dims, g)[3] = 0
            spread()
    return {"cv": t["cv"], "bv": t["bv"]}


class _Gas:
    """NASA7 thermodynamics, mixture-averaged transport and the rates of a mechanism in torch."""

    def __init__(self, mech):
        d = mech.d
        self.d, self.ns, self.nr = d, mech.ns, mech.nr
        self.mw = np.asarray(d["mw"], dtype=np.float64)
        self.r = R_U / self.mw
        table = lambda n, *s: np.asarray(d[n], dtype=np.float64).reshape(*s)  # noqa: E731
        self.lo, self.hi = table("low_temp_coeff", self.ns, 7), table("high_temp_coeff", self.ns, 7)
        self.tl, self.tm, self.th = (table(n, self.ns) for n in ("t_low", "t_mid", "t_high"))

    def coeff(self, s, t):
        inside = t.clamp(float(self.tl[s]), float(self.th[s]))
        low = (t < float(self.tm[s])).to(F)
        return inside, [low * float(a) + (1 - low) * float(b) for a, b in zip(self.lo[s], self.hi[s])]

    def h_cp(self, s, t):
        tt, c = self.coeff(s, t)
        cp = c[0] + tt * (c[1] + tt * (c[2] + tt * (c[3] + tt * c[4])))
        h = tt * (c[0] + tt * (c[1] / 2 + tt * (c[2] / 3 + tt * (c[3] / 4 + tt * c[4] / 5)))) + c[5] + cp * (t - tt)
        return h * float(self.r[s]), cp * float(self.r[s])

    def gibbs(self, s, t):
        tt, c = self.coeff(s, t)
        return c[0] * (1 - torch.log(tt)) - tt * (c[1] / 2 + tt * (c[2] / 6 + tt * (c[3] / 12 + tt * c[4] / 20))) + c[5] / tt - c[6]

    def sound(self, t, y):
        te = t.clamp(min=1.0)
        e = r = cp = cv = 0
        for s in range(self.ns):
            h, c = self.h_cp(s, te)
            rs = float(self.r[s])
            e, r, cp, cv = e + y[s] * (h - rs * te), r + y[s] * rs, cp + y[s] * c, cv + y[s] * (c - rs)
        gam = cp / cv
        return gam, torch.sqrt(gam * r * te), e

    def temperature(self, e, y, r, t, tol, most):
        """Newton from t until the relative step is within tol, each node on its own."""
        live = torch.ones_like(t, dtype=torch.bool)
        for _ in range(most):
            h = cp = 0
            for s in range(self.ns):
                a, b = self.h_cp(s, t)
                h, cp = h + a * y[s], cp + b * y[s]
            t1 = t - (h - r * t - e) / (cp - r)
            step = (1 - t1 / t).abs()
            t = torch.where(live, t1, t)
            live = live & (step > tol)
            if not bool(live.any()):
                break
        return t

    def rates(self, t, c):
        """Forward and backward rates of progress per reaction, mol/(cm^3 s)."""
        d, ns = self.d, self.ns
        sf, sb = (np.asarray(d[n]).reshape(self.nr, ns) for n in ("stoi_f", "stoi_b"))
        third = np.asarray(d["third_body_coeff"], dtype=np.float64).reshape(self.nr, ns)
        g = [self.gibbs(s, t) for s in range(ns)]
        k = lambda r, x: float(d["A" + x][r]) * torch.exp(float(d["b" + x][r]) * torch.log(t) - float(d["Ea" + x][r]) / t)  # noqa: E731
        out = []
        for r in range(self.nr):
            ty, rev = int(d["reac_type"][r]), int(d["rev_type"][r])
            kf = k(r, "")
            cc = sum(float(w) * x for w, x in zip(third[r], c)) if ty > 3 else None
            if ty == 3:
                kf = kf + k(r, "2")
            elif ty == 4:
                kf = kf * cc
            elif ty > 4:
                low = k(r, "2")
                pr = low * cc / kf
                fall = 1.0
                if ty > 5:
                    al = float(d["troe_alpha"][r])
                    fc = (1 - al) * torch.exp(-t / float(d["troe_t3"][r])) + al * torch.exp(-t / float(d["troe_t1"][r]))
                    if ty == 7:
                        fc = fc + torch.exp(-float(d["troe_t2"][r]) / t)
                    lf = torch.log10(fc)
                    x = torch.log10(pr) - 0.4 - 0.67 * lf
                    fall = 10.0 ** (lf / (1 + _sq(x / (0.75 - 1.27 * lf - 0.14 * x))))
                kf = torch.where((kf < 1e-25) & (low < 1e-25), torch.zeros_like(kf), kf * pr / (1 + pr) * fall)
            kb = torch.zeros_like(kf)
            if ty != 0 and rev == 1:
                kb = k(r, "2") * (cc if ty == 4 else 1.0)
            elif ty not in (0, 2):
                dg = sum(g[s] * float(sb[r, s] - sf[r, s]) for s in range(ns) if sb[r, s] != sf[r, s])
                kb = kf / torch.exp(float(d["reac_order"][r]) * torch.log(101325.0 / R_U * 1e-3 / t) - dg)
            for s in range(ns):
                for _ in range(int(sf[r, s])):
                    kf = kf * c[s]
                for _ in range(int(sb[r, s])):
                    kb = kb * c[s]
            out.append((kf, kb))
        return out, sf, sb

    def source(self, t, rho_y):
        """omega_k in kg/(m^3 s), the destruction rate, and the rates of progress."""
        q, sf, sb = self.rates(t, [rho_y[s] / float(self.mw[s]) * 1e-3 for s in range(self.ns)])
        om, de = [], []
        for s in range(self.ns):
            cre = sum(b * float(sf[r, s]) + f * float(sb[r, s]) for r, (f, b) in enumerate(q) if sf[r, s] or sb[r, s])
            des = sum(f * float(sf[r, s]) + b * float(sb[r, s]) for r, (f, b) in enumerate(q) if sf[r, s] or sb[r, s])
            zero = torch.zeros_like(t)
            om.append((cre - des) * (1e3 * float(self.mw[s])) + zero)
            de.append(des * (1e3 * float(self.mw[s])) + zero)
        return om, de, q, sf, sb

    def transport(self, t, y, cp):
        d, ns = self.d, self.ns
        tab = lambda n, *s: np.asarray(d[n], dtype=np.float64).reshape(*s)  # noqa: E731
        kbe, bdc = tab("kb_over_eps_jk", ns, ns), tab("binary_diffusivity_coeff", ns, ns)
        w14, sq8 = tab("WjDivWi_to_One4th", ns, ns), tab("sqrt_WiDivWjPl1Mul8", ns, ns)
        lj, vc, geo, zr = (tab(n, ns) for n in ("LJ_potent_inv", "vis_coeff", "geometry", "ZRotF298"))
        omega = lambda x: 1.0548 * x ** -0.15504 + (x + 0.55909) ** -2.1705  # noqa: E731
        X = [y[s] / float(self.mw[s]) for s in range(ns)]
        total = sum(X)
        X = [x / total for x in X]
        vs = [float(vc[s]) * torch.sqrt(t) / (1.147 * (t * float(lj[s])) ** -0.145 + 1 / _sq(t * float(lj[s]) + 0.5)) for s in range(ns)]
        mu = kap = 0
        for a in range(ns):
            R = float(self.r[a])
            lam = 3.75 * vs[a] * R
            if geo[a] in (1, 2):
                tr = t * float(kbe[a, a])
                x = torch.sqrt(math.pi / tr) * math.pi
                FT = 1 + 0.5 * x + (2 + 0.25 * math.pi ** 2) / tr + x / tr
                rd = float(bdc[a, a]) * t ** 1.5 / (omega(tr) * R * t)
                lin = geo[a] == 1
                ab = (2.5 * vs[a] - rd) / (math.pi * float(zr[a]) / FT * vs[a] + (10 / 3 if lin else 5.0) * vs[a] + 2 * rd)
                lam = lam - (5 if lin else 7.5) * ab * vs[a] * R + rd * cp[a] + rd * ((2 if lin else 3) * ab - 2.5) * R
            den = X[a]
            for b in range(ns):
                if b != a:
                    den = den + _sq(1 + torch.sqrt(vs[a] / vs[b]) * float(w14[a, b])) * float(sq8[a, b]) * X[b]
            mu = mu + vs[a] * X[a] / den
            kap = kap + lam * X[a] / (1.065 * den - 0.065 * X[a])
        heavy = [(X[s] + 1e-12) * float(self.mw[s]) for s in range(ns)]
        both = sum(heavy)
        inv = [0] * ns
        for a in range(ns):
            for b in range(a + 1, ns):
                x = omega(t * float(kbe[a, b])) / (float(bdc[a, b]) * t ** 1.5)
                inv[a] = inv[a] + (X[b] + 1e-12) * x
                inv[b] = inv[b] + (X[a] + 1e-12) * x
        return mu, kap, [(both - heavy[s]) / (t * R_U * inv[s]) for s in range(ns)]


def _h2_cv(t, gas):
    bv, sv = t["bv"], t["sv"]
    E = 0.5 * (bv[1] ** 2 + bv[2] ** 2 + bv[3] ** 2)
    for s in range(gas.ns):
        E = E + gas.h_cp(s, bv[5])[0] * sv[s]
    return torch.cat([bv[:1], bv[0] * bv[1:4], (E * bv[0] - bv[4])[None], bv[0] * sv])


def _h2_properties(t, gas):
    bv, sv = t["bv"], t["sv"]
    T = bv[5]
    cp = [gas.h_cp(s, T)[1] for s in range(gas.ns)]
    cpm = sum(sv[s] * cp[s] for s in range(gas.ns))
    r = sum(sv[s] * float(gas.r[s]) for s in range(gas.ns))
    gam = cpm / (cpm - r)
    t["gamma"][0] = gam
    t["acoustic_speed"][0] = torch.sqrt(gam * r * T)
    t["mach"][0] = torch.sqrt(bv[1] ** 2 + bv[2] ** 2 + bv[3] ** 2) / t["acoustic_speed"][0]
    mu, kap, rd = gas.transport(T, sv, cp)
    t["mul"][0], t["thermal_conductivity"][0] = mu, kap
    for s in range(gas.ns):
        t["rho_D"][s] = rd[s]


def _exact_h2_properties(case, seed, device):
    t, dims, g, mech = _h2_block(case, seed, device)
    _h2_properties(t, _Gas(mech))
    return {n: t[n] for n in PROPERTIES}


def _viscous2(t, dims, g, dq, gas):
    """2nd-order face fluxes of a mixture and their differences."""
    ns = gas.ns
    for d in range(3):
        axis = 2 - d

        def at(a, off=(0, 0, 0)):
            """a on the left nodes of faces -1/2 .. m-1/2 (direction d), shifted by off = (di, dj, dk)."""
            sl = []
            for ax in range(3):
                m, o = dims[2 - ax], off[2 - ax]
                sl.append(slice(g - 1 + o, g + m + o) if ax == axis else slice(g + o, g + m + o))
            return a[(Ellipsis, *sl)]

        one = tuple(1 if x == d else 0 for x in range(3))
        mean = lambda a: 0.5 * (at(a) + at(a, one))  # noqa: E731
        met = [mean(t["metric"][c]) for c in range(9)]

        def grad(a):
            dd = []
            for x in range(3):
                if x == d:
                    dd.append(at(a, one) - at(a))
                else:
                    e = [0, 0, 0]
                    e[x] = 1
                    up, dn = tuple(e), tuple(-v for v in e)
                    both = lambda o: tuple(i + j for i, j in zip(o, one))  # noqa: E731
                    dd.append(0.25 * (at(a, up) - at(a, dn) + at(a, both(up)) - at(a, both(dn))))
            return [sum(dd[x] * met[3 * x + c] for x in range(3)) for c in range(3)]

        G = [grad(t["bv"][v]) for v in (1, 2, 3)]
        tau = _stress(G, mean(t["mul"][0]))
        jac = t["jac"][0]
        k = [mean(t["metric"][3 * d + c] * jac) for c in range(3)]
        dot = lambda v: sum(a * b for a, b in zip(k, v))  # noqa: E731
        f = [dot(tau[c]) for c in range(3)]
        e = sum(mean(t["bv"][1 + c]) * f[c] for c in range(3)) + mean(t["thermal_conductivity"][0]) * dot(grad(t["bv"][5]))
        Y = [mean(t["sv"][s]) for s in range(ns)]
        D = [mean(t["rho_D"][s]) for s in range(ns)]
        gy = [dot(grad(t["sv"][s])) for s in range(ns)]
        iw = [1.0 / float(w) for w in gas.mw]
        mw = 1 / sum(y * w for y, w in zip(Y, iw))
        gw = sum(a * w for a, w in zip(gy, iw))
        corr = sum(a * b for a, b in zip(D, gy)) - mw * sum(a * b for a, b in zip(D, Y)) * gw
        T = mean(t["bv"][5])
        js = []
        for s in range(ns):
            j = D[s] * (gy[s] - mw * Y[s] * gw) - Y[s] * corr
            e = e + gas.h_cp(s, T)[0] * j
            js.append(j)
        for c, x in enumerate(f + [e] + js):
            n = x.shape[x.dim() - 3 + axis] - 1
            dq[1 + c] += x.narrow(x.dim() - 3 + axis, 1, n) - x.narrow(x.dim() - 3 + axis, 0, n)


def _h2_residual(case, t, dims, g, gas):
    dq = torch.zeros((5 + gas.ns, dims[2], dims[1], dims[0]), dtype=F, device=t["bv"].device)
    _viscous2(t, dims, g, dq, gas)
    bv, sv, jac = (_inner(t[n], dims, g) for n in ("bv", "sv", "jac"))
    om, de, *_ = gas.source(bv[5], [bv[0] * sv[s] for s in range(gas.ns)])
    scale = torch.full_like(bv[0], 1e6)
    for s in range(gas.ns):
        dq[5 + s] += jac[0] * om[s]
        use = (sv[s] > 1e-25) & (de[s].abs() > 1e-25)
        scale = torch.where(use, torch.minimum(scale, (bv[0] * sv[s] / de[s]).abs()), scale)
    _inner(t["reaction_timeScale"], dims, g)[0] = scale
    _primitive_flux(case, t, dims, g, dq, gas)
    return dq


def _exact_h2_rhs(case, seed, device):
    t, dims, g, mech = _h2_block(case, seed, device)
    gas = _Gas(mech)
    _h2_properties(t, gas)
    return {"dq": _h2_residual(case, t, dims, g, gas), "reaction_timeScale": t["reaction_timeScale"]}


def _exact_h2_step(case, seed, device):
    t, dims, g, mech = _h2_block(case, seed, device)
    gas = _Gas(mech)
    t["cv"][:] = _h2_cv(t, gas)
    _h2_properties(t, gas)
    dt = _h2_dt(case)
    qn = _inner(t["cv"], dims, g).clone()
    for stage in STAGES:
        a, b, c = stage
        q = a * qn + b * _inner(t["cv"], dims, g) + c * dt / _inner(t["jac"][0], dims, g) * _h2_residual(case, t, dims, g, gas)
        q[5:] = q[5:].clamp(min=0)
        q[5:] *= q[0] / q[5:].sum(0)
        bv, sv = _inner(t["bv"], dims, g), _inner(t["sv"], dims, g)
        sv[...] = q[5:] / q[0]
        bv[0] = q[0]
        bv[1:4] = q[1:4] / q[0]
        r = sum(sv[s] * float(gas.r[s]) for s in range(gas.ns))
        bv[5] = gas.temperature(q[4] / q[0] - 0.5 * (bv[1] ** 2 + bv[2] ** 2 + bv[3] ** 2), sv, r, bv[5].clone(), 1e-5, 1000)
        bv[4] = q[0] * bv[5] * r
        _inner(t["cv"], dims, g)[...] = q
        for name in ("bv", "sv"):  # 2nd-order viscous terms: faces reach into the edges' ghosts
            for d in range(3):
                _wrap(t[name], d, dims, g, g)
        new = _h2_cv(t, gas)
        inside = torch.zeros_like(new[0], dtype=torch.bool)
        inside[g + 1:g + dims[2] - 1, g + 1:g + dims[1] - 1, g + 1:g + dims[0] - 1] = True
        t["cv"][:] = torch.where(inside, t["cv"], new)
        del new, q
        _h2_properties(t, gas)
    return {n: t[n] for n in ("cv", "bv", "sv")}


def _exact_reactors(case, seed, device):
    """The adaptive ROK4E integrator (Tranquilli and Sandu) with the full chemistry Jacobian, all
    reactors at once."""
    mech, (T0, p0, y0, _) = _reactor_requests(case, seed, device)
    gas, ns = _Gas(mech), mech.ns
    mw = torch.from_numpy(gas.mw).to(device)
    gam = 0.572816062482135
    a21, a31, a32 = 0.432364435748567, -0.51421131687617, 1.38227114461736
    g21, g31, g32 = -0.602765307997356 / gam, -1.389195789724843 / gam, 1.072950969011413 / gam
    g41, g42, g43 = 0.992356412977094 / gam, -1.390032613873701 / gam, -0.440875890223325 / gam
    b1, b2, b4 = 0.194335256262729, 0.483167813989227, 0.322496929748044
    e1, e2, e3, e4 = -0.217819895945721 - b1, 1.03130847478467 - b2, 0.186511421161047, -b4
    imw = (y0 / mw).sum(1)
    rho = p0 / (T0 * R_U * imw)
    E = sum(y0[:, s] * gas.h_cp(s, T0)[0] for s in range(ns)) - p0 / rho
    Y, T, p = (y0 * rho[:, None]).clone(), T0.clone(), p0.clone()
    n = T.numel()
    time, h = torch.zeros_like(T), torch.full_like(T, REACTOR_H0)
    err_last, step, rej = torch.zeros_like(T), torch.zeros_like(T), torch.zeros_like(T)

    def omega(t, y):
        om, _, q, sf, sb = gas.source(t, [y[:, s] for s in range(ns)])
        return torch.stack(om, 1), q, sf, sb

    def newton(y, t):
        yk = y / rho[:, None]
        im = (yk / mw).sum(1)
        return gas.temperature(E, [yk[:, s] for s in range(ns)], R_U * im, t, 1e-8, 100), im

    for _ in range(case["attempts"]):
        w1, q, sf, sb = omega(T, Y)
        qf, qb = torch.stack([a for a, _ in q], 1), torch.stack([b for _, b in q], 1)
        sf, sb = (torch.from_numpy(np.asarray(x, dtype=np.float64)).to(device) for x in (sf, sb))
        J = torch.einsum("qr,nqc->nrc", sb - sf, qf[:, :, None] * sf - qb[:, :, None] * sb)
        J = torch.where(Y[:, None, :] > 1e-30, J / Y[:, None, :].clamp(min=1e-300), torch.zeros_like(J)) * (1e3 * mw)[None, :, None]
        A = torch.eye(ns, dtype=F, device=device) - (h * gam)[:, None, None] * J
        solve = lambda b: torch.linalg.solve(A, b[:, :, None])[:, :, 0]  # noqa: E731
        hh = h[:, None]
        k1 = solve(w1)
        y = Y + hh * a21 * k1
        ts, _ = newton(y, T)
        k2 = solve(omega(ts, y)[0] + g21 * k1) - g21 * k1
        y = Y + hh * (a31 * k1 + a32 * k2)
        ts, _ = newton(y, ts)
        w3 = omega(ts, y)[0]
        k3 = solve(w3 + g31 * k1 + g32 * k2) - (g31 * k1 + g32 * k2)
        k4 = solve(w3 + g41 * k1 + g42 * k2 + g43 * k3) - (g41 * k1 + g42 * k2 + g43 * k3)
        y = Y + hh * (b1 * k1 + b2 * k2 + b4 * k4)
        err = (_sq(hh * (e1 * k1 + e2 * k2 + e3 * k3 + e4 * k4) / (RTOL * y + ATOL)).sum(1) / ns).sqrt()
        factor = (0.8 * err_last ** 0.1 * (err + 1e-20) ** -0.175).clamp(0.2, 5.0)
        h_next = torch.where(step > 0, h * factor, torch.where(err > 1, 0.2 * h, h))
        ok = err <= 1
        t_new, im = newton(torch.where(ok[:, None], y, Y), T)
        Y, time = torch.where(ok[:, None], y, Y), torch.where(ok, time + h, time)
        T = torch.where(ok, t_new, T)
        p = torch.where(ok, rho * R_U * im * T, p)
        err_last = torch.where(ok, err, err_last)
        h, step, rej = h_next, step + ok.to(F), rej + (~ok).to(F)
    return {"rhoY": Y, "rho_E_T_p": torch.stack([rho, E, T, p], 1), "time_h": torch.stack([time, h], 1), "error": err_last, "counts": None}
