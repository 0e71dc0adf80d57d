"""The work a user of this framework has it do: explicit RHS + SSP-RK3 steps of wall-modelled
LES cases in both precisions, through ``Solver``, ``Batch`` and the diagnostics.

A case is a dict of plain values.  ``kind`` names the flow:

* ``channel``  periodic channel between wall-modelled walls, constant mass flux (one or two blocks)
* ``ramp``     smooth ramp: synthetic inflow, wall model, characteristic outflow, sponge
* ``cgrid``    NACA 0012 C-grid of four blocks with turned interfaces, far field, wall model
* ``box``      fully periodic box on a curvilinear (skewed) grid

and ``call`` what is done with it: ``step`` (the state-resident loop), ``advance`` (the
max_dt + advance loop of the example drivers), ``rhs``, ``output`` (derived fields, plane
statistics, wall stresses) or ``batch`` (several independent channels in one launch, as the
server steps them).

``exact`` restates the method in plain 64-bit torch on the same inputs.
"""
import math

import numpy as np
import torch

from wmles_jax_b200 import (Block, CharacteristicFarfield, ConstantMassFlux, EquilibriumWallModel, Gas, Hybrid, KEP,
                            Mesh, MUSCLHLLC, SlipWall, Solver, WallModel)
from wmles_jax_b200.output import derived_fields
from wmles_jax_b200.serving import Batch
from wmles_jax_b200.smooth_ramp import SmoothRampInflow, SmoothRampSponge
from wmles_jax_b200.stats import PlaneStats
from wmles_jax_b200.workloads import NACA_SPAN, RAMP_SPAN, naca_cgrid_nodes, ramp_nodes, ramp_profile, ramp_props

NG = 3
LX, LZ = 2.0 * math.pi, math.pi                # channel box
BOX = (1.0, 0.6, 0.5)
X_RANGE, SPONGE_START = (-0.76, 4.0), 3.0      # ramp, in ramp lengths
SGS_COEFF = {"none": 0.0, "smagorinsky": 0.1, "wale": 0.5, "vreman": 0.17}
SGS_KEY = {"smagorinsky": "Cs", "wale": "Cw", "vreman": "Cs"}
BATCH_GRIDS = ((48, 48, 48), (64, 48, 48), (96, 64, 64), (128, 96, 64))


# ---------------------------------------------------------------------------- the cases
def listed():
    channel = dict(kind="channel", call="step", blocks=1, beta=2.5, scheme="kep4", sgs="wale", n_match=3,
                   isothermal=True, mach=0.3, reynolds=20000.0)
    ramp = dict(kind="ramp", call="step", ni=384, nj=96, nk=64, modes=64, sgs="vreman", steps=2)
    cgrid = dict(kind="cgrid", call="step", scale=1, alpha=4.0, n_match=3, sgs="vreman", steps=2)
    return [
        # a small channel of two blocks: a case to try a set-up on, bound by launches
        dict(channel, name="channel_32x32x16_fp64", ni=32, nj=32, nk=16, blocks=2, beta=2.0, scheme="kep2",
             sgs="smagorinsky", precision="fp64", steps=4),
        # an ordinary channel production run, in both forms
        dict(channel, name="channel_256x128x128_fp64", ni=256, nj=128, nk=128, precision="fp64", steps=3),
        dict(channel, name="channel_256x128x128_mixed", ni=256, nj=128, nk=128, precision="mixed", steps=3),
        # a spatially developing flow: inflow synthesis, sponge, shock-capturing blend
        dict(ramp, name="ramp_384x96x64_fp64", precision="fp64"),
        dict(ramp, name="ramp_384x96x64_mixed", precision="mixed"),
        # an external flow on several blocks of different sizes
        dict(cgrid, name="cgrid_fp64", precision="fp64"),
        dict(cgrid, name="cgrid_mixed", precision="mixed"),
        # several users' channels stepped together
        dict(channel, name="batch_6_mixed", call="batch", members=6, precision="mixed", steps=2),
        # compressible turbulence in a box with a curvilinear grid of odd sizes, upwind scheme
        dict(name="box_75x53x37_muscl_fp64", kind="box", call="advance", ni=75, nj=53, nk=37, skew=0.03,
             scheme="muscl_minmod", sgs="none", precision="fp64", steps=2),
        # the same kind of grid, ordinary size, central scheme
        dict(name="box_160x96x72_kep4_mixed", kind="box", call="step", ni=160, nj=96, nk=72, skew=0.03,
             scheme="kep4", sgs="wale", precision="mixed", steps=2),
        # a residual evaluation (an outer time integrator of the user's own)
        dict(channel, name="rhs_96x64x64_fp64", call="rhs", ni=96, nj=64, nk=64, precision="fp64", steps=1),
        # sampling and output between steps
        dict(channel, name="output_192x96x96_fp64", call="output", ni=192, nj=96, nk=96, precision="fp64", steps=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    precision = rng.choice(("fp64", "mixed"))
    sgs = rng.choice(("none", "smagorinsky", "wale", "vreman", "wale", "vreman"))
    schemes = ("kep2", "kep4", "kep4", "muscl_minmod", "muscl_albada", "hybrid")
    steps = rng.randint(1, 3)
    pick = rng.random()
    if pick < 0.55:
        call = rng.choice(("step", "step", "step", "step", "advance", "batch", "rhs", "output"))
        case = dict(kind="channel", call=call, blocks=rng.choice((1, 1, 2)), beta=round(rng.uniform(1.6, 2.6), 2),
                    scheme=rng.choice(("kep2", "kep4", "kep4", "kep4", "hybrid")), sgs=sgs,
                    n_match=rng.randint(1, 3), isothermal=rng.random() < 0.7, mach=round(rng.uniform(0.15, 0.5), 3),
                    reynolds=round(math.exp(rng.uniform(math.log(5e3), math.log(1.2e5)))), precision=precision,
                    steps=steps)
        if call == "batch":
            return dict(case, scheme="kep4", blocks=1, members=rng.randint(2, 10))
        if call == "rhs":                      # the mixed form's residual is single precision: FP64 here
            case["precision"] = "fp64"
        case.update(ni=_log(rng, 16, 256), nj=_log(rng, 12, 128), nk=_log(rng, 8, 128))
        if case["blocks"] == 2:
            case["ni"] += case["ni"] % 2
        return case
    if pick < 0.75:
        return dict(kind="box", call=rng.choice(("step", "advance")), ni=_log(rng, 12, 192), nj=_log(rng, 12, 112),
                    nk=_log(rng, 10, 96), skew=round(rng.uniform(0.0, 0.04), 4), scheme=rng.choice(schemes), sgs=sgs,
                    precision=precision, steps=steps)
    if pick < 0.9:
        return dict(kind="ramp", call="step", ni=_log(rng, 48, 384), nj=_log(rng, 20, 96), nk=_log(rng, 8, 64),
                    modes=rng.choice((16, 32, 48, 64)), sgs=rng.choice(("vreman", "wale")), precision=precision,
                    steps=min(steps, 2))
    return dict(kind="cgrid", call="step", scale=rng.choice((1, 2, 4)), alpha=round(rng.uniform(0.0, 8.0), 2),
                n_match=rng.randint(1, 3), sgs=rng.choice(("vreman", "wale")), precision=precision, steps=min(steps, 2))


def _cells(case):
    if case["call"] == "batch":
        return sum(math.prod(BATCH_GRIDS[m % len(BATCH_GRIDS)]) for m in range(case["members"]))
    if case["kind"] == "cgrid":
        s = case["scale"]
        return (576 // s) * (64 // s) * (40 // s)
    return case["ni"] * case["nj"] * case["nk"]


def work(case):
    """Bytes and operations of the method per interior cell.  A stage cannot start before its
    neighbours' last stage is done, so each reads the state and the metrics (area vectors, volume,
    centre) and writes the state; stages 2 and 3 also read the step's first state.  Operations are
    additions and multiplications of one residual: inviscid faces, gradients, SGS, viscous faces."""
    cells = _cells(case)
    met = 104 if case["precision"] == "fp64" else 52
    flops = 900 + (0 if case["sgs"] == "none" else 60)
    flops += {"kep2": 90, "kep4": 330}.get(case.get("scheme", "hybrid"), 450)
    stage = 3 * (80 + met) + 2 * 40
    cfl = 40 + (80 if case["precision"] == "fp64" else 40)
    cmf = 80 if case["kind"] == "channel" else 0
    if case["call"] == "rhs":
        return dict(bytes=cells * (80 + met), flops=cells * flops)
    if case["call"] == "output":
        return dict(bytes=cells * (40 + met + 11 * 8), flops=cells * 330)
    return dict(bytes=case["steps"] * cells * (stage + cfl + cmf), flops=case["steps"] * cells * (3 * flops + 60))


# ---------------------------------------------------------------------------- inputs
def _linspace_nodes(x, y, z):
    return np.stack(np.meshgrid(x, y, z, indexing="ij"))


def _channel_nodes(case, n):
    ni, nj, nk = n
    y = 1.0 + np.tanh(case["beta"] * (2.0 * np.linspace(0.0, 1.0, nj + 1) - 1.0)) / np.tanh(case["beta"])
    x, z = np.linspace(0.0, LX, ni + 1), np.linspace(0.0, LZ, nk + 1)
    per = ni // case["blocks"]
    return [_linspace_nodes(x[b * per:(b + 1) * per + 1], y, z) for b in range(case["blocks"])]


def _box_nodes(case):
    X, Y, Z = _linspace_nodes(*(np.linspace(0.0, L, case[k] + 1) for L, k in zip(BOX, ("ni", "nj", "nk"))))
    s, kx, ky, kz = case["skew"], *(2.0 * math.pi / L for L in BOX)
    return [np.stack([X + s * np.sin(ky * Y) * np.sin(kz * Z), Y + 0.5 * s * np.sin(kx * X),
                      Z + 0.5 * s * np.sin(kx * X) * np.cos(ky * Y)])]


def _gas(case):
    """Nondimensional gas (rho = T = 1, |U| = 1 at the case's Mach number), air for the ramp."""
    if case["kind"] == "ramp":
        return Gas()
    mach, re = {"box": (0.4, 5000.0), "cgrid": (0.15, 1e6)}.get(case["kind"]) or (case["mach"], case["reynolds"])
    return Gas(gamma=1.4, R=1.0 / (1.4 * mach ** 2), mu_ref=1.0 / re, T_ref=1.0, S_suth=110.4 / 300.0)


def _far(case, gas):
    """Free-stream primitives of the external flows."""
    if case["kind"] == "ramp":
        p = ramp_props(gas)
        return np.array([p["rho_inf"], p["U_inf"], 0.0, 0.0, p["p_inf"]])
    a = math.radians(case["alpha"])
    return np.array([1.0, math.cos(a), math.sin(a), 0.0, gas.R])


def _layout(case, n=None):
    """The case's blocks as plain data: [(name, nodes, {face: boundary})], a boundary being
    ("link", block, face, axis mapping, flips, shift), ("wall", n_match, T_wall), ("slip",),
    ("far",) or ("inflow",)."""
    same = ((0, 1, 2), (False, False, False))
    kind = case["kind"]
    if kind == "channel":
        nodes = _channel_nodes(case, n or (case["ni"], case["nj"], case["nk"]))
        nb, wall = len(nodes), ("wall", case["n_match"], 1.0 if case["isothermal"] else None)
        out = []
        for b, x in enumerate(nodes):
            lo, hi = (b - 1) % nb, (b + 1) % nb
            out.append((f"B{b}", x, {
                "imin": ("link", lo, "imax", *same, (-LX if b == 0 else 0.0, 0.0, 0.0)),
                "imax": ("link", hi, "imin", *same, (LX if b == nb - 1 else 0.0, 0.0, 0.0)),
                "jmin": wall, "jmax": wall,
                "kmin": ("link", b, "kmax", *same, (0.0, 0.0, -LZ)),
                "kmax": ("link", b, "kmin", *same, (0.0, 0.0, LZ))}))
        return out
    if kind == "box":
        faces = {}
        for a, name in enumerate("ijk"):
            sh = [0.0, 0.0, 0.0]
            sh[a] = BOX[a]
            faces[name + "min"] = ("link", 0, name + "max", *same, tuple(-s for s in sh))
            faces[name + "max"] = ("link", 0, name + "min", *same, tuple(sh))
        return [("box", _box_nodes(case)[0], faces)]
    if kind == "ramp":
        length = ramp_props(_gas(case))["L"]
        span = RAMP_SPAN * length
        return [("ramp", ramp_nodes((case["ni"], case["nj"], case["nk"]), x_range=X_RANGE, L=length), {
            "imin": ("inflow",), "imax": ("far",), "jmin": ("wall", 1, None), "jmax": ("slip",),
            "kmin": ("link", 0, "kmax", *same, (0.0, 0.0, -span)),
            "kmax": ("link", 0, "kmin", *same, (0.0, 0.0, span))})]
    nodes = naca_cgrid_nodes(case["scale"])
    names = ("wake_lower", "section", "section_aft", "wake_upper")
    flip_j, turn = ((0, 1, 2), (False, True, False)), ((1, 0, 2), (False, False, False))
    wall, z3 = ("wall", min(case["n_match"], min(x.shape[2] - 1 for x in nodes.values())), None), (0.0, 0.0, 0.0)
    faces = [
        {"imin": ("link", 1, "imin", *flip_j, z3), "imax": ("far",), "jmin": ("far",), "jmax": ("link", 3, "jmin", *same, z3)},
        {"imin": ("link", 0, "imin", *flip_j, z3), "imax": ("link", 2, "jmax", *turn, z3), "jmin": wall, "jmax": ("far",)},
        {"jmax": ("link", 1, "imax", *turn, z3), "jmin": ("link", 3, "imin", *turn, z3), "imin": wall, "imax": ("far",)},
        {"imin": ("link", 2, "jmin", *turn, z3), "jmin": ("link", 0, "jmax", *same, z3), "jmax": ("far",), "imax": ("far",)}]
    out = []
    for b, name in enumerate(names):
        faces[b]["kmin"] = ("link", b, "kmax", *same, (0.0, 0.0, -NACA_SPAN))
        faces[b]["kmax"] = ("link", b, "kmin", *same, (0.0, 0.0, NACA_SPAN))
        out.append((name, nodes[name], faces[b]))
    return out


def _scheme(case):
    name = case.get("scheme", "hybrid")
    if name.startswith("kep"):
        return KEP(int(name[3:]))
    return MUSCLHLLC(name[6:]) if name.startswith("muscl") else Hybrid(KEP(4))


def _inflow(case, seed, gas):
    return SmoothRampInflow(ramp_props(gas), ramp_profile(), (0.1, 0.02, 0.03), seed % 100003, case["modes"], case["nk"])


def _solver(case, seed, n=None):
    """What a user's program builds once: mesh, gas, boundary conditions, solver."""
    gas, layout, wm = _gas(case), _layout(case, n), EquilibriumWallModel()
    blocks = [Block(name, x) for name, x, _ in layout]
    mesh = Mesh(blocks)
    for b, (_, _, faces) in enumerate(layout):
        for face, bc in faces.items():
            if bc[0] == "link":
                if (b, face) <= (bc[1], bc[2]):
                    mesh.connect(blocks[b], face, blocks[bc[1]], bc[2], shift=bc[5])
            elif bc[0] == "wall":
                blocks[b].set_bc(face, WallModel(wm, T_wall=bc[2], n_match=bc[1]))
            elif bc[0] == "slip":
                blocks[b].set_bc(face, SlipWall())
            elif bc[0] == "far":
                blocks[b].set_bc(face, CharacteristicFarfield(_far(case, gas)))
            else:
                blocks[b].set_bc(face, _inflow(case, seed, gas))
    mesh.finalize(device=True)
    kw = dict(scheme=_scheme(case), sgs=case["sgs"], cfl=0.5, precision=case["precision"])
    if case["sgs"] != "none":
        kw["sgs_kwargs"] = {SGS_KEY[case["sgs"]]: SGS_COEFF[case["sgs"]]}
    if case["kind"] == "channel":
        kw["constraints"] = [ConstantMassFlux(0, 1.0)]
    if case["kind"] == "ramp":
        kw["sources"] = (SmoothRampSponge(ramp_props(gas), SPONGE_START, X_RANGE[1], 1.0),)
    return Solver(mesh, gas, **kw)


def _noise(shape, seed, block):
    g = torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) + block)
    return torch.randn((3,) + tuple(shape), dtype=torch.float64, device="cuda", generator=g)


def _initial(case, seed, geo, ref_gas):
    """Conservative states at the ghosted cell centres: a mean profile with the fluctuations a
    developed flow has (tapered at walls), drawn from the seed."""
    out = []
    for b, (xc, shape) in enumerate(geo):
        x, y, z = xc
        one = torch.ones(shape, dtype=torch.float64, device="cuda")
        e = _noise(shape, seed, b)
        p = ref_gas["R"] * one
        rho = one.clone()
        if case["kind"] == "channel":
            s = (1.0 - (1.0 - y).abs()).clamp(min=0.0, max=1.0) ** (1.0 / 7.0)
            u, v, w = (s * (8.0 / 7.0 + 0.08 * e[0]), s * 0.08 * e[1], s * 0.08 * e[2])
        elif case["kind"] == "box":
            kx, ky, kz = (2.0 * math.pi / L for L in BOX)
            u = torch.sin(ky * y) + 0.3 * torch.cos(kz * z) + 0.03 * e[0]
            v = 0.4 * torch.sin(kx * x) * torch.sin(kz * z) + 0.03 * e[1]
            w = 0.3 * torch.cos(kx * x) + 0.03 * e[2]
            rho = 1.0 + 0.05 * torch.sin(kx * x) * torch.cos(kz * z)
            p = ref_gas["R"] * (1.0 + 0.15 * torch.tanh(8.0 * torch.cos(kx * x) * torch.sin(ky * y)))
        elif case["kind"] == "ramp":
            f = torch.as_tensor(ref_gas["far"], device="cuda")
            L, h = ref_gas["L"], 0.22
            xi = (x / L).clamp(0.0, 1.0)
            eta = ((y / L - h * (1.0 - (10.0 * xi ** 3 - 15.0 * xi ** 4 + 6.0 * xi ** 5))) / 0.028).clamp(0.0, 1.0)
            u, v, w = (f[1] * eta ** (1.0 / 7.0) * (1.0 + 0.02 * e[0]), f[1] * 0.02 * e[1], f[1] * 0.02 * e[2])
            rho, p = f[0] * one, f[4] * one
        else:
            f = torch.as_tensor(ref_gas["far"], device="cuda")
            u, v, w = f[1] + 0.01 * e[0], f[2] + 0.01 * e[1], 0.01 * e[2]
        E = p / (ref_gas["gamma"] - 1.0) + 0.5 * rho * (u * u + v * v + w * w)
        out.append(torch.stack([rho, rho * u, rho * v, rho * w, E]))
    return out


def _constants(case):
    g = _gas(case)
    c = dict(gamma=g.gamma, R=g.R, Pr=g.Pr, Prt=g.Pr_t, mu=g.mu_ref, T0=g.T_ref, S=g.S_suth, cp=g.gamma * g.R / (g.gamma - 1.0))
    if case["kind"] in ("ramp", "cgrid"):
        c["far"] = _far(case, g)
    if case["kind"] == "ramp":
        c["L"] = ramp_props(g)["L"]
    return c


def _member(case, m):
    """Channel m of a batch: its grid, Mach and Reynolds number."""
    one = {k: v for k, v in case.items() if k not in ("name", "members")}
    n = BATCH_GRIDS[m % len(BATCH_GRIDS)]
    return dict(one, call="step", ni=n[0], nj=n[1], nk=n[2], mach=min(0.5, case["mach"] * (0.8 + 0.1 * (m % 5))),
                reynolds=case["reynolds"] * (1.0 + 0.25 * m))


def _begin(case, seed):
    s = _solver(case, seed)
    layout = _layout(case)
    geo = [(xc, xc.shape[1:]) for xc in (_centres(X) for X in _ghost_nodes(layout))]
    Q = s.apply_bcs(tuple(q.contiguous() for q in _initial(case, seed, geo, _constants(case))), time=0.0)
    return s, Q


def prepare(case, seed):
    if case["call"] != "batch":
        s, Q = _begin(case, seed)
        return dict(case=case, s=s, Q=Q)
    pairs = [_begin(_member(case, m), seed + 7919 * m) for m in range(case["members"])]
    solvers, qa = [s for s, _ in pairs], [q for _, q in pairs]
    bufs = [[tuple(torch.zeros_like(b) for b in q) for q in qa] for _ in range(2)]
    dts = [[torch.zeros((), dtype=torch.float64, device="cuda") for _ in qa] for _ in range(2)]
    return dict(case=case, batch=Batch(solvers), solvers=solvers, qa=qa, da=[s.max_dt(q) for s, q in pairs], bufs=bufs, dts=dts)


def run(state):
    case = state["case"]
    if case["call"] == "batch":
        q, dt = state["qa"], state["da"]
        for k in range(case["steps"]):
            qn, dn = state["bufs"][k % 2], state["dts"][k % 2]
            state["batch"].step(q, qn, dt, dn)
            q, dt = qn, dn
        return [[list(x) for x in q], list(dt)]
    s, Q, t = state["s"], state["Q"], 0.0
    if case["call"] == "rhs":
        return list(s.rhs(Q, t))
    if case["call"] == "output":
        stats = PlaneStats(s.mesh, s)
        stats.accumulate(Q)
        y, mean = stats.result()
        fields = derived_fields(s, Q, as_numpy=False)
        walls = s.wall_stats_device(Q)
        return [fields[0], mean, stats.mean_tau_w, [walls[k] for k in sorted(walls)]]
    for _ in range(case["steps"]):
        if case["call"] == "advance":
            dt = s.max_dt(Q, t)
            Q = s.advance(Q, dt, t)
        else:
            Q, dt = s.step(Q, t)
        t += float(dt)
    return [list(Q), dt]


# ---------------------------------------------------------------------------- the method in plain torch, 64 bits
def _at(d, s, other=slice(None), lead=1):
    """Index tuple: `s` on spatial axis d, `other` on the other two, behind `lead` axes."""
    t = [slice(None)] * lead + [other] * 3
    t[lead + d] = s
    return tuple(t)


def _cut(a, d, lo, hi):
    """Interior of `a` with the axis d running over [NG + lo, N - NG + hi)."""
    lead = a.dim() - 3
    t = [slice(None)] * lead + [slice(NG, a.shape[lead + x] - NG) for x in range(3)]
    t[lead + d] = slice(NG + lo, a.shape[lead + d] - NG + hi)
    return a[tuple(t)]


def _inner(a):
    return _cut(a, 0, 0, 0)


def _face(name):
    return "ijk".index(name[0]), int(name[1:] == "max")


def _exchange(dst, src, face, bc, node):
    """Ghost layers of `dst` at `face` from the interior layers of the linked face of `src`."""
    a, s = face
    b, r = _face(bc[2])
    lo_src = (NG + node) if r == 0 else src.shape[1 + b] - 2 * NG - node
    layers = src.narrow(1 + b, lo_src, NG)
    if r == 1:
        layers = layers.flip(1 + b)
    layers = layers.permute(0, *(1 + m for m in bc[3]))
    turned = [1 + t for t in range(3) if bc[4][t]] + ([1 + a] if s == 0 else [])
    layers = layers.flip(turned) if turned else layers.clone()
    dst.narrow(1 + a, 0 if s == 0 else dst.shape[1 + a] - NG, NG).copy_(layers)
    return dst.narrow(1 + a, 0 if s == 0 else dst.shape[1 + a] - NG, NG)


def _ghost_nodes(layout):
    """Node arrays with NG ghost layers: neighbours' nodes across links, mirrored elsewhere."""
    Xs = []
    for _, nodes, _ in layout:
        x = torch.as_tensor(np.ascontiguousarray(nodes), dtype=torch.float64, device="cuda")
        X = torch.zeros((3,) + tuple(n + 2 * NG for n in x.shape[1:]), dtype=torch.float64, device="cuda")
        X[:, NG:-NG, NG:-NG, NG:-NG] = x
        Xs.append(X)
    for _ in range(3):
        for a in range(3):
            for b, (_, _, faces) in enumerate(layout):
                for s, end in enumerate(("min", "max")):
                    bc, X = faces["ijk"[a] + end], Xs[b]
                    if bc[0] == "link":
                        ghosts = _exchange(X, Xs[bc[1]], (a, s), bc, 1)
                        ghosts += torch.tensor(bc[5], dtype=torch.float64, device="cuda").view(3, 1, 1, 1)
                    else:
                        n = X.shape[1 + a]
                        edge = X.narrow(1 + a, NG if s == 0 else n - NG - 1, 1)
                        inner = X.narrow(1 + a, NG + 1 if s == 0 else n - 2 * NG - 1, NG).flip(1 + a)
                        X.narrow(1 + a, 0 if s == 0 else n - NG, NG).copy_(2.0 * edge - inner)
    return Xs


def _centres(X):
    c = 0.0
    for a in (0, 1):
        for b in (0, 1):
            for d in (0, 1):
                c = c + X[:, a:X.shape[1] - 1 + a, b:X.shape[2] - 1 + b, d:X.shape[3] - 1 + d]
    return c / 8.0


def _geometry(X):
    N = [n - 1 for n in X.shape[1:]]
    S, xf, vol = [], [], 0.0
    for d in range(3):
        t1, t2 = (d + 1) % 3, (d + 2) % 3

        def corner(a, b):
            t = [slice(None)] * 4
            t[1 + t1], t[1 + t2] = slice(a, N[t1] + a), slice(b, N[t2] + b)
            return X[tuple(t)]
        c00, c10, c01, c11 = corner(0, 0), corner(1, 0), corner(0, 1), corner(1, 1)
        S.append(0.5 * torch.linalg.cross(c11 - c00, c01 - c10, dim=0))
        xf.append(0.25 * (c00 + c10 + c01 + c11))
        f = (xf[d] * S[d]).sum(0)
        vol = vol + (f[_at(d, slice(1, None), lead=0)] - f[_at(d, slice(None, -1), lead=0)])
    return dict(S=S, xf=xf, vol=vol / 3.0, xc=_centres(X))


class _Reference:
    def __init__(self, case, seed, layout, c):
        self.case, self.layout, self.c = case, layout, c
        self.geo = [_geometry(X) for X in _ghost_nodes(layout)]
        if case["kind"] == "ramp":
            g = _gas(case)
            self.props, self.profile = ramp_props(g), torch.as_tensor(ramp_profile(), device="cuda")
            self.modes = torch.as_tensor(_inflow(case, seed, g).mode_table(), device="cuda")

    # ---- gas
    def prim(self, q):
        u = q[1:4] / q[0]
        p = (self.c["gamma"] - 1.0) * (q[4] - 0.5 * q[0] * (u * u).sum(0))
        return torch.cat([q[:1], u, p[None]]), p / (q[0] * self.c["R"])

    def cons(self, w):
        return torch.cat([w[:1], w[:1] * w[1:4], (w[4] / (self.c["gamma"] - 1.0) + 0.5 * w[0] * (w[1:4] ** 2).sum(0))[None]])

    def mu(self, T):
        c = self.c
        return c["mu"] * (T / c["T0"]) ** 1.5 * (c["T0"] + c["S"]) / (T + c["S"])

    # ---- ghost cells
    def mirror(self, q, geo, face, bc):
        a, s = face
        n = q.shape[1 + a]
        S = geo["S"][a].narrow(1 + a, NG if s == 0 else n - NG, 1)
        nrm = S / (S * S).sum(0).sqrt()
        for m in range(NG):
            gi, ii = (NG - 1 - m, NG + m) if s == 0 else (n - NG + m, n - NG - 1 - m)
            w, T = self.prim(q.narrow(1 + a, ii, 1))
            if bc[0] in ("slip", "wall"):
                w = torch.cat([w[:1], w[1:4] - 2.0 * (w[1:4] * nrm).sum(0) * nrm, w[4:]])
            else:
                w = self.far(w, T, nrm if s == 1 else -nrm)
            q.narrow(1 + a, gi, 1).copy_(self.cons(w))

    def far(self, w, T, n):
        c = self.c
        f = torch.as_tensor(c["far"], device="cuda").view(5, 1, 1, 1)
        ri, ui, pi = f[0], f[1:4], f[4]
        ci = torch.sqrt(c["gamma"] * pi / ri)
        un, uni = (w[1:4] * n).sum(0), (ui * n).sum(0)
        a = torch.sqrt(c["gamma"] * c["R"] * T)
        drho, dp, dun = w[0] - ri, w[4] - pi, un - uni
        zero = torch.zeros_like(dp)
        ap = torch.where(un + a > 0.0, dp + ri * ci * dun, zero)
        am = torch.where(un - a > 0.0, dp - ri * ci * dun, zero)
        pb, ub = 0.5 * (ap + am), (ap - am) / (2.0 * ri * ci)
        out = un > 0.0
        rho = ri + pb / ci ** 2 + torch.where(out, drho - dp / ci ** 2, zero)
        tang = torch.where(out, w[1:4] - ui - dun * n, torch.zeros_like(n))
        return torch.cat([rho[None], ui + ub * n + tang, (pi + pb)[None]])

    def inflow(self, q, geo, t):
        p, tab, U = self.props, self.profile, self.props["U_inf"]
        nk = q.shape[3] - 2 * NG
        for m in range(NG):
            gi = NG - 1 - m
            y, z = geo["xc"][1, gi] / p["L"], geo["xc"][2, gi] / p["L"]
            fields = []
            for k in range(3):
                kx, ky, kz, ph = (v.view(-1, 1, 1) for v in self.modes[k])
                f = torch.cos(kx * (U * t / p["L"]) + ky * y + kz * z + ph).sum(0)
                f = f - f[:, NG:NG + nk].mean(1, keepdim=True)
                if k == 1:
                    f = f - (f * fields[0])[:, NG:NG + nk].mean(1, keepdim=True) * fields[0]
                fields.append(f / (f[:, NG:NG + nk] ** 2).mean(1, keepdim=True).clamp(min=1e-20).sqrt())
            i = (torch.searchsorted(tab[:, 0].contiguous(), y.contiguous(), right=True) - 1).clamp(0, len(tab) - 2)
            r = ((y - tab[i, 0]) / (tab[i + 1, 0] - tab[i, 0])).clamp(0.0, 1.0)
            col = [tab[i, k] + r * (tab[i + 1, k] - tab[i, k]) for k in range(7)]
            uu, vv, ww, uv = (v * U ** 2 for v in (col[3].clamp(min=0.0), col[4].clamp(min=0.0), col[5].clamp(min=0.0), col[6]))
            su = uu.sqrt()
            l10 = torch.where(su > 1e-14, uv / su.clamp(min=1e-14), torch.zeros_like(su))
            u = U * col[1] + su * fields[0]
            v = U * col[2] + l10 * fields[0] + (vv - l10 ** 2).clamp(min=0.0).sqrt() * fields[1]
            one = torch.ones_like(u)
            q[:, gi] = self.cons(torch.stack([p["rho_inf"] * one, u, v, ww.sqrt() * fields[2], p["p_inf"] * one]))

    def fill(self, Q, t):
        Q = [q.clone() for q in Q]
        for _ in range(2):
            for a in range(3):
                for b, (_, _, faces) in enumerate(self.layout):
                    for s, end in enumerate(("min", "max")):
                        bc = faces["ijk"[a] + end]
                        if bc[0] == "link":
                            _exchange(Q[b], Q[bc[1]], (a, s), bc, 0)
                        elif bc[0] == "inflow":
                            self.inflow(Q[b], self.geo[b], t)
                        else:
                            self.mirror(Q[b], self.geo[b], (a, s), bc)
        return Q

    def refresh(self, Q, t):
        """The ghost cells a residual reads (two deep on faces, one on edges) from their sources."""
        out = []
        for q, f in zip(Q, self.fill(Q, t)):
            depth = []
            for a in range(3):
                i, n = torch.arange(q.shape[1 + a], device="cuda"), q.shape[1 + a] - 2 * NG
                d = torch.maximum((NG - i).clamp(min=0), (i - NG - n + 1).clamp(min=0))
                depth.append(d.view([-1 if x == a else 1 for x in range(3)]).expand(q.shape[1:]))
            depth = torch.stack(depth)
            n, top = (depth > 0).sum(0), depth.amax(0)
            out.append(torch.where(((n == 1) & (top <= 2)) | ((n == 2) & (top == 1)), f, q))
        return out

    # ---- fluxes through the faces of direction d
    def central(self, order, w, S, d):
        g = self.c["gamma"]

        def pair(a, b):
            A, B = _cut(w, d, a, a + 1), _cut(w, d, b, b + 1)
            rho, u, p = (0.5 * (A[i] + B[i]) for i in (0, slice(1, 4), 4))
            e = 0.5 * sum(X[4] / ((g - 1.0) * X[0]) + 0.5 * (X[1:4] ** 2).sum(0) for X in (A, B))
            un = (u * S).sum(0)
            m = rho * un
            return torch.cat([m[None], m * u + p * S, (m * e + p * un)[None]])
        F = pair(-1, 0)
        return F if order == 2 else 4.0 / 3.0 * F - 1.0 / 6.0 * (pair(-1, 1) + pair(-2, 0))

    def upwind(self, limiter, w, S, d):
        L2, L, R, R2 = (_cut(w, d, i, i + 1) for i in (-2, -1, 0, 1))

        def lim(a, b):
            if limiter == "minmod":
                return 0.5 * (torch.sign(a) + torch.sign(b)) * torch.minimum(a.abs(), b.abs())
            return (a * (b * b + 1e-12) + b * (a * a + 1e-12)) / (a * a + b * b + 2e-12)
        l, r = L + 0.5 * lim(L - L2, R - L), R - 0.5 * lim(R - L, R2 - R)
        bad = (l[0] <= 0) | (l[4] <= 0) | (r[0] <= 0) | (r[4] <= 0)
        l, r = torch.where(bad, L, l), torch.where(bad, R, r)
        g, area = self.c["gamma"], (S * S).sum(0).sqrt()
        n = S / area
        (ul, ur), (cl, cr) = ([(x[1:4] * n).sum(0) for x in (l, r)], [torch.sqrt(g * x[4] / x[0]) for x in (l, r)])
        sl, sr = torch.minimum(ul - cl, ur - cr), torch.maximum(ul + cl, ur + cr)
        ss = (r[4] - l[4] + l[0] * ul * (sl - ul) - r[0] * ur * (sr - ur)) / (l[0] * (sl - ul) - r[0] * (sr - ur))

        def flux(x, un):
            q = self.cons(x)
            return torch.cat([(x[0] * un)[None], x[0] * un * x[1:4] + x[4] * n, ((q[4] + x[4]) * un)[None]]), q

        def star(x, un, s, F, q):
            f = x[0] * (s - un) / (s - ss)
            e = q[4] / x[0] + (ss - un) * (ss + x[4] / (x[0] * (s - un)))
            return F + s * (torch.cat([f[None], f * (x[1:4] + (ss - un) * n), (f * e)[None]]) - q)
        (Fl, ql), (Fr, qr) = flux(l, ul), flux(r, ur)
        right = torch.where(sr > 0, star(r, ur, sr, Fr, qr), Fr)
        return area * torch.where(sl >= 0, Fl, torch.where(ss >= 0, star(l, ul, sl, Fl, ql), right))

    def inviscid(self, w, S, d, theta):
        name = self.case.get("scheme", "hybrid")
        if name.startswith("kep"):
            return self.central(int(name[3:]), w, S, d)
        if name.startswith("muscl"):
            return self.upwind(name[6:], w, S, d)
        s = ((torch.maximum(_cut(theta, d, -1, 0), _cut(theta, d, 0, 1)) - 0.6) / (0.9 - 0.6)).clamp(0.0, 1.0)
        return (1.0 - s) * self.central(4, w, S, d) + s * self.upwind("albada", w, S, d)

    def gradient(self, phi, geo):
        acc = 0.0
        for d in range(3):
            lo, hi = _at(d, slice(None, -1)), _at(d, slice(1, None))
            f = (0.5 * (phi[lo] + phi[hi]))[:, None] * geo["S"][d][_at(d, slice(1, phi.shape[1 + d]))][None]
            acc = acc + f[_at(d, slice(1, None), slice(1, -1), 2)] - f[_at(d, slice(None, -1), slice(1, -1), 2)]
        return torch.nn.functional.pad(acc / geo["vol"][1:-1, 1:-1, 1:-1], (1,) * 6)

    def eddy(self, g, delta):
        name, c = self.case["sgs"], SGS_COEFF[self.case["sgs"]]
        if name == "none":
            return torch.zeros_like(delta)
        sym = 0.5 * (g + g.transpose(0, 1))
        ss = (sym * sym).sum((0, 1))
        if name == "smagorinsky":
            return (c * delta) ** 2 * torch.sqrt(2.0 * ss)
        if name == "wale":
            g2 = torch.stack([torch.stack([sum(g[i, k] * g[k, j] for k in range(3)) for j in range(3)]) for i in range(3)])
            sd = 0.5 * (g2 + g2.transpose(0, 1))
            tr = (g2[0, 0] + g2[1, 1] + g2[2, 2]) / 3.0
            for i in range(3):
                sd[i, i] -= tr
            sd = (sd * sd).sum((0, 1))
            return (c * delta) ** 2 * sd ** 1.5 / (ss ** 2.5 + sd ** 1.25 + 1e-30)
        b = torch.stack([torch.stack([delta ** 2 * sum(g[i, k] * g[j, k] for k in range(3)) for j in range(3)]) for i in range(3)])
        B = (b[0, 0] * b[1, 1] - b[0, 1] ** 2 + b[0, 0] * b[2, 2] - b[0, 2] ** 2 + b[1, 1] * b[2, 2] - b[1, 2] ** 2)
        return 2.5 * c ** 2 * torch.sqrt(B.clamp(min=0.0) / ((g * g).sum((0, 1)) + 1e-30))

    def wall(self, w, T, geo, a, s, n_match, T_wall):
        """Flux through a wall-modelled face and its (tau_w, q_w)."""
        c, n = self.c, w.shape[1 + a]

        def take(x, i):
            return _inner_of(x, a, i)
        fb, mi, ci = (NG, NG + n_match - 1, NG) if s == 0 else (n - NG, n - NG - n_match, n - NG - 1)
        S = take(geo["S"][a], fb)
        area = (S * S).sum(0).sqrt()
        out = S / area if s == 1 else -S / area
        h = -((take(geo["xc"], mi) - take(geo["xf"][a], fb)) * out).sum(0)
        u = take(w[1:4], mi)
        up = u - (u * out).sum(0) * out
        U = torch.sqrt((up * up).sum(0) + 1e-20)
        Th, ph, pb = take(T, mi), take(w[4], mi), take(w[4], ci)
        Um = U.clamp(min=1e-8)
        Tw = T_wall + 0.0 * Th if T_wall is not None else Th + c["Pr"] ** (1.0 / 3.0) * Um ** 2 / (2.0 * c["cp"])
        rw = ph / (c["R"] * Tw)
        mw = self.mu(Tw)
        k, ekb = 0.41, math.exp(-0.41 * 5.2)
        re = h * Um * rw / mw
        x = re.sqrt().clamp(1.0, 25.0)
        for _ in range(30):
            e = torch.exp(k * x)
            F = x + ekb * (e - 1.0 - k * x - 0.5 * (k * x) ** 2 - (k * x) ** 3 / 6.0) - re / x
            dF = 1.0 + ekb * k * (e - 1.0 - k * x - 0.5 * (k * x) ** 2) + re / x ** 2
            x = torch.minimum(torch.maximum(x - F / dF, 0.5 * x), torch.full_like(x, 100.0))
        ut = Um / x
        tau, q = rw * ut ** 2, torch.zeros_like(ut)
        if T_wall is not None:
            Pr = c["Pr"]
            yp = (h * ut * rw / mw).clamp(min=1e-6)
            gam = (0.01 * (Pr * yp) ** 4 / (1.0 + 5.0 * Pr ** 3 * yp)).clamp(min=1e-20)
            beta = (3.85 * Pr ** (1.0 / 3.0) - 1.3) ** 2 + 2.12 * math.log(Pr)
            q = rw * c["cp"] * ut * (Tw - Th) / (Pr * yp * torch.exp(-gam) + (2.12 * torch.log(1.0 + yp) + beta) * torch.exp(-1.0 / gam))
        F = torch.cat([torch.zeros_like(tau)[None], (pb * out + tau * up / U) * area, (-q * area)[None]])
        return (F if s == 1 else -F), tau, q

    # ---- residual, time step, step
    def residual(self, Q):
        out = []
        for b, (q, geo) in enumerate(zip(Q, self.geo)):
            c, (w, T) = self.c, self.prim(q)
            phi = torch.cat([w[1:4], T[None]])
            g = self.gradient(phi, geo)
            mu, mt = self.mu(T), w[0] * self.eddy(g[:3], geo["vol"] ** (1.0 / 3.0))
            muf, kf = mu + mt, c["cp"] * (mu / c["Pr"] + mt / c["Prt"])
            div = g[0, 0] + g[1, 1] + g[2, 2]
            vort = (g[2, 1] - g[1, 2]) ** 2 + (g[0, 2] - g[2, 0]) ** 2 + (g[1, 0] - g[0, 1]) ** 2
            theta = div ** 2 / (div ** 2 + vort + 1e-30)
            r = 0.0
            for d in range(3):
                def mean(x):
                    return 0.5 * (_cut(x, d, -1, 0) + _cut(x, d, 0, 1))
                S = geo["S"][d][tuple([slice(None)] + [slice(NG, q.shape[1 + x] - NG + (x == d)) for x in range(3)])]
                dx = _cut(geo["xc"], d, 0, 1) - _cut(geo["xc"], d, -1, 0)
                dist = (dx * dx).sum(0).sqrt()
                e, gb = dx / dist, mean(g)
                gf = gb + ((_cut(phi, d, 0, 1) - _cut(phi, d, -1, 0)) / dist - (gb * e).sum(1))[:, None] * e
                tau = gf[:3] + gf[:3].transpose(0, 1)
                tr = 2.0 / 3.0 * (gf[0, 0] + gf[1, 1] + gf[2, 2])
                ts = mean(muf) * ((tau * S).sum(1) - tr * S)
                visc = torch.cat([torch.zeros_like(tr)[None], -ts, (-(mean(phi[:3]) * ts).sum(0) - mean(kf) * (gf[3] * S).sum(0))[None]])
                F = self.inviscid(w, S, d, theta) + visc
                for s, end in enumerate(("min", "max")):
                    bc = self.layout[b][2]["ijk"[d] + end]
                    if bc[0] == "wall":
                        F.select(1 + d, 0 if s == 0 else -1).copy_(self.wall(w, T, geo, d, s, bc[1], bc[2])[0])
                r = r - (F[_at(d, slice(1, None))] - F[_at(d, slice(None, -1))])
                del gf, gb, tau, ts, visc, F
            r = r / _inner(geo["vol"])
            if self.case["kind"] == "ramp":
                qi, v, p = _inner(q), _inner(geo["vol"]), self.props
                eta = ((_inner(geo["xc"])[0] / p["L"] - SPONGE_START) / (X_RANGE[1] - SPONGE_START)).clamp(0.0, 1.0)
                sig = p["U_inf"] / p["L"] * eta ** 3 * (10.0 + eta * (-15.0 + 6.0 * eta))
                r = r - sig * (qi - (qi * v).sum(3, keepdim=True) / v.sum(2, keepdim=True))
            out.append(torch.nn.functional.pad(r, (NG,) * 6))
        return out

    def max_dt(self, Q):
        least = []
        for q, geo in zip(Q, self.geo):
            c, (w, T) = self.c, self.prim(q)
            a, lam, lamv = torch.sqrt(c["gamma"] * c["R"] * T), 0.0, 0.0
            nu = max(4.0 / 3.0, c["gamma"] / c["Pr"]) * self.mu(T) / w[0]
            for d in range(3):
                S = 0.5 * (geo["S"][d][_at(d, slice(None, -1))] + geo["S"][d][_at(d, slice(1, None))])
                A = (S * S).sum(0).sqrt()
                lam = lam + (w[1:4] * S).sum(0).abs() + a * A
                lamv = lamv + nu * A ** 2 / geo["vol"]
            least.append(_inner(0.5 * geo["vol"] / (lam + 4.0 * lamv)).min())
        return torch.stack(least).min()

    def step(self, Q, t):
        """(new state, dt, Q with the ghost cells of its residual refreshed)"""
        dt = self.max_dt(Q)
        Q = self.refresh(Q, t)
        Q1 = [q + dt * r for q, r in zip(Q, self.residual(Q))]
        Q1 = self.fill(Q1, t + float(dt))
        Q2 = [0.75 * q + 0.25 * (q1 + dt * r) for q, q1, r in zip(Q, Q1, self.residual(Q1))]
        Q2 = self.fill(Q2, t + 0.5 * float(dt))
        new = [q / 3.0 + 2.0 / 3.0 * (q2 + dt * r) for q, q2, r in zip(Q, Q2, self.residual(Q2))]
        for n, q in zip(new, Q):               # ghost cells are carried over
            keep = _inner(n).clone()
            n.copy_(q)
            _inner(n).copy_(keep)
        if self.case["kind"] == "channel":
            vols = [_inner(g["vol"]) for g in self.geo]
            shift = 1.0 - sum((_inner(n)[1] * v).sum() for n, v in zip(new, vols)) / sum(v.sum() for v in vols)
            for n in new:
                n[4] += (2.0 * n[1] * shift + shift * shift) / (2.0 * n[0])
                n[1] += shift
        return new, dt

    def output(self, Q):
        c, geo = self.c, self.geo[0]
        filled = self.fill(Q, 0.0)
        w, T = self.prim(filled[0])
        g = self.gradient(w[1:4], geo)
        mut = w[0] * self.eddy(g, geo["vol"] ** (1.0 / 3.0))
        sym, rot = 0.5 * (g + g.transpose(0, 1)), 0.5 * (g - g.transpose(0, 1))
        vort = torch.sqrt((g[1, 0] - g[0, 1]) ** 2 + (g[2, 0] - g[0, 2]) ** 2 + (g[2, 1] - g[1, 2]) ** 2)
        fields = dict(rho=w[0], velocity=w[1:4], pressure=w[4], temperature=T,
                      mach=(w[1:4] ** 2).sum(0).sqrt() / torch.sqrt(c["gamma"] * c["R"] * T), mu_t=mut, mu=self.mu(T),
                      vorticity_mag=vort, q_criterion=0.5 * ((rot ** 2).sum((0, 1)) - (sym ** 2).sum((0, 1))))
        fields = {k: _inner(v).contiguous() for k, v in fields.items()}
        u, v, z = fields["velocity"]
        planes = dict(rho=fields["rho"], u=u, v=v, w=z, uu=u * u, vv=v * v, ww=z * z, uv=u * v, uw=u * z, vw=v * z,
                      T=fields["temperature"], p=fields["pressure"])
        mean = {k: x.mean((0, 2)).cpu().numpy() for k, x in planes.items()}
        for a, b in ("uu", "vv", "ww", "uv", "uw", "vw"):
            mean[a + b] = mean[a + b] - mean[a] * mean[b]
        walls, taus = [], []
        for b, (_, _, faces) in enumerate(self.layout):
            w, T = self.prim(filled[b])
            for face in sorted(faces):
                bc = faces[face]
                if bc[0] == "wall":
                    _, tau, q = self.wall(w, T, self.geo[b], *_face(face), bc[1], bc[2])
                    walls.append(((self.layout[b][0], face), torch.stack([tau, q])))
                    taus.append(float(tau.mean()))
        return [fields, mean, sum(taus) / len(taus), [x for _, x in sorted(walls, key=lambda e: e[0])]]


def _inner_of(x, a, i):
    """Layer i of axis a, the other two axes over the interior."""
    lead = x.dim() - 3
    t = [slice(None)] * lead + [slice(NG, x.shape[lead + d] - NG) for d in range(3)]
    t[lead + a] = i
    return x[tuple(t)]


def exact(case, seed):
    if case["call"] == "batch":
        both = [_exact_one(_member(case, m), seed + 7919 * m) for m in range(case["members"])]
        # a batch hands on the next time step, a loop the last one
        return [[q for q, _, _ in both], [nxt for _, _, nxt in both]]
    return _exact_one(case, seed)[:2] if case["call"] in ("step", "advance") else _exact_one(case, seed)


def _exact_one(case, seed):
    layout, c = _layout(case), _constants(case)
    ref = _Reference(case, seed, layout, c)
    Q = _initial(case, seed, [(g["xc"], g["xc"].shape[1:]) for g in ref.geo], c)
    Q, t = ref.fill(Q, 0.0), 0.0
    if case["call"] == "rhs":
        return ref.residual(Q)
    if case["call"] == "output":
        return ref.output(Q)
    for _ in range(case["steps"]):
        Q, dt = ref.step(Q, t)
        t += float(dt)
    return [Q, dt, ref.max_dt(Q)]
