"""The work that users of this library have it do, as cases to be timed and checked.

A case is a dict of plain values.  Its "kind" is the kind of run:

``run``      one block swept by the split scheme: the state goes in as a device
             array, the time state is set, the main loop advances "steps"
             steps (two dt each), the state comes out as a device array
``blocks``   the same domain tiled by connected blocks of uneven sizes
``refined``  a blast on three refinement levels, ion MHD + neutral + dust
``unsplit``  one block advanced by the unsplit scheme
``grad``     the differentiable path: forward ("steps" steps, checkpointed) and
             backward of ``autograd.advance`` for a given cotangent, for one
             block or for "instances" independent ones stacked along z

Sizes and options are those of the repository's benchmark, tests and problem
recipes (16^3 smoke run to 256^3 turbulence, 2D Orszag-Tang to 512^2, the
Sedov blast, the three-level blast) and odd and non-cubic ones between them.

``exact`` restates the scheme in plain torch operations in 64 bits (which is
the precision the library itself computes in), cell by cell in the same
mathematical form and without any of the library's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from piernik_b200 import autograd, problems
from piernik_b200.config import BND_OUT, BND_PER, BND_REF, Setup
from piernik_b200.sim import Simulation

GAMMA = 5.0 / 3.0
F64 = torch.float64


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _case(kind, problem, n, steps, **kw):
    c = {"kind": kind, "problem": problem, "nx": n[0], "ny": n[1], "nz": n[2], "steps": steps, "limiter": "moncen",
         "interpolation": "linear", "arith": "bitexact", "cflcontrol": "none", "boundary": "periodic", "tuned": False,
         "graph": False, "instances": 1, "layout": 0}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest run (the library's smoke test): launches and latency
        dict(_case("run", "turbulence", (16, 16, 16), 2), name="mhd-16"),
        # the Sedov blast at the benchmarked size, as a program runs it that sets nothing
        dict(_case("run", "sedov", (64, 64, 64), 4, limiter="vanleer"), name="sedov-64"),
        # ordinary MHD run with the reference's step control (a step that breaks the CFL limit is redone)
        dict(_case("run", "turbulence", (128, 128, 128), 2, cflcontrol="redo"), name="mhd-128"),
        # the headline block in both arithmetics, with the tiles that the autotuner settled on
        dict(_case("run", "turbulence", (256, 256, 256), 1, tuned=True), name="mhd-256"),
        dict(_case("run", "turbulence", (256, 256, 256), 2, tuned=True, arith="fma"), name="mhd-256-fma"),
        # 2D run with long pencils
        dict(_case("run", "vortex", (512, 512, 1), 8, limiter="vanleer"), name="vortex-512"),
        # open box: outflow and reflecting walls, odd extents, gas only
        dict(_case("run", "sedov", (149, 93, 70), 1, limiter="minmod", boundary="open"), name="hd-open"),
        # one domain cut into connected blocks
        dict(_case("blocks", "turbulence", (128, 128, 128), 1, layout=3), name="blocks-128"),
        # adaptive refinement: the uneven-blocks workload, its steps replayed from a graph
        dict(_case("refined", "blast", (64, 64, 64), 1, limiter="vanleer", graph=True, layout=4), name="refined"),
        # the unsplit scheme
        dict(_case("unsplit", "turbulence", (128, 128, 128), 1, limiter="vanleer"), name="unsplit-128"),
        # gradients: the 2D vortex (launch- and latency-bound) and 3D turbulence
        dict(_case("grad", "vortex", (256, 256, 1), 6, limiter="vanleer"), name="grad-vortex-256"),
        dict(_case("grad", "turbulence", (128, 128, 128), 2), name="grad-128"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: extents over the whole range (odd ones among them),
    every limiter, both arithmetics, WENO3, graphs and step control."""
    kind = rng.choice(["run"] * 8 + ["blocks", "blocks", "unsplit", "unsplit", "grad", "grad", "grad", "refined"])
    lim = rng.choice(["vanleer", "minmod", "moncen", "superbee"])
    if kind == "run":
        problem = rng.choice(["turbulence", "turbulence", "turbulence", "vortex", "sedov", "sedov"])
        if problem == "vortex":
            n = (_log(rng, 32, 512), _log(rng, 32, 512), 1)
        else:
            n = tuple(_log(rng, 12, 224) for _ in range(3))
        return _case("run", problem, n, rng.randint(1, 2), limiter=lim,
                     interpolation=rng.choice(["linear"] * 4 + ["weno3"]),
                     arith=rng.choice(["bitexact", "bitexact", "fma"]),
                     cflcontrol=rng.choice(["none", "redo"]), graph=rng.random() < 0.25,
                     boundary=rng.choice(["periodic", "open"]) if problem == "sedov" else "periodic")
    if kind == "blocks":
        n = tuple(rng.choice([48, 64, 80, 96, 112, 128, 160]) for _ in range(3))
        return _case("blocks", "turbulence", n, 1, limiter=lim, layout=rng.randint(1, 999), graph=rng.random() < 0.5)
    if kind == "refined":
        return _case("refined", "blast", (64, 64, 64), 1, limiter=lim, layout=rng.randint(1, 999), graph=True)
    if kind == "unsplit":
        problem = rng.choice(["turbulence", "vortex"])
        n = (_log(rng, 32, 384), _log(rng, 32, 384), 1) if problem == "vortex" else tuple(_log(rng, 16, 160) for _ in range(3))
        return _case("unsplit", problem, n, rng.randint(1, 2), limiter=lim)
    problem = rng.choice(["turbulence", "vortex"])
    if problem == "vortex":
        return _case("grad", "vortex", (2 * _log(rng, 16, 256), 2 * _log(rng, 16, 256), 1), rng.randint(2, 5), limiter=lim)
    if rng.random() < 0.5:
        m = 2 * _log(rng, 8, 32)
        return _case("grad", "turbulence", (m, m, 4 * m), 2, limiter=lim, instances=4)
    return _case("grad", "turbulence", tuple(_log(rng, 12, 128) for _ in range(3)), 2, limiter=lim)


# ---------------------------------------------------------------------------
# set-ups and inputs
# ---------------------------------------------------------------------------

def _setup(case):
    n = (case["nx"], case["ny"], case["nz"])
    kw = {"n": n, "limiter": case["limiter"], "limiter_b": case["limiter"], "interpolation": case["interpolation"],
          "cflcontrol": case["cflcontrol"]}
    if case["kind"] == "unsplit":
        kw["solver"] = "unsplit"
    if case["boundary"] == "open":
        kw["bnd"] = ((BND_OUT, BND_OUT), (BND_REF, BND_OUT), (BND_REF, BND_REF))
    cell = 1.0 / 128.0                             # cubic cells, exact in binary
    box = {"xmin": (0.0, 0.0, 0.0), "xmax": tuple(cell * m for m in n)}
    if case["problem"] == "sedov":
        return Setup(fluids=[("neu", GAMMA)], magnetic=False, cfl=0.7, smalld=1.0e-3, **box, **kw)
    if case["problem"] == "vortex":
        return Setup(fluids=[("ion", GAMMA)], magnetic=True, cfl=0.8, smalld=1.0e-3, smallei=1.0e-5, **box, **kw)
    if case["problem"] == "blast":
        return Setup(fluids=[("ion", GAMMA), ("neu", 7.0 / 5.0), ("dst", -1.0)], magnetic=True, cfl=0.7, smalld=1.0e-4, **kw)
    return Setup(fluids=[("ion", GAMMA)], magnetic=True, cfl=0.5, smalld=1.0e-3, **box, **kw)


def _modes(n, rng):
    """Three real periodic fields (nz, ny, nx) of random-phase modes with
    1 <= |k| <= 4 and amplitude |k|^-2 (directions of one cell excluded)."""
    k = [torch.fft.fftfreq(m, 1.0 / m, dtype=F64, device="cuda") for m in n]
    kx = torch.fft.rfftfreq(n[0], 1.0 / n[0], dtype=F64, device="cuda")
    kk = torch.sqrt(k[2][:, None, None] ** 2 + k[1][None, :, None] ** 2 + kx[None, None, :] ** 2)
    amp = torch.where((kk >= 1) & (kk <= 4), kk.clamp(min=1.0) ** -2.0, torch.zeros_like(kk))
    out = []
    for _ in range(3):
        ph = 2 * math.pi * torch.rand(kk.shape, dtype=F64, device="cuda", generator=rng)
        out.append(torch.fft.irfftn(torch.polar(amp, ph), s=(n[2], n[1], n[0]), dim=(0, 1, 2)))
    return torch.stack(out)


def _conserved(rho, v, p, b=None, gamma=GAMMA):
    e = p / (gamma - 1.0) + 0.5 * rho * (v * v).sum(0)
    if b is None:
        return torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], e])
    e = e + 0.5 * (b * b).sum(0)
    return torch.stack([rho, rho * v[0], rho * v[1], rho * v[2], e, b[0], b[1], b[2], torch.zeros_like(rho)])


def _interior_state(case, rng):
    """The initial interior state (planes, nz, ny, nx) of a problem."""
    n = (case["nx"], case["ny"], case["nz"])
    shape = (n[2], n[1], n[0])

    def noise():
        return torch.randn(shape, dtype=F64, device="cuda", generator=rng)

    if case["problem"] == "turbulence":
        parts = []
        for _ in range(case["instances"]):
            m = (n[0], n[1], n[2] // case["instances"])
            v, a = _modes(m, rng), _modes(m, rng)
            v = v / torch.sqrt((v * v).sum(0).mean())               # rms Mach 1
            d = [(torch.roll(a, -1, 3 - k) - torch.roll(a, 1, 3 - k)) if m[k] > 2 else torch.zeros_like(a) for k in range(3)]
            b = torch.stack([d[1][2] - d[2][1], d[2][0] - d[0][2], d[0][1] - d[1][0]])
            b = b * (0.02 / torch.sqrt((b * b).sum(0).mean()))
            b[0] += 0.2
            rho = 1.0 + 0.01 * torch.randn(v.shape[1:], dtype=F64, device="cuda", generator=rng)
            parts.append(_conserved(rho, v, torch.full_like(rho, 1.0 / GAMMA), b))
        return torch.cat(parts, dim=1)
    if case["problem"] == "vortex":
        x = 2 * math.pi * (torch.arange(n[0], dtype=F64, device="cuda") + 0.5) / n[0]
        y = 2 * math.pi * (torch.arange(n[1], dtype=F64, device="cuda") + 0.5) / n[1]
        one = torch.ones(shape, dtype=F64, device="cuda")
        vx, vy = -torch.sin(y)[None, :, None] * one, torch.sin(x)[None, None, :] * one
        b0 = 1.0 / math.sqrt(4.0 * math.pi)
        b = torch.stack([b0 * vx, b0 * torch.sin(2 * x)[None, None, :] * one, torch.zeros_like(one)])
        v = torch.stack([vx, vy, torch.zeros_like(one)])
        return _conserved((25.0 / (36.0 * math.pi)) * (1.0 + 1e-3 * noise()), v, (5.0 / (12.0 * math.pi)) * one, b)
    # a point explosion, near the middle, in gas at rest
    at = torch.rand(3, dtype=F64, device="cuda", generator=rng) * 0.1 + 0.45
    ax = [torch.arange(m, dtype=F64, device="cuda") + 0.5 - at[k] * m for k, m in enumerate(n)]
    r = torch.sqrt(ax[2][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[0][None, None, :] ** 2)
    p = 1.0e-3 + 30.0 * torch.sigmoid(2.0 * (4.5 - r))
    return _conserved(1.0 + 1e-3 * noise(), torch.zeros((3,) + shape, dtype=F64, device="cuda"), p)


def _blast(setup, dom, level, off, dl0, centre, phase):
    """A refined block's state with guard cells: a hot ball in gas at rest, the
    density gently waved, uniform B, dust at rest."""
    dl = dl0 / 2 ** level
    ax = [(torch.arange(setup.ext[k], dtype=F64, device="cuda") - setup.guards[k] + 0.5 + off[k]) * (dl / dl0) for k in range(3)]
    z, y, x = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    r = torch.sqrt((x - centre[0]) ** 2 + (y - centre[1]) ** 2 + (z - centre[2]) ** 2)
    wave = 1.0 + 0.02 * torch.sin(2 * math.pi * (x / dom[0] + y / dom[1] + z / dom[2]) + phase)
    hot = torch.where(r < 4.0, torch.full_like(r, 10.0), torch.zeros_like(r))
    planes, emag = [], 0.5 * (0.1 ** 2 + 0.05 ** 2)
    for kind, gam in setup.fluids:
        rho = 0.01 * wave if kind == "dst" else wave
        planes += [rho, torch.zeros_like(r), torch.zeros_like(r), torch.zeros_like(r)]
        if kind != "dst":
            planes.append(1.0e-5 / (gam - 1.0) + hot + (emag if kind == "ion" else 0.0))
    planes += [torch.full_like(r, 0.1), torch.full_like(r, 0.05), torch.zeros_like(r), torch.zeros_like(r)]
    return torch.stack(planes)


def _cut(total, rng):
    """Uneven pieces of a connected domain's edge."""
    parts, left = [], total
    while left > 0:
        fit = [s for s in (16, 24, 32, 48, 64) if s <= left and (left - s == 0 or left - s >= 16)]
        parts.append(int(rng.choice(fit)))
        left -= parts[-1]
    return parts


def _pad(x, setup):
    """Interior state -> state with (zeroed) guard cells."""
    g = setup.guards
    return torch.nn.functional.pad(x, (g[0], g[0], g[1], g[1], g[2], g[2])).contiguous()


def _inside(x, setup):
    g, n = setup.guards, setup.n
    return x[:, g[2]:g[2] + n[2], g[1]:g[1] + n[1], g[0]:g[0] + n[0]]


def _refined_layout(case):
    """(dom, centre, [(level, off, n)]) of the three-level blast."""
    b = case["nx"]
    centre = (b // 2 + 3, b // 2 - 3, b // 2 + 1)
    r1, r2 = 52, 60
    regions = [(tuple(2 * c - r1 for c in centre), tuple(2 * c + r1 for c in centre)),
               (tuple(4 * c - r2 for c in centre), tuple(4 * c + r2 for c in centre))]
    return (b, b, b), centre, problems.refined_layout((b, b, b), regions, seed=case["layout"])


def prepare(case, seed):
    rng = torch.Generator(device="cuda")
    rng.manual_seed(seed)
    setup = _setup(case)
    st = {"case": case}
    if case["kind"] == "refined":
        dom, centre, layout = _refined_layout(case)
        dl0 = 2.0 ** -5
        phase = float(torch.rand(1, generator=rng, device="cuda")) * 2 * math.pi
        setups = [setup.replace(n=n, xmin=tuple(o * dl0 / 2 ** L for o in off),
                                xmax=tuple((o + m) * dl0 / 2 ** L for o, m in zip(off, n))) for L, off, n in layout]
        states = [_blast(s, dom, L, off, dl0, centre, phase) for s, (L, off, n) in zip(setups, layout)]
    elif case["kind"] == "blocks":
        pieces = np.random.RandomState(case["layout"])
        cuts = [_cut(m, pieces) for m in setup.n]
        full = _interior_state(case, rng)
        dom, layout, setups, states = setup.n, [], [], []
        for z0, nz in zip(np.cumsum([0] + cuts[2]), cuts[2]):
            for y0, ny in zip(np.cumsum([0] + cuts[1]), cuts[1]):
                for x0, nx in zip(np.cumsum([0] + cuts[0]), cuts[0]):
                    off, n = (int(x0), int(y0), int(z0)), (nx, ny, nz)
                    layout.append((0, off, n))
                    s = setup.replace(n=n, xmin=tuple(o * d for o, d in zip(off, setup.dl)),
                                      xmax=tuple((o + m) * d for o, m, d in zip(off, n, setup.dl)))
                    setups.append(s)
                    states.append(_pad(full[:, z0:z0 + nz, y0:y0 + ny, x0:x0 + nx], s))
    else:
        dom, layout, setups = None, None, [setup]
        x = _interior_state(case, rng)
        states = [x if case["kind"] == "grad" else _pad(x, setup)]
        if case["kind"] == "grad":
            st["cotangent"] = torch.randn(x.shape, dtype=F64, device="cuda", generator=rng)
    sim = Simulation(setups[0])
    for s in setups[1:]:
        sim.add_block(s)
    if dom is not None:
        sim.set_domain(dom)
        for i, (L, off, n) in enumerate(layout):
            sim.place_block(i, off, L)
    if case["instances"] > 1:
        sim.set_instances(case["instances"])
    if case["arith"] == "fma":
        sim.set_arithmetic("fma")
    if case["tuned"]:
        for d in range(3):
            sim.set_tile(d, 2, setup.n[d], 7)
    if case["graph"]:
        sim.use_graph()
    st.update(sim=sim, setups=setups, states=states, start=sim.time_state)
    if case["kind"] != "grad":                     # one buffer for all blocks' results
        sizes = [x.numel() for x in states]
        flat = torch.empty(sum(sizes), dtype=F64, device="cuda")
        st["flat"], st["out"] = flat, [o.view(x.shape) for o, x in zip(flat.split(sizes), states)]
    torch.cuda.synchronize()
    return st


def run(state):
    case, sim = state["case"], state["sim"]
    sim.time_state = state["start"]
    if case["kind"] == "grad":
        x = state["states"][0].detach().requires_grad_()
        out = autograd.advance(sim, x, case["steps"])
        grad, = torch.autograd.grad(out, x, grad_outputs=state["cotangent"])
        return {"state": out.detach(), "grad": grad}
    for i, x in enumerate(state["states"]):
        sim.upload_device(x.data_ptr(), block=i)
    if len(state["states"]) > 1:
        sim.update_boundaries()
    sim.run(case["steps"])
    for i, o in enumerate(state["out"]):
        sim.download_device(o.data_ptr(), block=i)
    if len(state["out"]) > 1:
        return {"states": state["flat"]}
    return {"state": _inside(state["out"][0], state["setups"][0])}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far correct results may lie apart
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: the state read and written once a step (every step ends in a
    time step that depends on all cells).  Operations: those of the scheme,
    each addition, product, quotient and root counted once: about 450 (MHD)
    or 200 (gas) per cell for one RK stage of one direction, counting
    primitives, slopes, the Riemann solver, the update and the floors."""
    if case["kind"] == "refined":
        _, _, layout = _refined_layout(case)
        cells = sum(n[0] * n[1] * n[2] for _, _, n in layout)
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    planes = {"sedov": 5, "blast": 18}.get(case["problem"], 9)
    per_stage = {"sedov": 200, "blast": 1000}.get(case["problem"], 450)
    dims = 2 if case["nz"] == 1 else 3
    stages = 2 * dims * (1 if case["kind"] == "unsplit" else 2)       # per step: one dt unsplit, two dt split
    byts, flops = 2.0 * 8 * planes * cells, float(per_stage * cells * stages)
    if case["kind"] == "grad":                     # forward, and backward with about twice the arithmetic
        byts, flops = 2.5 * byts, 3.0 * flops
    return {"bytes": byts * case["steps"], "flops": flops * case["steps"]}


def tolerance(case):
    """The default arithmetic is defined bit for bit: what it returns is
    compared exactly.  For the contracted arithmetic and the adjoint, about
    four times the largest distance from ``exact`` seen over listed and drawn
    cases: states 3.6e-16 (largest single difference 2.6e-15).  Gradients of
    smooth turbulence agree to 1e-15, but van Leer's slope 2 dl dr / (dl + dr)
    has a derivative that rounding decides where dl or dr is itself a
    rounding error (3.2e-10, 7e-8 in the vortex, which starts uniform along
    one axis), and the min / max limiters meet ties there (40 values of a
    370 x 310 vortex on the other branch: 3e-7, 1.3e-4)."""
    if case["kind"] == "grad":
        if case["limiter"] == "vanleer":
            return {"rel": 1.3e-9, "max": 3e-7}
        return {"rel": 1.2e-6, "max": 5e-4} if case["problem"] == "vortex" else {"rel": 4e-15, "max": 1e-13}
    if case["arith"] == "fma":
        return {"rel": 1.5e-15, "max": 1e-14}
    return "exact"


# ---------------------------------------------------------------------------
# the scheme in plain torch
# ---------------------------------------------------------------------------

def _abs(x):
    return torch.where(torch.signbit(x), -x, x)


def _min(a, b):
    return torch.where(b < a, b, a)


def _max(a, b):
    return torch.where(b > a, b, a)


def _sign(x):
    return torch.where(torch.signbit(x), torch.full_like(x, -1.0), torch.ones_like(x))


def _slope(lim, dl, dr):
    if lim == "vanleer":
        c = dl * dr
        up = c > 0.0
        return torch.where(up, (2.0 * c) / torch.where(up, dl + dr, torch.ones_like(c)), torch.zeros_like(c))
    s = _sign(dl) + _sign(dr)
    if lim == "minmod":
        return (s * _min(_abs(dl), _abs(dr))) * 0.5
    if lim == "moncen":
        return (s * _min(_min(2.0 * _abs(dl), 2.0 * _abs(dr)), 0.5 * _abs(dl + dr))) * 0.5
    m = torch.where(_abs(dl) > _abs(dr), _min(_abs(dl), _abs(2.0 * dr)), _min(_abs(2.0 * dl), _abs(dr)))
    return (s * 0.5) * m


def _weno3(qm, qc, qp, eps):
    b0, b1 = (qp - qc) * (qp - qc), (qc - qm) * (qc - qm)
    t = (qp - 2.0 * qc) + qm
    tau = t * t

    def side(ba, bb, near, far):
        a0, a1 = (2.0 / 3.0) * (1.0 + tau / (eps + ba)), (1.0 / 3.0) * (1.0 + tau / (eps + bb))
        return (a0 / (a0 + a1)) * (0.5 * (qc + near)) + (a1 / (a0 + a1)) * (0.5 * (3.0 * qc - far))

    return side(b0, b1, qp, qm), side(b1, b0, qm, qp)


def _spacing(x):
    a = torch.abs(x.detach())
    s = torch.exp2(torch.floor(torch.log2(torch.where(a > 0, a, torch.ones_like(a)))) - 52.0)
    return torch.where(a > 0, s, torch.full_like(a, 2.2250738585072014e-308))


def _sqrt(x):
    up = x > 0.0
    return torch.where(up, torch.sqrt(torch.where(up, x, torch.ones_like(x))), torch.zeros_like(x))


def _pick(c, a, b):
    return [torch.where(c, x, y) for x, y in zip(a, b)]


def _riemann(ql, qr, mhd, g, ch):
    """Fluxes through faces with primitive states ql, qr in swept order:
    HLLC for gas, HLLD with the GLM fluxes of B_n and psi for MHD."""
    if mhd:
        bl, br = ql[5:8], qr[5:8]
        bbl, bbr = ((b[0] * b[0] + b[1] * b[1]) + b[2] * b[2] for b in (bl, br))
    else:
        zero = torch.zeros_like(ql[0])
        bl = br = [zero, zero, zero]
        bbl = bbr = zero
    side = []
    for u, b, bb in ((ql, bl, bbl), (qr, br, bbr)):
        pr = u[4] + 0.5 * bb
        en = ((u[4] / (g - 1.0)) + ((0.5 * u[0]) * ((u[1] * u[1] + u[2] * u[2]) + u[3] * u[3]))) + 0.5 * bb
        gp = g * u[4]
        if mhd:
            a = gp + bb
            c = (a + _sqrt(a * a - ((4.0 * gp) * (b[0] * b[0])))) / u[0]
        else:
            c = gp / u[0]
        f = [u[0] * u[1], (u[0] * (u[1] * u[1]) + pr) - b[0] * b[0], (u[0] * u[2]) * u[1] - b[0] * b[1],
             (u[0] * u[3]) * u[1] - b[0] * b[2],
             (en + pr) * u[1] - b[0] * ((u[1] * b[0] + u[2] * b[1]) + u[3] * b[2])]
        if mhd:
            f += [b[1] * u[1] - b[0] * u[2], b[2] * u[1] - b[0] * u[3]]
        cons = [u[0], u[0] * u[1], u[0] * u[2], u[0] * u[3], en] + ([b[1], b[2]] if mhd else [])
        side.append((u, b, pr, en, c, f, cons))
    (ul, bl, prl, enl, cl, fl, ucl), (ur, br, prr, enr, cr, fr, ucr) = side
    cf = torch.sqrt((0.5 if mhd else 1.0) * _max(cl, cr))
    sl, sr = _min(ul[1], ur[1]) - cf, _max(ul[1], ur[1]) + cf
    left, right = sl >= 0.0, sr <= 0.0
    mid = ~(left | right)
    one = torch.ones_like(sl)
    auxl, auxr = (sl - ul[1]) * ul[0], (sr - ur[1]) * ur[0]
    flat = _abs(auxr - auxl) < _spacing(auxr + auxl)
    sm = torch.where(flat, (sl + sr) / 2.0, ((auxr * ur[1] - prr) - (auxl * ul[1] - prl)) / torch.where(flat, one, auxr - auxl))
    sm = torch.where(mid, sm, 0.5 * (sl + sr))
    dnl, dnr = ul[0] * (sl - ul[1]), ur[0] * (sr - ur[1])
    prt = 0.5 * ((prl + dnl * (sm - ul[1])) + (prr + dnr * (sm - ur[1])))
    blr = bl[0] * br[0]
    if mhd:
        hll = [((sr * br[k] - sl * bl[k]) - (fr[4 + k] - fl[4 + k])) / (sr - sl) for k in (1, 2)]
    star = []
    for u, b, pr, en, s, dn in ((ul, bl, prl, enl, sl, dnl), (ur, br, prr, enr, sr, dnr)):
        ssm, svx = torch.where(mid, s - sm, one), s - u[1]
        if mhd:
            co = dn * ssm - blr
            ok = (_abs(co) > _spacing(blr)) & (blr / g <= u[4])
            a, cs = dn * svx - blr, torch.where(ok, co, one)
            bs = [b[0]] + [torch.where(ok, (b[k] * a) / cs, hll[k - 1]) for k in (1, 2)]
            k = b[0] / torch.where(mid, dn, one)
            vs = [sm, u[2] + k * (b[1] - bs[1]), u[3] + k * (b[2] - bs[2])]
            vb, vbs = ((v[0] * x[0] + v[1] * x[1]) + v[2] * x[2] for v, x in ((u[1:4], b), (vs, bs)))
            e = ((((svx * en) - (pr * u[1])) + (prt * sm)) + (b[0] * (vb - vbs))) / ssm
        else:
            bs, vs, vbs = None, [sm, u[2], u[3]], None
            e = (((svx * en) - (pr * u[1])) + (prt * sm)) / ssm
        d = dn / ssm
        star.append(([d, d * vs[0], d * vs[1], d * vs[2], e] + (bs[1:] if mhd else []), vs, bs, vbs))
    (usl, vsl, bsl, vbl), (usr, vsr, bsr, vbr) = star
    stl = [f + sl * (s - c) for f, s, c in zip(fl, usl, ucl)]
    str_ = [f + sr * (s - c) for f, s, c in zip(fr, usr, ucr)]
    both = [0.5 * (((a + sl * (s - c)) + b) + sr * (t - d)) for a, s, c, b, t, d in zip(fl, usl, ucl, fr, usr, ucr)]
    out = _pick(sm > 0.0, stl, _pick(sm < 0.0, str_, both))
    if mhd:
        dl, dr = (torch.where(mid, x, one) for x in (usl[0], usr[0]))
        rl, rr = torch.sqrt(dl), torch.sqrt(dr)
        al, ar = sm - _abs(bl[0]) / rl, sm + _abs(br[0]) / rr
        sg = torch.where(bl[0] >= 0.0, one, -one)
        v2 = [sm] + [((rl * vsl[k] + rr * vsr[k]) + sg * (bsr[k] - bsl[k])) / (rl + rr) for k in (1, 2)]
        b2 = [0.5 * (bl[0] + br[0])] + [((rl * bsr[k] + rr * bsl[k]) + (sg * (rl * rr)) * (vsr[k] - vsl[k])) / (rl + rr) for k in (1, 2)]
        vb2 = (v2[0] * b2[0] + v2[1] * b2[1]) + v2[2] * b2[2]

        def alfven(f, us, uc, s, a, e):
            u2 = [us[0], us[0] * v2[0], us[0] * v2[1], us[0] * v2[2], e, b2[1], b2[2]]
            return [((x + a * p) - (a - s) * q) - s * c for x, p, q, c in zip(f, u2, us, uc)]

        fal = alfven(fl, usl, ucl, sl, al, usl[4] - (sg * rl) * (vbl - vb2))
        far = alfven(fr, usr, ucr, sr, ar, usr[4] + (sg * rr) * (vbr - vb2))
        inner = _pick(sm > 0.0, fal, _pick(sm < 0.0, far, [0.5 * (a + b) for a, b in zip(fal, far)]))
        inner = _pick(al > 0.0, stl, _pick(ar < 0.0, str_, inner))
        out = _pick(_abs(bl[0]) > 0.0, inner, out)
    out = _pick(left, fl, _pick(right, fr, out))
    if not mhd:
        return out
    psl, psr = ql[8], qr[8]
    return out[:5] + [0.5 * ((psr + psl) - ch * (br[0] - bl[0])), out[5], out[6],
                      ((ch * ch) * 0.5) * ((br[0] + bl[0]) - (psr - psl) / ch)]


class _Scheme:
    """The split and unsplit schemes on a list of interior planes [z, y, x]."""

    def __init__(self, setup):
        self.s, self.mhd, self.g = setup, setup.magnetic, setup.fluids[0][1]
        self.dirs = [d for d in range(3) if setup.n[d] > 1]
        self.mdl = min(setup.dl[d] for d in self.dirs)

    def swept(self, u, d):
        """Planes in the order of a sweep along d (the order is its own inverse)."""
        p = ((0, 1, 2), (1, 0, 2), (2, 1, 0))[d]
        out = [u[0]] + [u[1 + k] for k in p] + [u[4]]
        return out + ([u[5 + k] for k in p] + [u[8]] if self.mhd else [])

    def widened(self, x, d, v):
        """Two guard cells on either side of plane v (swept order) along d."""
        ax, n = 2 - d, x.shape[2 - d]
        lo, hi = self.s.bnd[d]
        if lo == BND_PER:
            return torch.cat([x.narrow(ax, n - 2, 2), x, x.narrow(ax, 0, 2)], ax)
        ends = []
        for kind, at, in_order in ((lo, (1, 0), False), (hi, (n - 1, n - 2), True)):
            if kind == BND_OUT:
                e = x.narrow(ax, at[0] if in_order else 0, 1)
                e = torch.cat([e, e], ax)
            else:
                e = torch.cat([x.narrow(ax, k, 1) for k in at], ax)
                e = -e if v == 1 else e
            ends.append(e)
        return torch.cat([ends[0], x, ends[1]], ax)

    def fluxes(self, u, d, ch):
        """Swept-order fluxes through the n + 1 faces along d from swept planes u."""
        ax = 2 - d
        w = [self.widened(x, d, v) for v, x in enumerate(u)]
        q = [w[0], w[1] / w[0], w[2] / w[0], w[3] / w[0]]
        ek = (0.5 * ((w[1] * w[1] + w[2] * w[2]) + w[3] * w[3])) / w[0]
        p = (self.g - 1.0) * (w[4] - ek)
        if self.mhd:
            p = p - (0.5 * (self.g - 1.0)) * ((w[5] * w[5] + w[6] * w[6]) + w[7] * w[7])
        q += [p] + w[5:]
        ql, qr = [], []
        for v, x in enumerate(q):
            m = x.shape[ax] - 2
            qm, qc, qp = (x.narrow(ax, k, m) for k in range(3))
            if self.s.interpolation == "weno3":
                a, b = _weno3(qm, qc, qp, self.s.w_epsilon)
            else:
                h = 0.5 * _slope(self.s.limiter_b if v >= 5 else self.s.limiter, qc - qm, qp - qc)
                a, b = qc + h, qc - h
            ql.append(a.narrow(ax, 0, m - 1))
            qr.append(b.narrow(ax, 1, m - 1))
        return _riemann(ql, qr, self.mhd, self.g, ch)

    def floored(self, u):
        u = [x + 0.0 for x in u[:5]] + u[5:]
        u[0] = _max(u[0], torch.full_like(u[0], self.s.smalld))
        kin = (0.5 * ((u[1] * u[1] + u[2] * u[2]) + u[3] * u[3])) / u[0]
        e = u[4] - kin
        if self.mhd:
            mag = 0.5 * ((u[5] * u[5] + u[6] * u[6]) + u[7] * u[7])
            e = e - mag
        e = _max(e, torch.full_like(e, self.s.smallei)) + kin
        u[4] = e + mag if self.mhd else e
        return u

    def stage(self, u0, u, d, c, ch):
        f = self.fluxes(u, d, ch)
        ax, n = 2 - d, u[0].shape[2 - d]
        return self.floored([x + c * (y.narrow(ax, 0, n) - y.narrow(ax, 1, n)) for x, y in zip(u0, f)])

    def sweep(self, d, dt, ch, fac, *u):
        u = self.swept(u, d)
        h = self.stage(u, u, d, (0.5 * dt) / self.s.dl[d], ch)
        u = self.stage(u, h, d, dt / self.s.dl[d], ch)
        if self.mhd:
            u[8] = u[8] * fac
        return tuple(self.swept(u, d))

    def time_step(self, u, dt_old):
        u = [x.detach() for x in u]
        v = [torch.abs(u[1 + d] / u[0]) for d in range(3)]
        ek = (0.5 * ((u[1] * u[1] + u[2] * u[2]) + u[3] * u[3])) / u[0]
        if self.mhd:
            pm = 0.5 * ((u[5] * u[5] + u[6] * u[6]) + u[7] * u[7])
            p = ((u[4] - ek) * (self.g - 1.0) + (2.0 - self.g) * pm) - pm
            cs = torch.sqrt(torch.abs((2.0 * pm + self.g * p) / u[0]))
        else:
            cs = torch.sqrt(torch.abs((self.g * ((u[4] - ek) * (self.g - 1.0))) / u[0]))
        dt = self.s.cfl * min(self.s.dl[d] / float((v[d] + cs).max()) for d in self.dirs)
        dt = dt if dt_old is None else min(dt, 2.0 * dt_old)
        ch = (self.s.cfl_glm * self.mdl) / dt
        return dt, ch

    def damping(self, ch, dt):
        return math.exp(-(self.s.glm_alpha * ch) / (self.mdl / dt))

    def split(self, u, steps, remember=False):
        dt = None
        for _ in range(steps):
            dt, ch = self.time_step(u, dt)
            for order in (self.dirs, self.dirs[::-1]):
                for k, d in enumerate(order):
                    fac = self.damping(ch, dt) if k == len(order) - 1 else 1.0
                    if remember:
                        u = torch.utils.checkpoint.checkpoint(self.sweep, d, dt, ch, fac, *u, use_reentrant=False)
                    else:
                        u = self.sweep(d, dt, ch, fac, *u)
        return list(u)

    def unsplit(self, u, steps):
        u, dt = list(u), None
        for _ in range(steps):
            dt, ch = self.time_step(u, dt)
            fac = self.damping(ch, dt / 2.0)
            if self.mhd:
                u[8] = u[8] * fac
            at = u
            for rk, last in ((0.5, False), (1.0, True)):
                new = list(u)
                for d in self.dirs:
                    f = self.swept(self.fluxes(self.swept(at, d), d, ch), d)
                    ax, n, c = 2 - d, self.s.n[d], (dt / self.s.dl[d]) * rk
                    new = [x + c * (y.narrow(ax, 0, n) - y.narrow(ax, 1, n)) for x, y in zip(new, f)]
                new = [x + 0.0 for x in new[:5]] + new[5:]
                for d in self.dirs if last else []:
                    new = self.swept(self.floored(self.swept(new, d)), d)
                at = new
            u = at
            if self.mhd:
                u[8] = u[8] * fac
        return u


def exact(case, seed):
    """The outputs of ``run`` from plain torch operations; None for the
    refined domain, whose per-block multi-level form takes minutes so."""
    if case["kind"] == "refined":
        return None
    setup = _setup(case)
    st = prepare(case, seed)
    if case["kind"] == "blocks":                   # one periodic domain, cut again at the end
        full = torch.empty((9, setup.n[2], setup.n[1], setup.n[0]), dtype=F64, device="cuda")
        at = [tuple(int(round(a / d)) for a, d in zip(s.xmin, setup.dl)) for s in st["setups"]]
        for s, o, x in zip(st["setups"], at, st["states"]):
            full[:, o[2]:o[2] + s.n[2], o[1]:o[1] + s.n[1], o[0]:o[0] + s.n[0]] = _inside(x, s)
        new = torch.stack(_Scheme(setup).split(list(full), case["steps"]))
        index = [torch.arange(-4, m + 4, device="cuda") % m for m in setup.n]
        parts = [new[:, index[2][o[2]:o[2] + s.ext[2]]][:, :, index[1][o[1]:o[1] + s.ext[1]]]
                 [:, :, :, index[0][o[0]:o[0] + s.ext[0]]].reshape(-1) for s, o in zip(st["setups"], at)]
        return {"states": torch.cat(parts)}
    if case["kind"] == "grad":
        m = setup.n[2] // case["instances"]
        one = _Scheme(setup.replace(n=(setup.n[0], setup.n[1], m), xmax=(setup.xmax[0], setup.xmax[1], m / 128.0)))
        outs, grads = [], []
        for i in range(case["instances"]):
            x = st["states"][0][:, i * m:(i + 1) * m].clone().requires_grad_()
            out = torch.stack(one.split(list(x), case["steps"], remember=True))
            g, = torch.autograd.grad(out, x, grad_outputs=st["cotangent"][:, i * m:(i + 1) * m])
            outs.append(out.detach())
            grads.append(g)
        return {"state": torch.cat(outs, 1), "grad": torch.cat(grads, 1)}
    scheme = _Scheme(setup)
    u = list(_inside(st["states"][0], setup))
    u = scheme.unsplit(u, case["steps"]) if case["kind"] == "unsplit" else scheme.split(u, case["steps"])
    return {"state": torch.stack(u)}
