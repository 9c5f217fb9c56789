"""The performance cases of the GAMERA step: what a program has this framework do, through its public front end
(kaiju_b200.gamera and the problem set-ups beside it), over the range of sizes, options and precisions it is used
with. Every stepping case is one coupling or output interval of a host program: some steps on the device, then the
state (Gas, magFlux, Bxyz, ghosts included) in the host's page-locked Fortran-layout arrays, where the next
component or the writer reads it. The problems are the repository's own: the Orszag-Tang vortex and the warped
blast wave, the magnetosphere on its LFM grid, the Kelvin-Helmholtz ensemble, and decaying turbulence with the
learned closure attached and in training.
"""
import math

import numpy as np
import torch

from kaiju_b200 import closure_train as ct
from kaiju_b200 import gamera as gm
from kaiju_b200 import magnetosphere as ms
from kaiju_b200 import turbulence as tu

NG = 4
GAMMA = 5.0 / 3.0
TINY = 1.0e-12
# End times of the runs. CalcDT clamps dt to them, so a run that is stepped past its end stays in its final state.
T_END = {"ot": 1.0, "bw": 0.25, "msph": 2.0, "kh": 2.0}
# Kelvin-Helmholtz member widths, repeated over the members of an ensemble
KH_SIZES = (512, 64, 128, 256, 64, 128, 64, 256)


def listed():
    return [
        # a small problem stepped one call at a time by a host that looks at dt and t after each step
        # (launches and latency count)
        dict(name="ot_32x32x4_fp64_step", kind="ot", ni=32, nj=32, nk=4, prec="fp64", rmeth="8CENT", steps=10, each=True),
        # the Orszag-Tang configuration at its own size, steps issued together
        dict(name="ot_128x128x4_fp64", kind="ot", ni=128, nj=128, nk=4, prec="fp64", rmeth="8CENT", steps=20, each=False),
        # 2.5D, the size of the accuracy cases
        dict(name="ot_256x256x1_fp64_7up", kind="ot", ni=256, nj=256, nk=1, prec="fp64", rmeth="7UP", steps=20, each=False),
        # 3-D periodic, sizes that are no multiples of the tiles, single-precision fluxes
        dict(name="ot_96x83x70_fp32", kind="ot", ni=96, nj=83, nk=70, prec="fp32flux", rmeth="8CENT", steps=10, each=False),
        # curvilinear grid, ragged, the 7-point upwind reconstruction
        dict(name="bw_72x57x45_fp64_7up", kind="bw", ni=72, nj=57, nk=45, prec="fp64", rmeth="7UP", steps=10, each=False),
        # the headline problem: the 256^3 blast wave on the warped grid, in both precisions
        dict(name="bw_256_fp64", kind="bw", ni=256, nj=256, nk=256, prec="fp64", rmeth="8CENT", steps=20, each=False),
        dict(name="bw_256_fp32", kind="bw", ni=256, nj=256, nk=256, prec="fp32flux", rmeth="8CENT", steps=20, each=False),
        # the magnetosphere at the configuration's size: background dipole, Boris, rings, hooks
        dict(name="msph_96x96x128_fp64", kind="msph", ni=96, nj=96, nk=128, prec="fp64", rmeth="7UP", steps=10, each=False),
        # a smaller magnetosphere with single-precision fluxes
        dict(name="msph_48x42x64_fp32", kind="msph", ni=48, nj=42, nk=64, prec="fp32flux", rmeth="7UP", steps=10, each=False),
        # many small problems of uneven sizes advanced together
        dict(name="kh_24_fp32", kind="kh", members=24, prec="fp32flux", steps=20),
        # a turbulence run with the learned closure in every step
        dict(name="closure_step_128", kind="closure_step", n=128, prec="fp64", steps=10),
        # training the closure: forward, loss, backward and Adam on captured samples
        dict(name="closure_train_32", kind="closure_train", n=32, slots=4, steps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ot", "ot", "ot", "bw", "bw", "bw", "msph", "msph", "kh", "closure_step", "closure_train"])
    prec = rng.choice(["fp64", "fp32flux"])
    rmeth = rng.choice(["8CENT", "7UP"])
    if kind == "ot":
        ni, nj = 8 * _log(rng, 2, 32), _log(rng, 12, 256)
        nk = rng.choice([1, 4, _log(rng, 4, 128)])
        return dict(kind="ot", ni=ni, nj=nj, nk=nk, prec=prec, rmeth=rmeth, steps=rng.randint(5, 20),
                    each=bool(rng.randint(0, 1)))
    if kind == "bw":
        return dict(kind="bw", ni=8 * _log(rng, 3, 32), nj=_log(rng, 20, 256), nk=_log(rng, 20, 256), prec=prec,
                    rmeth=rmeth, steps=rng.randint(5, 20), each=False)
    if kind == "msph":
        return dict(kind="msph", ni=8 * rng.randint(4, 12), nj=rng.randint(24, 96), nk=rng.choice([32, 64, 128]),
                    prec=prec, rmeth="7UP", steps=rng.randint(5, 15), each=False)
    if kind == "kh":
        return dict(kind="kh", members=rng.randint(3, 24), prec=prec, steps=rng.randint(8, 20))
    if kind == "closure_step":
        return dict(kind="closure_step", n=8 * rng.randint(4, 16), prec=prec, steps=rng.randint(4, 10))
    return dict(kind="closure_train", n=8 * rng.randint(2, 5), slots=rng.randint(2, 6), steps=rng.randint(4, 12))


# ------------------------------------------------------------------------------------------ inputs
def _pinned(shape, dtype=torch.float64):
    """A page-locked Fortran-order host array, as a host program keeps for the state."""
    t = torch.empty(int(np.prod(shape)), dtype=dtype, pin_memory=torch.cuda.is_available())
    return t.numpy().reshape(shape, order="F")


def _ot_bounds(case):
    return (0.0, 1.0, 0.0, 1.0, 0.0, case["nk"] / 128.0) if case["nk"] > 1 else (0.0, 1.0, 0.0, 1.0, -0.5, 0.5)


def _ot_fields(case, seed):
    """The Orszag-Tang vortex with seeded phases and a weak seeded third dimension, on the active cells: Gas and the
    lower face fluxes (circulations of an edge potential, so each cell's flux sum vanishes to rounding)."""
    rng = np.random.default_rng(seed)
    px, py, pz, pb = rng.uniform(0.0, 1.0, 4)
    n = (case["ni"], case["nj"], case["nk"])
    b = _ot_bounds(case)
    h = [(b[2 * d + 1] - b[2 * d]) / n[d] for d in range(3)]
    x, y, z = np.meshgrid(*[(np.arange(m) + 0.5) / m for m in n], indexing="ij")
    tp = 2.0 * np.pi
    rho = 25.0 / (36.0 * np.pi) * (1.0 + 0.1 * np.cos(tp * (x + y + px)))
    P = np.full(n, 5.0 / (12.0 * np.pi))
    wz = 0.05 if case["nk"] > 1 else 0.0
    v = [-np.sin(tp * (y + py)) * (1.0 + wz * np.cos(tp * (z + pz))), np.sin(tp * (x + px)),
         0.2 * np.sin(tp * (x + pb)) * np.cos(tp * y)]
    E = P / (GAMMA - 1.0) + 0.5 * rho * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
    gas = np.stack([rho, rho * v[0], rho * v[1], rho * v[2], E], axis=-1)
    # edge potentials at the lower edges (x and y at corners), times the edge length
    cx, cy, cz = np.meshgrid(*[np.arange(m) / m for m in n], indexing="ij")
    B0 = 1.0 / math.sqrt(4.0 * math.pi)
    Az = (B0 / (2.0 * tp) * np.cos(2.0 * tp * (cx + pb)) + B0 / tp * np.cos(tp * (cy + py))) * h[2]
    Ax = 0.03 * B0 / tp * np.sin(tp * cy) * np.cos(tp * (x + px)) * h[0]
    Ay = 0.03 * B0 / tp * np.cos(tp * cx) * np.sin(tp * (y + pz)) * h[1]
    up = lambda a, d: np.roll(a, -1, axis=d)  # noqa: E731
    mf = np.stack([up(Az, 1) - Az - up(Ay, 2) + Ay, up(Ax, 2) - Ax - up(Az, 0) + Az, up(Ay, 0) - Ay - up(Ax, 1) + Ax],
                  axis=-1)
    return gas, mf, h


def _ghosts(gas, mf):
    """Periodic ghost layers: Gas (4 each side) and the face fluxes (one more layer above)."""
    g = np.asfortranarray(np.pad(gas, ((NG, NG),) * 3 + ((0, 0),), mode="wrap"))
    m = np.asfortranarray(np.pad(mf, ((NG, NG + 1),) * 3 + ((0, 0),), mode="wrap"))
    return g, m


def _warped(case, seed):
    """Corners of the blast wave's non-orthogonal grid (corners_warped with a seeded amplitude near 0.04)."""
    amp = 0.03 + 0.02 * np.random.default_rng(seed).uniform()
    n = (case["ni"], case["nj"], case["nk"])
    c = [-0.5 + np.arange(-NG, m + NG + 1) / m for m in n]
    s = [np.sin(2.0 * np.pi * q) for q in c]
    xyz = np.empty(tuple(len(q) for q in c) + (3,), order="F")
    ax = ((slice(None), None, None), (None, slice(None), None), (None, None, slice(None)))
    for d in range(3):
        e, f = (d + 1) % 3, (d + 2) % 3
        xyz[..., d] = c[d][ax[d]] + amp * (s[e][ax[e]] * s[f][ax[f]])
    return xyz


def _model(case, bc):
    return gm.Model(case["ni"], case["nj"], case["nk"], CFL=0.3, tFin=T_END[case["kind"]], rmeth=case["rmeth"], bc=(bc,) * 6)


def _precision(g, case):
    if case["prec"] == "fp32flux":
        g.set_precision(gm.GAM_FP32FLUX)


def _state_out(g):
    """The host's arrays for the state of one problem."""
    return {k: _pinned(g.shapes[k]) for k in ("gas", "magflux", "bxyz")}


def _closure(n, seed, stats):
    """A closure as it is before training: seeded weights, inputs normalised to the run's statistics."""
    c = gm.Closure(n, n, n, seed=seed)
    c.in_mean, c.in_std = stats
    c.set_norm(c.in_mean, c.in_std, np.full(8, 2.0e-3), np.full(5, 1.0e-3))
    c.set_norm_emf(np.full(3, 2.0e-3), np.full(3, 1.0e-4))
    return c


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ot":
        model = _model(case, gm.GAM_BC_PERIODIC)
        g = gm.GameraGPU.from_corners(model, gm.corners_uniform(model, _ot_bounds(case)), "OT2D")
        gas, mf = _ghosts(*_ot_fields(case, seed)[:2])
        g.sync_to_device(gas=gas, magflux=mf, ogas=gas, omagflux=mf, time=0.0, otime=0.0)
        g.init_dt()
    elif kind == "bw":
        g = gm.GameraGPU.from_corners(_model(case, gm.GAM_BC_ZEROGRAD), _warped(case, seed), "BW")
    elif kind == "msph":
        u = np.random.default_rng(seed).uniform(-1.0, 1.0, 3)
        wind = ms.Magnetosphere(wind_density=5.0 + u[0], wind_velocity=(-4.0e5 * (1.0 + 0.1 * u[1]), 0.0, 0.0),
                                wind_field=(0.0, 0.0, -5.0 + u[2]))
        g = ms.magnetosphere_problem((case["ni"], case["nj"], case["nk"]), wind, tFin=T_END["msph"])
    elif kind == "kh":
        rng = np.random.default_rng(seed)
        par = [dict(nx=KH_SIZES[m % len(KH_SIZES)], a=rng.uniform(0.01, 0.05), Bx=rng.uniform(0.0, 0.2), amp=0.01,
                    seed=m + (seed % 1000) * 64) for m in range(case["members"])]
        mem = [gm.kh_member(p, case["prec"] == "fp32flux", tFin=T_END["kh"]) for p in par]
        out = [{k: _pinned(g.shapes[k]) for k in ("gas", "magflux")} for g in mem]
        return dict(case=case, mem=mem, ens=gm.Ensemble(mem), out=out)
    elif kind == "closure_step":
        g = tu.turbulence_problem(case["n"], seed % (1 << 31))
        c = _closure(case["n"], seed % (1 << 31), ct.primitive_stats(g))
        _precision(g, case)
        g.set_closure(c)
        return dict(case=case, g=g, closure=c, out=_state_out(g))
    else:
        n = case["n"]
        c = _closure(n, seed % (1 << 31), (np.zeros(8), np.ones(8)))
        c.reserve(case["slots"])
        slots = ct.collect(c, n, [seed % (1 << 31)], case["slots"], 2, 0)
        ct.set_output_norm(c, n, slots)
        return dict(case=case, closure=c, slots=[slots[s % len(slots)] for s in range(case["steps"])])
    _precision(g, case)
    return dict(case=case, g=g, out=_state_out(g))


def run(state):
    case = state["case"]
    if case["kind"] == "closure_train":
        c = state["closure"]
        loss = c.train(state["slots"], 1.0e-3)
        return dict(loss=loss, params=c.params(), grads=c.grads())
    if case["kind"] == "kh":
        state["ens"].run_steps(case["steps"])
        for g, o in zip(state["mem"], state["out"]):
            g.sync_to_host(**o)
        return state["out"]
    g, out = state["g"], state["out"]
    if case.get("each"):
        for _ in range(case["steps"]):
            dt, ts, t = g.step()
    else:
        g.run_steps(case["steps"])
    g.sync_to_host(**out)
    return out


# ------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Per zone and step: State n and n-1 in and n+1 out (24 doubles) and the grid metrics once (88 values, in the
    precision of the fluxes), about 3.1 kflop; and the state written to the host's arrays once per pass."""
    kind = case["kind"]
    if kind == "closure_train":
        z = case["n"] ** 3
        net = 2 * 27 * (8 * 32 + 2 * 32 * 32 + 32 * 27)
        return {"bytes": float(case["steps"] * z * 4 * (8 + 8)), "flops": float(case["steps"] * z * 3 * net)}
    b = 24 * 8 + 88 * (8 if case["prec"] == "fp64" else 4)
    f = 3100
    if kind == "kh":
        sizes = [KH_SIZES[m % len(KH_SIZES)] for m in range(case["members"])]
        z = sum(n * (n // 2) * 4 for n in sizes)
        out = sum((n + 8) * (n // 2 + 8) * 12 * 8 * 8 for n in sizes)
    else:
        n = (case["n"],) * 3 if kind == "closure_step" else (case["ni"], case["nj"], case["nk"])
        z = n[0] * n[1] * n[2]
        out = (n[0] + 8) * (n[1] + 8) * (n[2] + 8) * 11 * 8
        if kind == "closure_step":
            f += 2 * 27 * (8 * 32 + 2 * 32 * 32 + 32 * 27)
        if kind == "msph":
            b += 24 * (8 if case["prec"] == "fp64" else 4)   # the background field's planes
    return {"bytes": float(case["steps"] * z * b + out), "flops": float(case["steps"] * z * f)}


def tolerance(case):
    """From the largest difference seen when the same pass is taken from a state (or weights) whose values are off in
    the last places, over one and two passes, and for single-precision fluxes when the fluxes are taken in double
    precision (fp64 4.6e-13, fp32flux 7.2e-7, closure steps 3.3e-6, gradients in training 6.4e-3)."""
    if case["kind"] == "closure_train":   # 16-bit activations; the gradients of the last of several Adam steps
        return {"rel": 2.5e-2, "max": 0.9}
    if case["kind"] == "closure_step":    # the corrections of a 16-bit net are about 1e-3 of the fluxes
        return {"rel": 1.0e-5, "max": 2.0e-4}
    if case["prec"] == "fp32flux":
        return {"rel": 3.0e-6, "max": 6.0e-5}
    return {"rel": 1.0e-11, "max": 5.0e-10}


# ------------------------------------------------------------------------------------------ the step in 64 bits
def _w8(dev):
    return torch.tensor([-3.0, 29.0, -139.0, 533.0, 533.0, -139.0, 29.0, -3.0], dtype=torch.float64, device=dev) / 840.0


_U7 = [-3.0, 25.0, -101.0, 319.0, 214.0, -38.0, 4.0]


def _at(q, d, m):
    """q of the m-th neighbour along axis d (periodic)"""
    return torch.roll(q, -m, dims=d)


def _recon8(q, d):
    w = _w8(q.device)
    return sum(w[m] * _at(q, d, m - 4) for m in range(8))


def _left_right(q, lim, d, rmeth, pdmb):
    """Left and right values on the lower d face of each cell: high-order interpolation of q, limited by PDM with lim."""
    v = [_at(lim, d, m - 2) for m in range(4)]
    lo, hi = torch.minimum(v[1], v[2]), torch.maximum(v[1], v[2])
    sgn = lambda a: torch.where(torch.signbit(a), -1.0, 1.0)  # noqa: E731
    s0, s1, s2 = (sgn(pdmb * (v[m + 1] - v[m])) for m in range(3))
    q0, q1 = (s0 + s1).abs() * (pdmb * (v[1] - v[0])).abs(), (s1 + s2).abs() * (pdmb * (v[3] - v[2])).abs()
    if rmeth == "8CENT":
        f = torch.maximum(lo, torch.minimum(_recon8(q, d), hi))
        return f - s1 * ((f - v[1]).abs() - q0).clamp(min=0.0), f + s1 * ((v[2] - f).abs() - q1).clamp(min=0.0)
    ql = sum(_U7[m] / 420.0 * _at(q, d, m - 4) for m in range(7))
    qr = sum(_U7[m] / 420.0 * _at(q, d, 3 - m) for m in range(7))
    ql, qr = (torch.maximum(lo, torch.minimum(a, hi)) for a in (ql, qr))
    return ql - s1 * ((ql - v[1]).abs() - q0).clamp(min=0.0), qr + s1 * ((v[2] - qr).abs() - q1).clamp(min=0.0)


def _prim(U):
    rho = U[0]
    V = [U[1] / rho, U[2] / rho, U[3] / rho]
    ke = 0.5 * rho * (V[0] ** 2 + V[1] ** 2 + V[2] ** 2)
    return [rho.clamp(min=TINY)] + V + [((GAMMA - 1.0) * (U[4] - ke)).clamp(min=TINY)]


def _cell_b(mf, area):
    return [0.5 * (mf[d] + _at(mf[d], d, 1)) / area[d] for d in range(3)]


def _wrap(q, lo, hi):
    """q with lo and hi periodic layers below and above along every axis"""
    for d in range(3):
        q = q.index_select(d, torch.arange(-lo, q.shape[d] + hi, device=q.device) % q.shape[d])
    return q


def _curl(E):
    return [_at(E[2], 1, 1) - E[2] - _at(E[1], 2, 1) + E[1], _at(E[0], 2, 1) - E[0] - _at(E[2], 0, 1) + E[2],
            _at(E[1], 0, 1) - E[1] - _at(E[0], 1, 1) + E[0]]


def _next_dt(U, oU, omf, E, dt, area, h):
    """CalcDT runs before the boundary conditions, over the active cells and one ghost layer: its gas and most of its
    face fluxes are still those of the step before, and the faces on the upper sides have taken the edges beyond
    them, where E is not computed, as zero."""
    n = U[0].shape
    a, f = tuple(slice(1, m + 1) for m in n), tuple(slice(1, m + 2) for m in n)
    g, m = [_wrap(q, 1, 1) for q in oU], [_wrap(q, 1, 2) for q in omf]
    for q, new in zip(g, U):
        q[a] = new
    edge = []
    for e in range(3):
        q = torch.zeros(tuple(k + 2 for k in n), dtype=E[e].dtype, device=E[e].device)
        box = tuple(slice(0, k + (d != e)) for d, k in enumerate(n))
        q[box] = _wrap(E[e], 0, 1)[box]
        edge.append(q)
    inner = tuple(slice(0, k + 1) for k in n)
    for q, c in zip(m, _curl(edge)):
        q[f] = q[f] - dt * c[inner]
    b = []
    for d in range(3):
        lo = [slice(0, k + 2) for k in n]
        hi = list(lo)
        hi[d] = slice(1, n[d] + 3)
        b.append(0.5 * (m[d][tuple(lo)] + m[d][tuple(hi)]) / area[d])
    return _dt(g, b, h)


def _dt(U, b, h):
    rho = U[0]
    v2 = (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / rho ** 2
    P = (GAMMA - 1.0) * (U[4] - 0.5 * rho * v2)
    fast = torch.sqrt(GAMMA * P / rho + (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) / rho)
    return float((0.3 * min(h) / (torch.sqrt(v2) + fast)).min())


def _exact_ot(case, seed):
    """The step on a uniform periodic grid, where every face triad is a unit vector and all volumes are equal."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gas, mf0, h = _ot_fields(case, seed)
    U = [torch.from_numpy(np.ascontiguousarray(gas[..., v])).to(dev) for v in range(5)]
    mf = [torch.from_numpy(np.ascontiguousarray(mf0[..., d])).to(dev) for d in range(3)]
    area = [h[1] * h[2], h[0] * h[2], h[0] * h[1]]
    vol, rmeth, pdmb = h[0] * h[1] * h[2], case["rmeth"], 0.75
    oU, omf, b = [u.clone() for u in U], [m.clone() for m in mf], _cell_b(mf, area)
    odt = dt = _dt(U, b, h)
    for _ in range(case["steps"]):
        hmf = [m + 0.5 * dt * (m - o) / odt for m, o in zip(mf, omf)]
        hb = _cell_b(hmf, area)
        W, oW = _prim(U), _prim(oU)
        hW = [w + 0.5 * dt * (w - o) / odt for w, o in zip(W, oW)]
        hW[0], hW[4] = hW[0].clamp(min=TINY), hW[4].clamp(min=TINY)
        E = []
        for e in range(3):
            d1, d2 = (e + 1) % 3, (e + 2) % 3
            v1, v2 = (_recon8(_recon8(hW[1 + d], d1), d2) for d in (d1, d2))
            D = 0.25 * (hW[0] + _at(hW[0], d1, -1) + _at(hW[0], d2, -1) + _at(_at(hW[0], d1, -1), d2, -1))
            l1, r1 = _left_right(hmf[d1] / area[d1], mf[d1] / area[d1], d2, rmeth, pdmb)
            l2, r2 = _left_right(hmf[d2] / area[d2], mf[d2] / area[d2], d1, rmeth, pdmb)
            b1, b2 = 0.5 * (l1 + r1), 0.5 * (l2 + r2)
            vd = torch.sqrt(v1 ** 2 + v2 ** 2) + torch.sqrt(b1 ** 2 + b2 ** 2) / torch.sqrt(D)
            vd = vd.clamp(max=0.3 * h[e] / dt)
            E.append((-(v1 * b2 - v2 * b1) + 0.5 * vd * ((r2 - l2) - (r1 - l1))) * h[e])
        dg, dm = [torch.zeros_like(U[0]) for _ in range(5)], [torch.zeros_like(U[0]) for _ in range(3)]
        for d in range(3):
            LR = [_left_right(hW[v], W[v], d, rmeth, pdmb) for v in range(5)]
            BLR = [_left_right(hb[x], b[x], d, rmeth, pdmb) for x in range(3)]
            Bn = hmf[d] / area[d]
            G, M, va = [0.0] * 5, [0.0] * 3, 0.0
            jump = [0.0] * 5
            for s, sg in ((0, -1.0), (1, 1.0)):
                w, B = [q[s] for q in LR], [q[s] for q in BLR]
                vn, pb = w[1 + d], 0.5 * (B[0] ** 2 + B[1] ** 2 + B[2] ** 2)
                va2 = 2.0 * pb / w[0]
                m0 = 0.5 * torch.special.erfc(sg * vn / torch.sqrt(2.0 * w[4] / w[0] + va2))
                va = va + 0.5 * torch.sqrt(va2)
                for x in range(3):
                    M[x] = M[x] + m0 * ((pb if x == d else 0.0) - B[x] * Bn)
                e = 0.5 * w[0] * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) + w[4] / (GAMMA - 1.0)
                lam = w[0] / (2.0 * w[4])
                g0 = 0.5 * torch.special.erfc(sg * torch.sqrt(lam) * vn)
                g1 = vn * g0 - 0.5 * sg * torch.exp(-lam * vn ** 2) / torch.sqrt(math.pi * lam)
                G[0] = G[0] + w[0] * g1
                for x in range(3):
                    G[1 + x] = G[1 + x] + (w[0] * vn * g1 + w[4] * g0 if x == d else w[0] * w[1 + x] * g1)
                G[4] = G[4] + (e + 0.5 * w[4]) * g1 + 0.5 * w[4] * g0 * vn
                for v, q in enumerate((w[0], w[0] * w[1], w[0] * w[2], w[0] * w[3], e)):
                    jump[v] = jump[v] + sg * q
            for v in range(5):
                F = (G[v] - 0.25 * va * jump[v]) * area[d]
                dg[v] += (F - _at(F, d, 1)) / vol
            for x in range(3):
                F = M[x] * area[d]
                dm[x] += (F - _at(F, d, 1)) / vol
        oU, omf = U, mf
        N = [u + dt * g for u, g in zip(U, dg)]
        D = N[0].clamp(min=TINY)
        P = ((GAMMA - 1.0) * (N[4] - 0.5 * (N[1] ** 2 + N[2] ** 2 + N[3] ** 2) / D)).clamp(min=TINY)
        m = [N[1 + x] + dt * dm[x] for x in range(3)]
        U = [D, m[0], m[1], m[2], 0.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / D + P / (GAMMA - 1.0)]
        mf = [m - dt * c for m, c in zip(mf, _curl(E))]
        b = _cell_b(mf, area)
        odt, dt = dt, _next_dt(U, oU, omf, E, dt, area, h)
    host = lambda q: np.stack([a.cpu().numpy() for a in q], axis=-1)  # noqa: E731
    g, m = _ghosts(host(U), host(mf))
    start = _ghosts(gas, mf0)[1]
    # the last layer across another axis belongs to no cell and keeps what it was set to; so does, in 2.5D, the last
    # K layer, and with it the field of the last ghost cell
    for c in range(3):
        for d in range(3):
            if d != c or (d == 2 and case["nk"] == 1):
                last = [slice(None)] * 3
                last[d] = -1
                m[tuple(last) + (c,)] = start[tuple(last) + (c,)]
    bxyz = [0.5 * (m[:-1, :-1, :-1, 0] + m[1:, :-1, :-1, 0]) / area[0],
            0.5 * (m[:-1, :-1, :-1, 1] + m[:-1, 1:, :-1, 1]) / area[1],
            0.5 * (m[:-1, :-1, :-1, 2] + m[:-1, :-1, 1:, 2]) / area[2]]
    return {"gas": g, "magflux": m, "bxyz": np.stack(bxyz, axis=-1)}


def exact(case, seed):
    """The uniform periodic problems in 64 bits. The curvilinear ones (metrics by 12-point quadrature on every face
    and edge, ring averaging, hooks), the ensembles and the closure's samples (fine runs) take minutes in plain
    array code: none."""
    return _exact_ot(case, seed) if case["kind"] == "ot" else None
