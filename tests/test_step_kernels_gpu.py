"""The step's kernels at the sizes where their launch rules change (side branches, CalcDT's end, rings and axis rows that
meet) and where a tile, a run of faces or a ghost layer ends early. Against the oracle the bound is the parity tests' 1e-10; variants that differ only in the launch give the same
bits. The periodic sides' index map is checked on the CPU too, against the three sweeps it stands for."""
import numpy as np
import pytest

from helpers import mirror_to_gpu, oracle_and_gpu, per_var_rel, resync

TOL = 1e-10
STATE = ("gas", "magflux", "bxyz")


def _axis(n, normal, flat, ng=4):
    """Where each element of an axis of n active cells is taken from: the map of k_bc_periodic"""
    s, e = ng, ng + n - 1
    src = np.arange(n + 2 * ng + 1)
    for x in range(len(src)):
        up = 1 if normal and not flat else 0
        if x < s:
            src[x] = s if flat else e - (s - x - 1) % n
        elif flat:
            src[x] = s if x <= s + ng else x
        elif 1 <= x - up - e <= ng:
            src[x] = s + up + (x - up - e - 1) % n
    return src


def _sweeps(a, n, comp, d25, ng=4):
    """EnforceBCs of six periodic sides layer by layer (comp: 0-2 the faces across that axis, 3 the cells)"""
    a = a.copy()
    for d in range(3):
        v, s, e = np.moveaxis(a, d, 0), ng, ng + n[d] - 1
        flat, up = d == 2 and d25, 1 if comp == d else 0
        for m in range(ng):
            v[s - 1 - m] = v[s if flat else e - m % n[d]]
            if flat:
                v[s + 1 + m] = v[s]
            else:
                v[e + 1 + m + up] = v[s + m % n[d] + up]
    return a


@pytest.mark.parametrize("n,d25", [((8, 5, 6), False), ((8, 2, 3), False), ((16, 7, 1), True), ((8, 1, 1), True)])
def test_periodic_map_equals_sweeps(n, d25):
    for comp in range(4):
        a = np.random.default_rng(comp).normal(size=tuple(q + 9 for q in n))
        m = [_axis(n[d], comp == d, d == 2 and d25) for d in range(3)]
        want, got = _sweeps(a, n, comp, d25), a[np.ix_(*m)]
        if comp == 3:   # the cells end one element before the faces
            want, got = want[:-1, :-1, :-1], got[:-1, :-1, :-1]
        assert np.array_equal(want, got)
        assert all(np.array_equal(q[q], q) for q in m)   # nothing that is read is written


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "fp32flux"])
@pytest.mark.parametrize("n,kw", [((16, 5, 6), {}), ((16, 4, 4), dict(rmeth="7UP")), ((40, 9, 1), {}), ((32, 13, 1), dict(doMHD=False))])
def test_periodic_sides(gpu_lib, oracle_lib, n, kw, prec):
    """Steps with six periodic sides against the oracle, ghosts and the faces beyond them included, and the ghosts against
    the sweeps exactly."""
    from kaiju_b200 import gamera as gm
    o, g = oracle_and_gpu("ot", n, **kw)
    with g:
        if prec == "fp32flux":
            g.set_precision(gm.GAM_FP32FLUX)
        for _ in range(2):
            o.step()
            g.step()
            for name in STATE if prec == "fp64" else ():
                assert max(per_var_rel(g.fetch(name), o.get(name))) <= TOL, name
            for name in ("gas", "magflux"):
                a = g.fetch(name)
                for v in range(a.shape[3]):
                    ng1 = np.pad(a[..., v], ((0, 1),) * 3) if name == "gas" else a[..., v]
                    want = _sweeps(ng1, n, v if name == "magflux" else 3, n[2] == 1)
                    cut = slice(None, -1) if name == "gas" else slice(None)
                    assert np.array_equal(want[cut, cut, cut], a[..., v]), (name, v)
            resync(o, g)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(24, 11, 13), (16, 17, 9), (40, 8, 8)])
def test_odd_sizes(gpu_lib, oracle_lib, n):
    """Rows, runs of faces and tiles that end early, on the curvilinear grid."""
    o, g = oracle_and_gpu("bw", n)
    with g:
        for _ in range(2):
            o.step()
            g.step()
            for name in STATE + ("efld",):
                assert max(per_var_rel(g.fetch(name), o.get(name))) <= TOL, name
            resync(o, g)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n", [("ot", (32, 24, 4)), ("bw", (24, 16, 16)), ("ot", (40, 24, 1))])
def test_side_by_side_equals_one_stream(gpu_lib, oracle_lib, kind, n):
    """A small problem's step, captured with side branches, and the phase-timed step, one kernel after the other: the same
    bits. (Whether the branches run at the same time shows in the step's time only.)"""
    o, a = oracle_and_gpu(kind, n)
    b = mirror_to_gpu(o, a.model)
    with a, b:
        b.profile_phases(4)
        a.run_steps(b.status()["ts"])
        for name in STATE:
            assert np.array_equal(a.fetch(name), b.fetch(name)), name


@pytest.mark.gpu
def test_half_state_belongs_to_the_last_step(gpu_lib, oracle_lib):
    """The half state of the last step stays what it is while the precision is changed: a change writes no half state, and
    the planes of one mode do not stand for the other's step. (With FP32 fluxes the half state's gas is kept as floats for
    the fluxes only, so that mode's is not fetched.)"""
    from kaiju_b200 import gamera as gm
    o, g = oracle_and_gpu("bw", (16, 16, 16))
    with g:
        o.step()
        g.step()
        for mode in (gm.GAM_FP32FLUX, gm.GAM_FP64):   # a step in double precision, first fetched after the change
            g.set_precision(mode)
            for name in ("hgas", "hmagflux"):
                assert max(per_var_rel(g.fetch(name), o.get(name))) <= TOL, (mode, name)
        g.set_precision(gm.GAM_FP32FLUX)
        resync(o, g)
        o.step()
        g.step()   # a step with FP32 fluxes, whose face fluxes of the half state are still double
        for mode in (gm.GAM_FP32FLUX, gm.GAM_FP64):
            g.set_precision(mode)
            assert max(per_var_rel(g.fetch("hmagflux"), o.get("hmagflux"))) <= TOL, mode


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp64", "fp32flux"])
def test_given_cell_field(gpu_lib, oracle_lib, prec):
    """A Bxyz that is not bFlux2Fld of its fluxes (as a host may send) enters the limiter and the first step's old field
    only: the half state's field comes from the fluxes, as the oracle forms it."""
    from kaiju_b200 import gamera as gm
    o, g = oracle_and_gpu("bw", (16, 16, 16))
    b = o.get("bxyz")
    for name in ("bxyz", "obxyz"):
        o.set(name, o.get(name) * (1.0 + 0.01 * np.random.default_rng(3).uniform(size=b.shape)))
    with g:
        resync(o, g)
        if prec == "fp32flux":
            g.set_precision(gm.GAM_FP32FLUX)
        for _ in range(3):
            o.step()
            g.step()
        tol = 1e-9 if prec == "fp64" else 2e-5   # three free-running steps; single-precision fluxes
        for name in STATE:
            assert max(per_var_rel(g.fetch(name), o.get(name))) <= tol, name


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["bxyz", "obxyz"])
@pytest.mark.parametrize("cell", [(4, 4, 4), (27, 11, 19), (9, 8, 12)])
def test_given_field_of_one_cell(gpu_lib, oracle_lib, name, cell):
    """One cell of one of the two states is enough for the half state's field to come from the fluxes."""
    o, g = oracle_and_gpu("bw", (24, 8, 16))
    o.step()
    b = o.get(name)
    b[cell] = (0.3, -0.2, 0.4)
    o.set(name, b)
    with g:
        resync(o, g)
        for _ in range(2):
            o.step()
            g.step()
            for q in STATE:
                assert max(per_var_rel(g.fetch(q), o.get(q))) <= TOL, q


def _ot_device(n, **kw):
    from kaiju_b200 import gamera as gm
    m = gm.Model(*n, CFL=0.3, bc=(gm.GAM_BC_PERIODIC,) * 6, tFin=1.0e30, **kw)
    return gm.GameraGPU.from_corners(m, gm.corners_uniform(m, (0.0, 1.0, 0.0, 1.0, 0.0, n[2] / n[0])), "OT2D")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(48, 40, 31), (48, 40, 32), (312, 320, 1), (320, 320, 1)])
def test_either_side_of_the_branch_rule(gpu_lib, n):
    """60,000 cells, 100,000 in 2.5D: captured steps and the same kernels one after the other give the same bits."""
    with _ot_device(n) as a, _ot_device(n) as b:
        a.run_steps(3)
        b.profile_phases(3)
        for name in STATE:
            assert np.array_equal(a.fetch(name), b.fetch(name)), name


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(720, 720, 1), (728, 728, 1)])
def test_either_side_of_the_dt_rule(gpu_lib, n):
    """2,048 blocks: CalcDT over the active cells, its minimum taken in its own launch and in one more, against the dt of
    the state that the step leaves."""
    with _ot_device(n, dtActive=True) as g:
        for _ in range(2):
            dt, _, _ = g.step()
            act = (slice(4, -4),) * 3
            q, b = g.fetch("gas")[act], g.fetch("bxyz")[act]
            dl = np.minimum(np.minimum(g.fetch("di"), g.fetch("dj")), g.fetch("dk"))[act]
            v2 = (q[..., 1:4] ** 2).sum(-1) / q[..., 0] ** 2
            P = (g.model.gamma - 1.0) * (q[..., 4] - 0.5 * q[..., 0] * v2)
            fast = np.sqrt(g.model.gamma * P / q[..., 0] + (b ** 2).sum(-1) / q[..., 0])
            want = 0.3 * (dl / (np.sqrt(v2) + fast)).min()
            assert abs(dt - want) <= 1e-13 * want


@pytest.mark.gpu
@pytest.mark.parametrize("n,ring", [((16, 8, 32), dict(NumR=4, Nch=[8, 16, 32, 32])), ((16, 9, 32), dict(NumR=4, Nch=[8, 16, 32, 32])),
                                    ((16, 4, 32), dict(NumR=1, Nch=[16]))])
def test_rings_and_axis_rows_that_meet(gpu_lib, oracle_lib, n, ring):
    """Both poles' rings in one launch only where they do not meet; and as few rows between the axes as the ghosts take.
    (With fewer, the oracle's metrics and half state of the axis ghosts are not finite either.)"""
    o, g = oracle_and_gpu("lfmbw", n, ring=ring)
    with g:
        for _ in range(2):
            o.step()
            g.step()
            for name in STATE:
                assert max(per_var_rel(g.fetch(name), o.get(name))) <= TOL, name
            resync(o, g)


@pytest.mark.gpu
def test_single_precision_e_field_error(gpu_lib):
    """One step with FP32 fluxes and one without from the same state of the blast wave on the curvilinear grid: the E
    field's relative root mean square difference. 2.610e-7 with Mom2Face's products volume * velocity formed in double and
    rounded once (and in every build before they were dropped), 2.659e-7 with products of floats; the bound lies between."""
    from kaiju_b200 import gamera as gm
    m = gm.Model(64, 48, 40, CFL=0.3, bc=(gm.GAM_BC_ZEROGRAD,) * 6, tFin=1.0e30)
    x = gm.corners_warped(m, (-0.5, 0.5) * 3, 0.04)
    with gm.GameraGPU.from_corners(m, x, "BW") as g:
        g.run_steps(25)
        st, s, e = {q: g.fetch(q) for q in STATE + ("ogas", "omagflux", "obxyz")}, g.status(), []
        for prec in (gm.GAM_FP64, gm.GAM_FP32FLUX):
            with gm.GameraGPU.from_corners(m, x, "BW") as h:
                h.set_precision(prec)
                h.sync_to_device(time=s["time"], otime=s["otime"], **st)
                h.set_scalars(s["t"], s["dt"], s["dt0"], s["ts"], s["time"], s["otime"])
                h.step()
                e.append(h.fetch("efld")[4:-4, 4:-4, 4:-4])
    assert np.linalg.norm(e[1] - e[0]) <= 2.635e-7 * np.linalg.norm(e[0])
