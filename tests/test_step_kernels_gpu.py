"""The step's kernels at the sizes where their launch rules change and where a tile, a run of faces or a ghost layer ends
early. Against the oracle the bound is the parity tests' 1e-10; variants that differ only in the launch give the same
bits."""
import numpy as np
import pytest

from helpers import mirror_to_gpu, oracle_and_gpu, per_var_rel, resync

TOL = 1e-10
STATE = ("gas", "magflux", "bxyz")


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
    """A small problem's step on its side streams and the phase-timed step on one stream: the same bits."""
    o, a = oracle_and_gpu(kind, n)
    b = mirror_to_gpu(o, a.model)
    with a, b:
        b.profile_phases(4)
        a.run_steps(b.status()["ts"])
        for name in STATE:
            assert np.array_equal(a.fetch(name), b.fetch(name)), name


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
