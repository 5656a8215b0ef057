"""Device memory a case needs (jg_case_footprint, the serving engine's admission rule): host only."""
import dataclasses

import pytest

from myjoe_b200 import case, solver


@pytest.mark.parametrize("precision,limit", [(0, 3100), (1, 2320)])
def test_centres_are_held_once(precision, limit):
    """8,192 hexahedra: 288 bytes a cell of state, ~370 of gradients and face fluxes, 25 blocks of 25,
    and cell and face centres in their records only (24 bytes a cell and a face each)"""
    _, g, prm = case.bump_case(64, 32, 4)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="SGS")
    assert solver.case_footprint(g, prm, precision) / g.ncv <= limit


@pytest.mark.parametrize("flux", ["AUSMDV", "HAENEL"])
@pytest.mark.parametrize("model,b", [("SA", 6), ("SST", 7)])
def test_only_hllc_keeps_the_fp64_diagonal_of_a_mixed_handle(model, b, flux):
    """its blocks are inverted by a kernel of their own; the AUSM family inverts where it forms them"""
    _, g, prm = (case.sa_bump_case if model == "SA" else case.sst_bump_case)(32, 16, 2)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="SGS", SHOCK_FIX_TYPE="NONE")
    hllc, other = (solver.case_footprint(g, dataclasses.replace(prm, SPACE_INTEGRATION=f), 1) for f in ("HLLC", flux))
    assert hllc - other == 8 * b * b * g.ncv


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (3, 2, 1), (16, 8, 2)])
@pytest.mark.parametrize("model", ["NONE", "SA"])
def test_a_handle_holds_its_footprint(model, dims):
    """from the meshes whose matrix is smaller than their centres on, and the records are right: a step gives
    the oracle's residual"""
    import numpy as np
    from oracle.oracle import Oracle
    sa = model == "SA"
    _, g, prm = (case.sa_bump_case if sa else case.bump_case)(*dims)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="JACOBI")
    st = case.perturbed_state(g.x_cv, prm, 0.02)
    j = solver.JoeGpu(g, prm, precision=1)
    j.set_state(*st)
    assert j.device_bytes() == solver.case_footprint(g, prm, 1)
    if not sa:
        o = Oracle(g, prm)
        o.set_state(*st)
        o.calc_state()
        o.calc_dt()
        rho, rhou, rhoE, _ = o.calc_rhs(False)
        got = j.calcRhs(False)[:3]
        # sums of at most six face fluxes of the order of p u, rho u, rho E u
        for a, b, s in zip(got, (rho, rhou, rhoE), o.array("flux_scale").max(0)[[0, 1, 4]]):
            assert np.abs(a - np.reshape(b, a.shape)).max() <= 1e-11 * max(s, 1e-300)
