"""jg_get_gradients: the device's padded gradient records reach the caller's packed arrays in a few
copies, whatever the number of cells."""
import dataclasses
import time

import numpy as np
import pytest

from myjoe_b200 import case, solver
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

NAMES = ("grad_u", "grad_rho", "grad_p", "grad_enthalpy")


@pytest.mark.parametrize("renumber", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (7, 3, 1), (33, 9, 2)])
def test_gradients_match_the_oracle_from_one_cell_on(dims, renumber):
    """the records go through a staging area that holds five doubles a cell, the nine of grad_u in lots"""
    _, g, prm = case.bump_case(*dims)
    prm = dataclasses.replace(prm, MU_REF=1.0e-3)
    st = case.perturbed_state(g.x_cv, prm, 0.05)
    o = Oracle(g, prm)
    o.set_state(*st)
    o.calc_state()
    o.calc_dt()
    o.calc_rhs(False)
    j = solver.JoeGpu(g, prm, renumber=renumber)
    j.set_state(*st)
    j.calcDt()
    j.calcRhs(False)
    got = j.gradients()
    scale = {"grad_u": np.abs(st[1] / st[0][:, None]).max(), "grad_rho": st[0].max(), "grad_p": 1.0e5,
             "grad_enthalpy": 4.0e5}
    lsq = max(np.abs(g.nbocv_lsg_coeff).max(), np.abs(g.boundary_fa_lsg_coeff).max())
    for k in NAMES:
        # a gradient is a sum of at most 7 weights times values: rounding of 1e-12 of the largest of them
        assert np.abs(got[k].ravel() - o.array(k).ravel()).max() <= 1e-12 * lsq * scale[k], k


def test_gradients_cost_a_few_state_reads():
    """18 doubles a cell against get_state's 5: 3.6 times its bytes in four more copies; a copy per
    record is above a hundred times its time"""
    _, g, prm = case.plate_case(256, 96, 2)
    j = solver.JoeGpu(g, prm)
    j.set_state(*case.perturbed_state(g.x_cv, prm, 0.02))
    j.calcGrad()

    def ms(f):
        t = []
        for _ in range(9):
            a = time.perf_counter()
            f()
            t.append(time.perf_counter() - a)
        return 1e3 * float(np.median(t))
    assert ms(j.gradients) <= 15.0 * ms(j.get_state)


# 148 SMs: up to 444 blocks of 128 cells are a wave of three resident blocks per SM, up to 592 of four
@pytest.mark.parametrize("dims", [(200, 142, 2), (200, 143, 2), (200, 189, 2), (200, 190, 2), (360, 200, 2)])
def test_gradients_match_the_oracle_where_the_kernel_changes(dims):
    """the least-squares kernel compiled for three or for four resident blocks per SM"""
    _, g, prm = case.bump_case(*dims)
    prm = dataclasses.replace(prm, MU_REF=1.0e-3)
    st = case.perturbed_state(g.x_cv, prm, 0.05)
    o = Oracle(g, prm)
    o.set_state(*st)
    o.calc_state()
    o.calc_dt()
    o.calc_rhs(False)
    j = solver.JoeGpu(g, prm)
    j.set_state(*st)
    got = j.calcGrad()
    scale = {"grad_u": np.abs(st[1] / st[0][:, None]).max(), "grad_rho": st[0].max(), "grad_p": 1.0e5,
             "grad_enthalpy": 4.0e5}
    lsq = max(np.abs(g.nbocv_lsg_coeff).max(), np.abs(g.boundary_fa_lsg_coeff).max())
    for k in NAMES:
        assert np.abs(got[k].ravel() - o.array(k).ravel()).max() <= 1e-12 * lsq * scale[k], k
