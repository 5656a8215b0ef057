"""The coupled path's Jacobian and inverse kernels (csrc/jg_coupled.cu: 64 and 32 cells a block) at the
edges of their blocks, against the oracle."""
import dataclasses

import numpy as np
import pytest

from myjoe_b200 import case, solver

pytestmark = pytest.mark.gpu


def _nrel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


@pytest.mark.parametrize("model", ["sa", "sst"])
@pytest.mark.parametrize("dims", [(8, 4, 1), (11, 3, 1), (9, 7, 1), (8, 8, 1), (13, 5, 1)])
def test_steps_match_oracle_at_block_edges(model, dims):
    from oracle.oracle import OracleSA
    make = case.sa_bump_case if model == "sa" else case.sst_bump_case
    _, g, prm = make(*dims, stretch=1.15, mach=0.5, re=1.0e5)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="SGS", LS_MAX_ITER=4, CFL=2.0)
    st = case.perturbed_state(g.x_cv, prm, 0.02)
    phi = (np.full((g.ncv, 1), prm.NUSA_INITIAL) if model == "sa"
           else np.tile([prm.KINE_INITIAL, prm.OMEGA_INITIAL], (g.ncv, 1)))
    o = OracleSA(g, prm)
    o.set_state(*st)
    o.set_scalar(phi)
    o.calc_state()
    want = o.step(2)
    j = solver.JoeGpu(g, prm)
    j.set_state(*st)
    j.set_scalars(phi)
    # two steps of the same FP64 arithmetic in another order: the bound of the fixtures' step tests
    assert _nrel(j.runBackwardEuler(2)[-1], want) <= 1e-10
    for a, b in zip(j.get_state(), o.get_state()):
        assert _nrel(a, b) <= 1e-10
    a, b = (np.asarray(x).reshape(g.ncv, -1) for x in (j.get_scalars(), o.get_scalar()))
    for s in range(prm.nscal):
        assert _nrel(a[:, s], b[:, s]) <= 1e-10
