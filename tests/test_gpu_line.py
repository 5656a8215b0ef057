"""LINE relaxation (JG_LS_LINE) on the GPU against the oracle's jo_line_relax.

Block line-Jacobi: the block-tridiagonal system of every line of the
reference's initializeLinelet solved exactly, block Jacobi on the other
cells.  Checked on the 5x5 path (one solve on the reference's own system,
backward-Euler steps) and on the coupled SA/SST paths (steps), FP64 against
the oracle at 1e-12 (one solve) / 1e-10 (steps) relative, and converged
fields of the FP64 and mixed forms at 1e-8 relative L2.
"""
import dataclasses
import glob
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(__file__)


def nrel(a, b):
    a, b = np.asarray(a, float).ravel(), np.asarray(b, float).ravel()
    return float(np.abs(a - b).max() / np.abs(b).max())


def rel_l2(a, b):
    a, b = np.asarray(a, float).ravel(), np.asarray(b, float).ravel()
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _fixture(name):
    from tests.golden.make_golden import load
    return load(os.path.join(HERE, "golden", name + ".npz"))


@pytest.mark.parametrize("name", ["plate_roe_linelet", "mixed_bump_roe_laminar_linelet"])
def test_line_solve_matches_oracle(name):
    from myjoe_b200 import build, solver
    from oracle.oracle import Oracle
    build.build()
    g = _fixture(name)
    prm = dataclasses.replace(g["params"], LINEAR_SOLVER_NS="LINE")
    A = g["A"].copy()
    vol_dt = g["cv_volume"] / g["local_dt"]
    for i in range(5):
        A[g["nbocv_i"][:-1], i, i] += vol_dt
    rhs = g["rhs_sys"].reshape(-1, 5)
    o = Oracle(dict(g), prm)
    for sweeps in (1, 7):
        dq_o, _ = o.solve(A, rhs, 0, 0, sweeps, 5)
        j = solver.JoeGpu(dict(g), prm)
        dq_g, it = j.solveCoupledLinSysNS(A, rhs, 0, 0, sweeps)
        assert it == sweeps
        assert nrel(dq_g, dq_o) <= 1e-12


def test_line_steps_match_oracle_5x5():
    from myjoe_b200 import build, solver
    from oracle.oracle import Oracle
    build.build()
    g = _fixture("plate_roe_linelet")
    prm = dataclasses.replace(g["params"], LINEAR_SOLVER_NS="LINE", LS_MAX_ITER=6, CFL=5.0)
    o = Oracle(dict(g), prm)
    o.set_state(g["init_rho"], g["init_rhou"].reshape(-1, 3), g["init_rhoE"])
    o.calc_state()
    j = solver.JoeGpu(dict(g), prm)
    j.set_state(g["init_rho"], g["init_rhou"].reshape(-1, 3), g["init_rhoE"])
    ro = np.array([o.step(1) for _ in range(10)])
    rg = j.runBackwardEuler(10)
    assert nrel(rg, ro) <= 1e-10
    for a, b in zip(j.get_state(), o.get_state()):
        assert nrel(a, b) <= 1e-10


@pytest.mark.parametrize("name", ["sa_bump_farfield", "sst_mixed_bump_farfield"])
def test_line_steps_match_oracle_coupled(name):
    from myjoe_b200 import build, solver
    from oracle.oracle import OracleSA
    build.build()
    g = _fixture(name)
    prm = dataclasses.replace(g["params"], LINEAR_SOLVER_NS="LINE", LS_MAX_ITER=6, CFL=5.0)
    phi = np.stack([g["init_scal%d" % s] for s in range(prm.nscal)], 1)
    o = OracleSA(dict(g), prm)
    o.set_state(g["init_rho"], g["init_rhou"].reshape(-1, 3), g["init_rhoE"])
    o.set_scalar(phi)
    o.calc_state()
    j = solver.JoeGpu(dict(g), prm)
    j.set_state(g["init_rho"], g["init_rhou"].reshape(-1, 3), g["init_rhoE"])
    j.set_scalars(phi)
    ro = o.step(4)
    rg = j.runBackwardEuler(4)
    assert nrel(rg[-1], ro) <= 1e-10
    for a, b in zip(j.get_state(), o.get_state()):
        assert nrel(a, b) <= 1e-10
    assert nrel(j.get_scalars(), o.get_scalar()) <= 1e-10


@pytest.mark.parametrize("precision", [0, 1])
def test_line_converged_sa_field_matches_oracle(precision):
    from myjoe_b200 import build, case, solver
    from oracle.oracle import OracleSA
    build.build()
    raw, g, prm = case.sa_bump_case(24, 16, 2, stretch=1.25, seed=1, mach=0.5, re=1.0e5, n_prism=4,
                                    alternate=True, shuffle=True)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="LINE", LS_MAX_ITER=6, CFL=1.0, CFL_RAMP=(10, 5, 1.2, 50.0))
    st = case.perturbed_state(g.x_cv, prm, 0.0)
    phi0 = np.full(g.ncv, prm.NUSA_INITIAL)
    o = OracleSA(g, prm)
    o.set_state(*st)
    o.set_scalar(phi0)
    o.calc_state()
    ro = o.step(1500)
    j = solver.JoeGpu(g, prm, precision=precision, renumber=True)
    j.set_state(*st)
    j.set_scalars(phi0)
    rg = j.runBackwardEuler(1500)
    assert rg[-1, 4] / rg[0, 4] < 1e-9 and ro[4] / rg[0, 4] < 1e-9
    for a, b in zip(j.get_state(), o.get_state()):
        assert rel_l2(a, b) <= 1e-8
    assert rel_l2(j.get_scalars(), o.get_scalar()) <= 1e-8


@pytest.mark.parametrize("renumber", [0, 3])
@pytest.mark.parametrize("precision", [0, 1])
def test_line_solve_where_a_cell_has_two_wall_faces(precision, renumber):
    """the cell is on one line: one sweep is the oracle's, and the sweeps converge to the system's solution"""
    import scipy.sparse
    import scipy.sparse.linalg
    from myjoe_b200 import build, solver
    from oracle.oracle import Oracle
    from tests.test_lines import two_wall_face_case
    build.build()
    g, prm = two_wall_face_case(shuffle=True)
    rng = np.random.default_rng(4)
    A = rng.standard_normal((g.nbocv_v.shape[0], 5, 5))
    A[g.nbocv_i[:-1]] += 40.0 * np.eye(5)
    b = rng.standard_normal((g.ncv, 5))
    j = solver.JoeGpu(g, prm, precision=precision, renumber=renumber)
    o = Oracle(g, prm)
    eps = np.finfo(np.float32).eps if precision else np.finfo(np.float64).eps
    # rows of at most 7 blocks of 5 and a diagonal of about 40: a solve loses a few tens of roundings, and
    # a sweep contracts the ones before it
    for sweeps in (1, 4):
        assert nrel(j.solveCoupledLinSysNS(A, b, 0, 0, sweeps)[0], o.solve(A, b, 0, 0, sweeps, 5)[0]) <= 200 * eps
    M = scipy.sparse.bsr_matrix((A, g.nbocv_v, g.nbocv_i), shape=(5 * g.ncv, 5 * g.ncv)).tocsc()
    want = scipy.sparse.linalg.spsolve(M, b.ravel())
    assert nrel(j.solveCoupledLinSysNS(A, b, 0, 0, 60)[0], want) <= 200 * eps


# a stage of the substitutions' ring holds 4 positions of a line in FP64, 8 in FP32: 1 to 3 stages and a
# step less and more; two lines of each length, so that a warp's four have several, and the last warp two
RING_LENGTHS = (2, 3, 4, 5, 6, 8, 9, 10, 13, 14, 17, 18, 25, 26, 27)


def _towers(shuffle=True):
    """Separate blocks of 2 x L x 1 flat hexahedra on a wall: two lines of L cells each."""
    from myjoe_b200 import geometry, meshgen
    names = {"imin": "inlet", "imax": "outlet", "jmin": "lower", "jmax": "upper", "kmin": "sides", "kmax": "sides"}
    parts, x_no, zones = [], [], {}
    nno = nfa = ncv = 0
    for i, n in enumerate(RING_LENGTHS):
        X, Y = np.meshgrid(0.1 * (np.arange(3.0) + 4 * i), 0.01 * np.arange(n + 1.0), indexing="ij")
        b = meshgen.structured_hex(X, Y, np.array([0.0, 0.1]), lambda side, *ijk: np.full(len(ijk[0]), names[side]))
        parts.append((b.fa_nodes + nno, b.fa_nno, np.where(b.cvofa >= 0, b.cvofa + ncv, -1)))
        x_no.append(b.x_no)
        for name, f in b.zones:
            zones.setdefault(str(name), []).append(f + nfa)
        nno, nfa, ncv = nno + len(b.x_no), nfa + b.nfa, ncv + b.ncv
    raw = meshgen.RawMesh(x_no=np.concatenate(x_no), ncv=ncv, zones=[(k, np.concatenate(v)) for k, v in zones.items()],
                          **{k: np.concatenate([p[j] for p in parts])
                             for j, k in enumerate(("fa_nodes", "fa_nno", "cvofa"))})
    return geometry.build_cv_mesh(raw, seed=6, shuffle=shuffle)


@pytest.mark.parametrize("precision", [0, 1])
def test_line_lengths_around_the_ring_5x5(precision):
    from myjoe_b200 import build, case, solver
    from oracle.oracle import Oracle
    build.build()
    g = _towers()
    prm = dataclasses.replace(case.sa_bump_case(6, 4, 1)[2], TURB_MODEL="NONE", scalar_bcs={}, LINEAR_SOLVER_NS="LINE")
    o = Oracle(g, prm)
    assert sorted(np.diff(o.relax_lines()[0])) == sorted(2 * RING_LENGTHS)
    rng = np.random.default_rng(9)
    A = rng.standard_normal((g.nbocv_v.shape[0], 5, 5))
    A[g.nbocv_i[:-1]] += 40.0 * np.eye(5)
    b = rng.standard_normal((g.ncv, 5))
    j = solver.JoeGpu(g, prm, precision=precision)
    eps = np.finfo(np.float32).eps if precision else np.finfo(np.float64).eps
    for sweeps in (1, 3):
        # a row sums at most 4 blocks of 5 and the chain along a line contracts: tens of roundings
        assert nrel(j.solveCoupledLinSysNS(A, b, 0, 0, sweeps)[0], o.solve(A, b, 0, 0, sweeps, 5)[0]) <= 200 * eps


@pytest.mark.parametrize("model", ["SA", "SST"])
def test_line_lengths_around_the_ring_coupled(model):
    from myjoe_b200 import build, case, solver
    from oracle.oracle import OracleSA
    build.build()
    g = _towers()
    sa = model == "SA"
    prm = (case.sa_bump_case if sa else case.sst_bump_case)(6, 4, 1)[2]
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="LINE", LS_MAX_ITER=3, CFL=1.0)
    st = case.perturbed_state(g.x_cv, prm, 0.01)
    phi = np.full(g.ncv, prm.NUSA_INITIAL) if sa else np.tile([prm.KINE_INITIAL, prm.OMEGA_INITIAL], (g.ncv, 1))
    o = OracleSA(g, prm)
    o.set_state(*st)
    o.set_scalar(phi)
    o.calc_state()
    o.step(1)
    out = []
    for precision in (0, 1):
        j = solver.JoeGpu(g, prm, precision=precision)
        j.set_state(*st)
        j.set_scalars(phi)
        j.runBackwardEuler(1)
        out.append([*j.get_state(), j.get_scalars()])
        j.close()
    for a, m, b, s in zip(out[0], out[1], [*o.get_state(), o.get_scalar()], [*st, phi]):
        a, m, b, s = (np.asarray(x, float).reshape(g.ncv, -1) for x in (a, m, b, s))
        groups = [slice(0, 3)] if a.shape[1] == 3 else [slice(k, k + 1) for k in range(a.shape[1])]
        for k in groups:   # the momentum as one vector, each scalar by itself
            assert nrel(a[:, k], b[:, k]) <= 1e-10
            # FP32 blocks: the update to single precision, of which the conditioning of the blocks takes at
            # most a factor 1e3
            assert np.abs(m[:, k] - a[:, k]).max() <= 1e-4 * np.abs(a[:, k] - s[:, k]).max()
