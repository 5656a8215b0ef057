"""The block relaxation passes (csrc/jg_sweep.cuh) at the sizes where their launch changes: the last
slice of a mesh, rows wider than one chunk of columns, and the grids around one wave of resident
blocks, where the pass takes the whole row, three columns or one column at a time."""
import dataclasses

import numpy as np
import pytest

from myjoe_b200 import case, geometry, meshgen, solver

pytestmark = pytest.mark.gpu


def _mesh(nx, ny, nz, n_prism=0):
    prm = case.bump_case(4, 2, 2)[2]
    if not n_prism:
        return case.bump_case(nx, ny, nz)[1], prm
    raw = meshgen.channel_bump_mixed(nx, ny, nz, n_prism=n_prism, alternate=True)
    return geometry.build_cv_mesh(raw, seed=3, shuffle=True), prm


def _system(g, rng):
    """A diagonally dominant random block system in the reference's CSR layout."""
    nnz = g.nbocv_v.shape[0]
    A = rng.standard_normal((nnz, 5, 5))
    A[g.nbocv_i[:-1]] += 60.0 * np.eye(5)
    return A, rng.standard_normal((g.ncv, 5))


def _colors(g):
    """First-fit colours in cell order, as the handle gives them."""
    col = np.zeros(g.ncv, int)
    for c in range(g.ncv):
        used = {col[n] for n in g.nbocv_v[g.nbocv_i[c] + 1:g.nbocv_i[c + 1]] if n < c}
        col[c] = next(k for k in range(256) if k not in used)
    return col


def _relax(g, A, b, sweeps, colors=None):
    row = np.repeat(np.arange(g.ncv), np.diff(g.nbocv_i))
    off = np.ones(len(row), bool)
    off[g.nbocv_i[:-1]] = False
    Di = np.linalg.inv(A[g.nbocv_i[:-1]])
    x = np.zeros_like(b)

    def new():
        r = b.copy()
        np.subtract.at(r, row[off], np.einsum("nij,nj->ni", A[off], x[g.nbocv_v[off]]))
        return np.einsum("nij,nj->ni", Di, r)
    for it in range(sweeps):
        if colors is None:
            x = new()
            continue
        order = range(colors.max() + 1)
        for q in (order if it % 2 == 0 else reversed(order)):   # every pass, repeated colours too
            x = np.where((colors == q)[:, None], new(), x)
    return x


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", ["JACOBI", "SGS"])
@pytest.mark.parametrize("dims,n_prism", [((3, 1, 1), 0), ((11, 3, 1), 0), ((9, 7, 3), 0), ((12, 8, 3), 3)])
def test_relaxation_matches_plain_numpy(dims, n_prism, name, precision):
    g, prm = _mesh(*dims, n_prism=n_prism)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS=name, LS_MAX_ITER=5)
    A, b = _system(g, np.random.default_rng(7))
    j = solver.JoeGpu(g, prm, precision=precision)
    for sweeps in (1, 2, 5):
        x, _ = j.solveCoupledLinSysNS(A, b, 0.0, 0.0, sweeps)
        want = _relax(g, A, b, sweeps, _colors(g) if name == "SGS" else None)
        # a pass sums at most 8 blocks x 5 products and 5 more for Dinv, whose condition is below 3
        # here: 50 eps a pass, damped from pass to pass (dominance), a factor 10 over that
        tol = 500.0 * (np.finfo(np.float32).eps if precision else np.finfo(np.float64).eps)
        assert np.abs(x - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("nx,ny", [(197, 96), (148, 128), (183, 104), (182, 208), (148, 256), (158, 240), (333, 168)])
def test_sweep_kernels_agree_bitwise_around_one_wave(nx, ny):
    """the slice kernel at every chunk width against the thread-per-cell kernel"""
    g, prm = _mesh(nx, ny, 1)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="JACOBI", LS_MAX_ITER=4)
    out = []
    for variant in (0, 1):
        j = solver.JoeGpu(g, prm)
        j.set_launch_config(36, variant)
        j.set_state(*case.perturbed_state(g.x_cv, prm, 0.02))
        r = j.runBackwardEuler(2)
        out.append([r, *j.get_state()])
        j.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


# FP32 rows: 160 threads of 80 registers, five blocks per SM, so 740 slices (23,680 cells) are one wave of the
# whole-row kernel; above it runs capped at 64 registers
@pytest.mark.parametrize("nx,ny", [(148, 128), (197, 120), (197, 124), (350, 230)])
def test_fp32_sweep_kernels_agree_bitwise_around_one_wave(nx, ny):
    g, prm = _mesh(nx, ny, 1)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="JACOBI", LS_MAX_ITER=4)
    A, b = _system(g, np.random.default_rng(2))
    out = []
    for variant in (0, 1):
        j = solver.JoeGpu(g, prm, precision=1)
        j.set_launch_config(36, variant)
        out.append(j.solveCoupledLinSysNS(A, b, 0.0, 0.0, 4)[0])
        j.close()
    np.testing.assert_array_equal(*out)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx,ny,renumber", [(197, 120, 0), (250, 200, 0)])
def test_sgs_matches_plain_numpy_around_one_wave(nx, ny, renumber, precision):
    g, prm = _mesh(nx, ny, 1)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="SGS", LS_MAX_ITER=3)
    A, b = _system(g, np.random.default_rng(7))
    j = solver.JoeGpu(g, prm, precision=precision, renumber=renumber)
    x, _ = j.solveCoupledLinSysNS(A, b, 0.0, 0.0, 3)
    want = _relax(g, A, b, 3, _colors(g))
    tol = 500.0 * (np.finfo(np.float32).eps if precision else np.finfo(np.float64).eps)   # as above
    assert np.abs(x - want).max() <= tol * np.abs(want).max()


# coupled blocks: one wave of the whole-row kernel is at most 592 slices of 6x6 FP64 (four blocks per SM),
# less of 7x7, more of FP32; 36k cells are 1,125 slices
@pytest.mark.parametrize("name", ["JACOBI", "SGS"])
@pytest.mark.parametrize("model", ["SA", "SST"])
def test_coupled_steps_match_the_oracle_above_one_wave(model, name):
    from oracle.oracle import OracleSA
    sa = model == "SA"
    _, g, prm = (case.sa_bump_case if sa else case.sst_bump_case)(180, 100, 2, stretch=1.03)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS=name, LS_MAX_ITER=4, CFL=1.0)
    st = case.perturbed_state(g.x_cv, prm, 0.0)
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
            assert np.abs(a[:, k] - b[:, k]).max() <= 1e-10 * np.abs(b[:, k]).max()   # as the steps of test_gpu_sa
            # FP32 blocks: the update to single precision, of which the conditioning of the blocks takes at
            # most a factor 1e3
            assert np.abs(m[:, k] - a[:, k]).max() <= 1e-4 * np.abs(a[:, k] - s[:, k]).max()
