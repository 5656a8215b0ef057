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
