"""The device-driven BiCGSTAB (csrc/jg_bicgstab.cu): its iterates on small systems at the edges of its
slices and reductions, and its stopping rules."""
import dataclasses

import numpy as np
import pytest
import scipy.sparse

from myjoe_b200 import case, geometry, meshgen, solver

pytestmark = pytest.mark.gpu


def _system(dims, n_prism, rng):
    prm = dataclasses.replace(case.bump_case(4, 2, 2)[2], LINEAR_SOLVER_NS="BCGSTAB")
    if n_prism:
        raw = meshgen.channel_bump_mixed(*dims, n_prism=n_prism, alternate=True)
        g = geometry.build_cv_mesh(raw, seed=3, shuffle=True)
    else:
        g = case.bump_case(*dims)[1]
    A = rng.standard_normal((g.nbocv_v.shape[0], 5, 5))
    A[g.nbocv_i[:-1]] += 40.0 * np.eye(5)
    return g, prm, A, rng.standard_normal((g.ncv, 5))


def _bicgstab(g, A, b, iterations):
    """The reference's recurrence from zero, block-diagonal preconditioner."""
    M = scipy.sparse.bsr_matrix((A, g.nbocv_v, g.nbocv_i), shape=(5 * g.ncv, 5 * g.ncv)).tocsr()
    Di = np.linalg.inv(A[g.nbocv_i[:-1]])
    pre = lambda y: np.einsum("nij,nj->ni", Di, y.reshape(-1, 5)).ravel()  # noqa: E731
    b = b.ravel()
    x, r = np.zeros_like(b), b.copy()
    r0, p, v = r.copy(), np.zeros_like(b), np.zeros_like(b)
    rho = alpha = omega = 1.0
    for _ in range(iterations):
        old, rho = -omega * rho, r @ r0
        beta = alpha * rho / old
        p = r - beta * (p - omega * v)
        ph = pre(p)
        v = M @ ph
        alpha = rho / (v @ r0)
        s = r - alpha * v
        sh = pre(s)
        t = M @ sh
        omega = (s @ t) / (t @ t)
        x = x + alpha * ph + omega * sh
        r = b - M @ x
    return x.reshape(-1, 5)


@pytest.mark.parametrize("dims,n_prism", [((3, 1, 1), 0), ((16, 2, 1), 0), ((11, 3, 1), 0), ((12, 8, 3), 3),
                                          ((60, 29, 3), 0)])
def test_iterates_match_plain_numpy(dims, n_prism):
    g, prm, A, b = _system(dims, n_prism, np.random.default_rng(21))
    j = solver.JoeGpu(g, prm)
    for iterations in (1, 2, 3):
        x, it = j.solveCoupledLinSysNS(A, b, -1.0, -1.0, iterations - 1)
        assert it == iterations
        want = _bicgstab(g, A, b, iterations)
        # each iteration divides sums of ~1e4 products (1e-14 relative) that lose at most a factor
        # 1e2 to cancellation on these well-conditioned systems: 1e-12 an iteration, growing by less
        # than ten from one to the next
        assert np.abs(x - want).max() <= 1e-12 * 10 ** (iterations - 1) * np.abs(want).max()


@pytest.mark.parametrize("max_iter", [0, 1, 2, 5])
def test_iteration_limit(max_iter):
    g, prm, A, b = _system((11, 3, 1), 0, np.random.default_rng(12))
    j = solver.JoeGpu(g, prm)
    # no residual meets a negative rule: the loop ends when its count passes the limit
    x, it = j.solveCoupledLinSysNS(A, b, -1.0, -1.0, max_iter)
    assert it == max_iter + 1
    y, it = j.solveCoupledLinSysNS(A, b, -1.0, -1.0, max_iter)   # the same handle, the same bits again
    assert it == max_iter + 1
    np.testing.assert_array_equal(x, y)
    _, it = j.solveCoupledLinSysNS(A, b, 1e30, 0.0, max_iter)    # met at once
    assert it == 1


def test_reported_count_is_that_of_the_stopping_iteration():
    """the host reads the count while the iteration after the one it waited for may be running: with
    every threshold and again and again, the count is that of the iteration that met it"""
    g, prm, A, b = _system((11, 3, 1), 0, np.random.default_rng(5))
    j = solver.JoeGpu(g, prm)
    Di = np.linalg.inv(A[g.nbocv_i[:-1]])
    M = scipy.sparse.bsr_matrix((A, g.nbocv_v, g.nbocv_i), shape=(5 * g.ncv, 5 * g.ncv)).tocsr()

    def norm(x):
        r = b - (M @ x.ravel()).reshape(-1, 5)
        return np.abs(np.einsum("nij,nj->ni", Di, r)).max()
    n = [norm(np.zeros_like(b))] + [norm(j.solveCoupledLinSysNS(A, b, -1.0, -1.0, k)[0]) for k in range(6)]
    for k in range(1, 7):
        # halfway (in the logarithm) between the smallest norm before the k-th and its own: the first met there
        if n[k] >= 0.5 * min(n[:k]):
            continue
        rule = np.sqrt(n[k] * min(n[:k]))
        for _ in range(60):
            assert j.solveCoupledLinSysNS(A, b, rule, 0.0, 50)[1] == k


def test_iterates_above_the_reductions_grid_cap():
    """270,000 unknowns: the dot products' 1,024 blocks stride over them and fill the partial sums"""
    g, prm, A, b = _system((300, 180, 1), 0, np.random.default_rng(8))
    j = solver.JoeGpu(g, prm)
    for iterations in (1, 2, 3):
        x, it = j.solveCoupledLinSysNS(A, b, -1.0, -1.0, iterations - 1)
        assert it == iterations
        want = _bicgstab(g, A, b, iterations)
        # as on the small systems; the sums are seven times longer than the largest of them
        assert np.abs(x - want).max() <= 1e-11 * 10 ** (iterations - 1) * np.abs(want).max()
