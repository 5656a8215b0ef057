"""Launch shapes of the 5x5 path (jg_set_launch_config / jg_autotune).

The two Jacobi sweep kernels do the same arithmetic in the same order, so a
step gives bit-identical results with either; the face-loop shapes (fused or
split into residual and Jacobian kernels, lanes per cell) change only the
order of each cell's diagonal-block and residual sums and the form of the Roe
dissipation matrix, so steps agree to rounding (1e-12 relative after 10 steps).  The autotuner
returns a valid shape and per-shape times, and a batch and its cases alone
stay bit-identical under a shared shape."""
import dataclasses

import numpy as np
import pytest

from myjoe_b200 import case, solver

pytestmark = pytest.mark.gpu


def _plate(solver_name="JACOBI"):
    _, g, prm = case.plate_case(96, 48, 2)
    return g, dataclasses.replace(prm, LINEAR_SOLVER_NS=solver_name, LS_MAX_ITER=8, CFL=5.0)


def _run(g, prm, shape=None, nsteps=10):
    j = solver.JoeGpu(g, prm)
    if shape:
        j.set_launch_config(*shape)
    j.set_state(*case.perturbed_state(g.x_cv, prm, 0.02))
    r = j.runBackwardEuler(nsteps)
    st = j.get_state()
    cfg = j.launch_config()
    j.close()
    return st, r, cfg


def test_sweep_kernels_are_bitwise_equal():
    g, prm = _plate()
    a = _run(g, prm, (2, 0))
    b = _run(g, prm, (2, 1))
    assert b[2] == (2, 1)
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)


# fused shapes (1, 4, 17) and split shapes (residual and Jacobian kernels: 32 + lanes per cell)
@pytest.mark.parametrize("cl", [1, 4, 17, 33, 34, 36, 40])
def test_lanes_per_cell_agree_to_rounding(cl):
    g, prm = _plate("SGS")
    a = _run(g, prm, (2, 0))
    b = _run(g, prm, (cl, 0))
    for x, y in zip(a[0], b[0]):
        assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()
    np.testing.assert_allclose(b[1], a[1], rtol=1e-10)


def test_autotune_picks_a_valid_shape_and_keeps_results():
    g, prm = _plate("SGS")
    j = solver.JoeGpu(g, prm)
    j.set_state(*case.perturbed_state(g.x_cv, prm, 0.02))
    cl, rv, ms = j.autotune(3)
    shapes = (1, 2, 4, 17, 33, 34, 36, 40)
    assert cl in shapes and rv in (0, 1)
    assert all(v > 0.0 for v in ms.values())
    assert ms["flux_cl%d" % cl] == min(ms["flux_cl%d" % s] for s in shapes)
    r = j.runBackwardEuler(10)   # the tuned shape is captured at the next step
    assert np.all(np.isfinite(r))
    ref = _run(g, prm, (cl, rv))
    for x, y in zip(j.get_state(), ref[0]):
        np.testing.assert_array_equal(x, y)
    j.close()


def test_batch_bitwise_under_a_shared_shape():
    cs = []
    for k, (nx, ny) in enumerate([(24, 12), (40, 16)]):
        _, g, prm = case.bump_case(nx, ny, 2, jitter=0.1, seed=k)
        cs.append((g, dataclasses.replace(prm, LINEAR_SOLVER_NS="SGS", LS_MAX_ITER=6, CFL=2.0)))
    b = solver.JoeGpuBatch(cs)
    b.set_launch_config(4, 1)
    for k, (g, prm) in enumerate(cs):
        b.set_case_state(k, *case.perturbed_state(g.x_cv, prm, 0.02))
    b.runBackwardEulerCases(8)
    for k, (g, prm) in enumerate(cs):
        st, _, _ = _run(g, prm, (4, 1), nsteps=8)
        for x, y in zip(b.get_case_state(k), st):
            np.testing.assert_array_equal(x, y)
    b.close()


def _sweep_kernels(j, g):
    """names of the kernels of one Jacobi solve"""
    from torch.profiler import ProfilerActivity, profile
    rng = np.random.default_rng(3)
    A = rng.standard_normal((g.nbocv_v.shape[0], 5, 5))
    A[g.nbocv_i[:-1]] += 40.0 * np.eye(5)
    b = rng.standard_normal((g.ncv, 5))
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        x, _ = j.solveCoupledLinSysNS(A, b, 0.0, 0.0, 3)
    names = {e.key for e in prof.key_averages()}
    return x, {k for k in ("k_sweep", "k_jacobi") if any(k in n for n in names)}


# an FP32 sweep a cell per thread where its grid fills the GPU: 9k cells no, 224k in one layer yes, 350k
# (a wave and a fifth of it) no, 500k (a wave and two thirds) yes; FP64 never
@pytest.mark.parametrize("dims,precision,default", [((96, 48, 2), 1, 0), ((560, 400, 1), 1, 1), ((560, 400, 1), 0, 0),
                                                    ((500, 350, 2), 1, 0), ((714, 350, 2), 1, 1)])
def test_the_sweep_kernel_asked_for_runs(dims, precision, default):
    _, g, prm = case.bump_case(*dims)
    prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="JACOBI", LS_MAX_ITER=3)
    j = solver.JoeGpu(g, prm, precision=precision)
    assert j.launch_config() == (36, default)
    out = []
    for variant in (None, 0, 1):
        if variant is not None:
            j.set_launch_config(36, variant)
        x, ran = _sweep_kernels(j, g)
        assert ran == {("k_sweep", "k_jacobi")[default if variant is None else variant]}
        out.append(x)
    np.testing.assert_array_equal(out[1], out[0])
    np.testing.assert_array_equal(out[2], out[0])
    j.close()


def test_autotune_times_the_split_shape_once():
    """its four names are one shape: one time, and the name chosen is the default's, not the noise's"""
    g, prm = _plate()
    j = solver.JoeGpu(g, prm, jac_lag=4)   # a lagged handle has the split shape only
    j.set_state(*case.perturbed_state(g.x_cv, prm, 0.02))
    for _ in range(4):
        cl, _, ms = j.autotune(2)
        assert cl == 36 and len({ms["flux_cl%d" % (32 + k)] for k in (1, 2, 4, 8)}) == 1
    j.close()
