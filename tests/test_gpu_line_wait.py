"""A wait of the LINE substitutions that runs out: the kernel ends by itself, the call reports
JG_ERR_CUDA, and the handle works again.  A library loaded before libjoe_b200.so stands in for
launch_line_relax and passes it on with no tries for a wait, so nothing hangs."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

STAND_IN = r"""
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
#include "jg_internal.h"
static int no_tries = 0;
extern "C" void stand_in_set(int on) { no_tries = on; }
namespace jg {
void launch_line_relax(const Mesh& m, const Params& p, State& st, const Lines& L, int bs, int sweeps, cudaStream_t s,
                       int tries) {
  typedef void (*F)(const Mesh&, const Params&, State&, const Lines&, int, int, cudaStream_t, int);
  static F real = (F)dlsym(dlopen(getenv("JOE_LIB"), RTLD_NOLOAD | RTLD_LAZY),
                           "_ZN2jg17launch_line_relaxERKNS_4MeshERKNS_6ParamsERNS_5StateERKNS_5LinesEiiP11CUstream_sti");
  if (!real) abort();
  real(m, p, st, L, bs, sweeps, s, no_tries ? 0 : tries);
}
}
"""

RUN = r"""
import ctypes, dataclasses, os, sys
import numpy as np
sys.path.insert(0, os.environ["JOE_ROOT"])
from myjoe_b200 import case, solver
stand_in = ctypes.CDLL(os.environ["LD_PRELOAD"])
call, model, precision = sys.argv[1], sys.argv[2], int(sys.argv[3])
if model == "SA":
    _, g, prm = case.sa_bump_case(24, 16, 2, stretch=1.25, n_prism=4, alternate=True)
elif model == "SST":
    _, g, prm = case.sst_bump_case(24, 16, 2, stretch=1.25, n_prism=4, alternate=True)
else:
    _, g, prm = case.plate_case(24, 16, 2)
prm = dataclasses.replace(prm, LINEAR_SOLVER_NS="LINE", LS_MAX_ITER=3)
st = case.perturbed_state(g.x_cv, prm, 0.01)

def handle():
    j = solver.JoeGpu(g, prm, precision=precision)
    j.set_state(*st)
    if model == "SA":
        j.set_scalars(np.full(g.ncv, prm.NUSA_INITIAL))
    if model == "SST":
        j.set_scalars(np.tile([prm.KINE_INITIAL, prm.OMEGA_INITIAL], (g.ncv, 1)))
    return j

def run(j):
    if call == "step":
        return [j.runBackwardEuler(2), *j.get_state()]
    if call == "step_host":
        h = [np.array(x, order="C") for x in st]
        j.step_host(*h, 1)
        return h
    rng = np.random.default_rng(1)
    A = rng.standard_normal((g.nbocv_v.shape[0], 5, 5))
    A[g.nbocv_i[:-1]] += 40.0 * np.eye(5)
    return [j.solveCoupledLinSysNS(A, rng.standard_normal((g.ncv, 5)), 0.0, 0.0, 3)[0]]

ok = handle()
want = run(ok)
stand_in.stand_in_set(1)
j = handle()
try:
    run(j)
    print("no error")
except solver.JoeGpuError as e:
    print("code", e.code, e)
stand_in.stand_in_set(0)
again = handle()                       # the context still works
for a, b in zip(want, run(again)):
    np.testing.assert_array_equal(a, b)
if call == "solve":                    # this very handle too: its call keeps nothing but the matrix
    for a, b in zip(want, run(j)):
        np.testing.assert_array_equal(a, b)
print("done")
"""


@pytest.fixture(scope="module")
def stand_in(tmp_path_factory):
    from myjoe_b200 import build
    build.build()
    d = tmp_path_factory.mktemp("stand_in")
    src, so = d / "stand_in.cpp", d / "stand_in.so"
    src.write_text(STAND_IN)
    subprocess.run([build._nvcc(), "-std=c++17", "-x", "cu", *build.NVCC_FLAGS[:2], "-shared", "-Xcompiler", "-fPIC",
                    "-I" + build.CSRC, str(src), "-o", str(so), "-ldl"], check=True)
    return str(so), build.LIB


def _run(stand_in, *args):
    so, lib = stand_in
    env = dict(os.environ, LD_PRELOAD=so, JOE_LIB=lib, JOE_ROOT=ROOT)
    r = subprocess.run([sys.executable, "-c", RUN, *args], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout


@pytest.mark.parametrize("model,precision", [("none", 0), ("none", 1), ("SA", 0), ("SA", 1), ("SST", 0), ("SST", 1)])
def test_a_step_whose_wait_runs_out_is_a_cuda_error(stand_in, model, precision):
    out = _run(stand_in, "step", model, str(precision))
    assert "code -2" in out and "asynchronous copy" in out and "done" in out, out


@pytest.mark.parametrize("call", ["step_host", "solve"])
@pytest.mark.parametrize("model,precision", [("none", 0), ("none", 1)])
def test_every_call_reports_it(stand_in, call, model, precision):
    """not as a diverged state (step_host), nor as success (one linear solve)"""
    out = _run(stand_in, call, model, str(precision))
    assert "code -2" in out and "asynchronous copy" in out and "done" in out, out
