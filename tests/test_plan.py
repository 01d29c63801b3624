"""The library's host arithmetic of bounds and memory plans (spc_plan.h),
compiled by itself."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import ROOT

DRIVER = """
#include "spc_plan.h"
extern "C" double csr_bound(int n, const int* rp, const int* cl, const double* v) {
  return spc::csr_norm_bound(n, rp, cl, v);
}
// a sweep of m basis vectors and states of one unit, partial sums of `part` a node
extern "C" int grad_plan(int nsteps, int nq, int K, double avail, double slack, double m, double part, int* out) {
  const spc::GradPlan p = spc::plan_gradient(nsteps, nq, K, avail, slack, [&](int k, bool keep, int nodes) {
    return m + 4.0 + nodes * (1.0 + part) + (nsteps / k + 1) + (k + 1) + (keep ? (double)k * nq : (double)nq);
  });
  out[0] = p.K;
  out[1] = p.keep;
  out[2] = p.nodes;
  return p.fits;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, so = d / "driver.cpp", d / "driver.so"
    src.write_text(DRIVER)
    cxx = shutil.which(os.environ.get("CXX", "g++")) or "g++"
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "spin_dynamics_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.csr_bound.restype = C.c_double
    return lib


def bound(plan, A):
    A = sp.csr_matrix(A)
    rp, cl = A.indptr.astype(np.int32), A.indices.astype(np.int32)
    v = np.ascontiguousarray(A.data.astype(np.complex128))
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    return plan.csr_bound(A.shape[0], ptr(rp), ptr(cl), ptr(v))


@pytest.mark.parametrize("n", [4, 40, 400])
@pytest.mark.parametrize("hermitian", [True, False])
def test_norm_bound(plan, n, hermitian):
    """At least the 2-norm, at most the row sum of a Hermitian matrix, whatever
    the dimension."""
    rng = np.random.default_rng(n)
    A = sp.random(n, n, 0.2, random_state=rng, format="csr") + 1j * sp.random(n, n, 0.2, random_state=rng, format="csr")
    if hermitian:
        A = A + A.getH()
    b = bound(plan, A)
    assert b >= np.linalg.norm(A.toarray(), 2) * (1.0 - 1e-12)
    sums = abs(A.real) + abs(A.imag)
    row, col = sums.sum(1).max(), sums.sum(0).max()
    assert b <= np.sqrt(row * col) * (1.0 + 1e-12)
    if hermitian:
        assert b <= row * (1.0 + 1e-12)


def test_norm_bound_of_undefined_entries(plan):
    assert np.isnan(bound(plan, np.diag([1.0, np.nan, 2.0, 3.0])))
    assert bound(plan, np.zeros((4, 4))) == 0.0
    assert np.isfinite(bound(plan, np.eye(4) * 1e300))


def planned(plan, nsteps, nq, K, avail, slack=0.0, m=16.0, part=0.0):
    out = (C.c_int * 3)()
    fits = plan.grad_plan(nsteps, nq, K, C.c_double(avail), C.c_double(slack), C.c_double(m), C.c_double(part), out)
    return tuple(out) + (bool(fits),)


def need(nsteps, nq, K, keep, nodes, m=16.0, part=0.0):
    return m + 4 + nodes * (1 + part) + (nsteps // K + 1) + (K + 1) + (K * nq if keep else nq)


@pytest.mark.parametrize("part", [0.0, 0.5, 30.0])
@pytest.mark.parametrize("K", [0, 1, 5, 40])
@pytest.mark.parametrize("nsteps, nq", [(1, 1), (40, 6), (40, 16)])
def test_gradient_plan(plan, nsteps, nq, K, part):
    """At every size of memory: the plan fits; kept node states and the spacing
    are those that one costate state at a time allows, so that more of them never
    cost a build; partial sums shrink the nodes before they refuse a call."""
    K = min(K, nsteps)
    least = need(nsteps, nq, K or max(1, round(nsteps ** 0.5)), False, 1, part=part)
    for avail in np.unique(np.concatenate([np.arange(least - 3, least + 60), np.linspace(least, 900, 200)])):
        k, keep, nodes, fits = planned(plan, nsteps, nq, K, avail, part=part)
        kept = [c for c in ([K] if K else range(1, nsteps + 1)) if need(nsteps, nq, c, True, 1, part=part) <= avail]
        assert fits == (bool(kept) or avail >= least)
        assert bool(keep) == bool(kept)
        if K:
            assert k == K
        elif kept:
            assert (nsteps - 1) // k * k == min((nsteps - 1) // c * c for c in kept)
        if fits:
            assert need(nsteps, nq, k, bool(keep), nodes, part=part) <= avail
            assert nodes == nq or need(nsteps, nq, k, bool(keep), nodes + 1, part=part) > avail


def test_gradient_plan_uses_the_reserve_for_small_buffers(plan):
    assert planned(plan, 40, 6, 8, need(40, 6, 8, False, 1) - 5, slack=5.0)[3]
    assert not planned(plan, 40, 6, 8, need(40, 6, 8, False, 1) - 6, slack=5.0)[3]
