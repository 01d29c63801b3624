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
