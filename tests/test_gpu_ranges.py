"""Hamiltonians far from the builders' units and of uneven scale, against the
CPU oracle in ordinary units. Scaling H by a power of two and dt back changes no
digit of a product, and a part of H that the state never enters changes
nothing, so each case has the rounding of the plain one: of order 1e-15 a step,
at most 60 steps, 1e-12 of populations of at most 1. Lost bits show at 1e-10 and
above."""
import numpy as np
import pytest

from conftest import iso_csr
from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300.spinsys import GAMMA_E

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000
KEYS = ("P_S", "P_T0", "P_Tp", "P_Tm")


def worst(got, ref):
    return max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS)


def given(sampler, rp, col, val, zk, dt, steps, m, method, mode):
    sampler.set_krylov(method)
    sampler.set_sample_path(mode)
    try:
        sampler.set_h(rp, col, val)
        return sampler.trace_sampling(zk, dt, steps * dt, m, 1e-6)
    finally:
        sampler.set_sample_path("auto")
        sampler.set_krylov("mgs")


@pytest.mark.parametrize("mode", ["off", "on", "single"])
@pytest.mark.parametrize("m", [9, 17])
@pytest.mark.parametrize("power", [-150, 130, 150])
def test_past_single_precision(sampler, oracle, mode, m, power):
    """Coefficients past the range of single precision."""
    s = W.small_pair()
    rp, col, val = iso_csr(oracle, s, 0.05)
    zk = W.random_phase_samples(s.Z, 5, seed=3)
    ref = oracle.trace_sampling(rp, col, val, zk, DT, 40 * DT, m, 1e-6)
    assert worst(given(sampler, rp, col, val * 2.0**power, zk, DT * 2.0**-power, 40, m, "mgs", mode), ref) <= 1e-12


@pytest.mark.parametrize("mode", ["off", "on", "single"])
@pytest.mark.parametrize("method", ["mgs", "auto"])
@pytest.mark.parametrize("power", [-480, -420, 420, 480])
def test_units_to_the_range_of_squares(sampler, oracle, mode, method, power):
    """Square norms to the ends of a double's range."""
    s = W.small_pair()
    rp, col, val = iso_csr(oracle, s, 0.05)
    zk = W.random_phase_samples(s.Z, 5, seed=3)
    ref = oracle.trace_sampling(rp, col, val, zk, DT, 40 * DT, 17, 1e-6)
    assert worst(given(sampler, rp, col, val * 2.0**power, zk, DT * 2.0**-power, 40, 17, method, mode), ref) <= 1e-12


def beside(rp, col, val, scale):
    """H on one half of the nuclear indices and scale * H on the other: the CSR
    of both, interleaved as (electron, half, index)."""
    n = len(rp) - 1
    Z = n // 4
    row = np.repeat(np.arange(n), np.diff(rp))

    def place(r, half):
        return (r // Z) * 2 * Z + half * Z + r % Z

    r = np.concatenate([place(row, k) for k in (0, 1)])
    c = np.concatenate([place(np.asarray(col, np.int64), k) for k in (0, 1)])
    v = np.concatenate([val, val * scale])
    o = np.lexsort((c, r))
    rp2 = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=2 * n))])
    return rp2.astype(np.int32), c[o].astype(np.int32), v[o]


@pytest.mark.parametrize("mode", ["off", "on", "single"])
@pytest.mark.parametrize("method, kT", [("mgs", 0.0), ("auto", 0.0), ("mgs", 1e-3), ("mgs", 0.3)])
@pytest.mark.parametrize("m", [9, 17])
@pytest.mark.parametrize("power", [0, 20, 30, 40, 50])
def test_large_part_beside(sampler, oracle, mode, method, kT, m, power):
    """States confined to a part of H that a larger one bounds."""
    s = W.small_pair()
    s.kS, s.kT = 0.0, kT
    rp, col, val = iso_csr(oracle, s, 0.05)
    zk = W.random_phase_samples(s.Z, 5, seed=3)
    ref = oracle.trace_sampling(rp, col, val, zk, DT, 40 * DT, m, 1e-6)
    z2 = np.concatenate([zk, np.zeros_like(zk)], axis=1)
    assert worst(given(sampler, *beside(rp, col, val, 2.0**power), z2, DT, 40, m, method, mode), ref) <= 1e-12
