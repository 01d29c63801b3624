"""The per-sample kernels at the edges of their layouts: vectors by components and by
rows (from 512 rows on), blocks of 1 to 9 vectors whose dots one or several
warps take, and one or two CTAs in an SM; against the CPU oracle. Rounding of order 1e-15
a step over at most 20 steps: 1e-12 leaves a factor of fifty."""
import numpy as np
import pytest

from conftest import general_csr
from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300.spinsys import GAMMA_E, Electron, SysParam

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000
KEYS = ("P_S", "P_T0", "P_Tp", "P_Tm")
B = np.array([0.01, 0.03, 0.04])


def pair(g1, g2, kT):
    rng = np.random.default_rng(4)
    A1, A2 = (W._tensors(rng, len(g), -2.0, 2.0, True) for g in (g1, g2))
    return SysParam.from_input_units(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.01,
                                     D=W.axial_dipolar(-0.4), kS_per_us=1.0, kT_per_us=kT)


def check(sampler, oracle, s, M, m, method, mode, steps=20):
    rp, col, val = general_csr(oracle, s, B)
    zk = W.random_phase_samples(s.Z, M, seed=m)
    t_end = (steps if m > 2 else 3) * DT
    ref = oracle.trace_sampling(rp, col, val, zk, DT, t_end, m, 1e-6)
    sampler.set_krylov(method)
    sampler.set_sample_path(mode)
    try:
        sampler.build_h(s, B, "general")
        got = sampler.trace_sampling(zk, DT, t_end, m, 1e-6)
        assert sampler.stats()["rounds"] == 1  # a single launch
    finally:
        sampler.set_sample_path("auto")
        sampler.set_krylov("mgs")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12


# dims 432, 576, 864 and 1728
@pytest.mark.parametrize("g1, g2", [((2, 2, 3), (3, 3)), ((2, 2, 3, 2), (3, 2)), ((2, 2, 3), (3, 3, 2)), ((2, 2, 3, 2), (3, 3, 2))])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16, 17])
@pytest.mark.parametrize("method, kT", [("mgs", 0.3), ("mgs", 1.0), ("auto", 1.0)])
@pytest.mark.parametrize("mode", ["on", "single"])
def test_rows(sampler, oracle, g1, g2, m, method, kT, mode):
    check(sampler, oracle, pair(g1, g2, kT), 2, m, method, mode)


@pytest.mark.parametrize("m", [8, 9, 16, 17, 20, 24, 32])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("method, kT", [("mgs", 0.3), ("auto", 1.0)])
def test_ctas_of_an_sm(sampler, oracle, m, more, method, kT):
    """As many samples as SMs, and one more (two CTAs in an SM where their shared
    memory allows)."""
    import torch
    M = torch.cuda.get_device_properties(0).multi_processor_count + more
    check(sampler, oracle, pair((2,), (2, 3), kT), M, m, method, "on")
