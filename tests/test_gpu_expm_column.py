"""The stepwise yields' exponential columns (a Taylor series of the vector, and
the full exponential past ||dt H|| = 64) against the dense model, in Krylov
spaces that hold the whole space (m = n), so that the exponential is the only
approximation. A step's phase carries rounding of eps ||dt H|| <= 4e-14 here, a
window of 8 steps 3e-13 of a population of at most 1: 1e-11 leaves a factor of
thirty; a wrong substep or branch shows at order one."""
import numpy as np
import pytest

import dense
from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300.dynamics import num_time_points
from spin_dynamics_gb300.spinsys import GAMMA_E, Electron, SysParam

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000


# dt ||H||: below 1, some substeps, just under the line, past it
@pytest.mark.parametrize("Bz", [0.05, 20.0, 150.0, 600.0])
@pytest.mark.parametrize("g1, g2", [((2,), (2,)), ((3,), (2, 2)), ((2,), (2, 3))])
@pytest.mark.parametrize("method", ["mgs", "lanczos"])
def test_yields_of_strong_fields(sampler, Bz, g1, g2, method):
    rng = np.random.default_rng(6)
    A1, A2 = (W._tensors(rng, len(g), -1.5, 1.5, True) for g in (g1, g2))
    s = SysParam(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.03, D=W.axial_dipolar(-0.3),
                 kS=0.2, kT=0.2)
    B = np.array([0.1 * Bz, 0.0, Bz])
    zk = W.random_phase_samples(s.Z, 3, seed=2)
    t_end = 8 * DT
    sampler.set_krylov(method)
    try:
        got = sampler.stepwise_yields(s, B, zk, DT, t_end, 4 * s.Z)
    finally:
        sampler.set_krylov("mgs")
    H = dense.hamiltonian(s.e1.g_I, A1, s.e2.g_I, A2, B, s.J, s.D, s.kS, s.kT)
    ref = dense.stepwise_yields(H, zk, DT, num_time_points(DT, t_end), s.kS, s.kT)
    assert np.max(np.abs(np.subtract(got, ref))) <= 1e-11


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 32])
@pytest.mark.parametrize("method", ["mgs", "lanczos"])
def test_gradient_basis_per_sample(sampler, m, method):
    """The per-sample basis build of small gradients against the tiled one,
    over blocks of eight vectors and uneven jobs (dims 12, 48 and 288): the
    same model, so gradients differ by rounding of the steps, below 1e-13 of
    their norm for 4 steps (a wrong vector shows at its own size)."""
    rng = np.random.default_rng(9)
    systems = []
    for g1, g2 in (((3,), ()), ((2,), (2, 3)), ((2, 2, 3), (3, 2))):
        A1, A2 = (W._tensors(rng, len(g), -1.5, 1.5, True) for g in (g1, g2))
        systems.append(SysParam(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.03,
                                D=W.axial_dipolar(-0.3), kS=0.02, kT=0.02))
    fields = [np.array([0.02, 0.03, 0.04])] * 3
    zks = [W.random_phase_samples(s.Z, M, seed=M) for s, M in zip(systems, (1, 33, 5))]
    out = {}
    sampler.set_krylov(method)
    try:
        for mode in ("auto", "off"):
            sampler.set_sample_path(mode)
            out[mode] = sampler.yield_gradient_batch(systems, fields, zks, DT, 4 * DT, m)
    finally:
        sampler.set_sample_path("auto")
        sampler.set_krylov("mgs")
    for a, b in zip(out["auto"], out["off"]):
        assert abs(a.Phi_S - b.Phi_S) <= 1e-13 and abs(a.Phi_T - b.Phi_T) <= 1e-13
        assert np.linalg.norm(a.raw - b.raw) <= 1e-13 * np.linalg.norm(b.raw)


@pytest.mark.parametrize("method, m", [("mgs", 1), ("mgs", 7), ("mgs", 9), ("mgs", 17), ("mgs", 32), ("lanczos", 16)])
@pytest.mark.parametrize("g1, g2, M, kT", [((3, 2), (2, 2), 1, 0.02), ((3, 3), (3,), 7, 0.02), ((2, 2, 3), (3, 2), 3, 0.05),
                                           ((3, 2), (2, 3), 40, 0.02)])
def test_gradient_basis_on_clusters(sampler, method, m, g1, g2, M, kT):
    """A sample's rows over clusters of four and two CTAs (dims 96, 108, 288 and
    144) against the tiled build, to the same 1e-13."""
    if method == "lanczos":
        kT = 0.02  # equal rates
    rng = np.random.default_rng(11)
    A1, A2 = (W._tensors(rng, len(g), -1.5, 1.5, True) for g in (g1, g2))
    s = SysParam(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.03, D=W.axial_dipolar(-0.3), kS=0.02,
                 kT=kT)
    zk = W.random_phase_samples(s.Z, M, seed=M)
    out = {}
    sampler.set_krylov(method)
    try:
        for mode in ("auto", "off"):
            sampler.set_sample_path(mode)
            out[mode] = sampler.yield_gradient_batch([s], [np.array([0.02, 0.03, 0.04])], [zk], DT, 4 * DT, m)[0]
    finally:
        sampler.set_sample_path("auto")
        sampler.set_krylov("mgs")
    a, b = out["auto"], out["off"]
    assert abs(a.Phi_S - b.Phi_S) <= 1e-13 and abs(a.Phi_T - b.Phi_T) <= 1e-13
    assert np.linalg.norm(a.raw - b.raw) <= 1e-13 * np.linalg.norm(b.raw)
