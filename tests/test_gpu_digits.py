"""The tensor-core kernels on exact digits and the orthogonalisation in blocks
of eight with integer sums, against the CPU oracle on the tiled path. Every step carries rounding of order 1e-15 of populations of at
most 1 and the windows have at most 60 steps, so 1e-12 leaves a factor of
over ten; a wrong fragment, edge or digit shows at 1e-3 and above (the digit
weights are 1/256 apart)."""
import numpy as np
import pytest

from conftest import general_csr, iso_csr
from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300._native import SpcError
from spin_dynamics_gb300.spinsys import GAMMA_E, Electron, SysParam

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000
KEYS = ("P_S", "P_T0", "P_Tp", "P_Tm")


def pair(g1, g2, seed=4, iso=False, kT=1.0):
    rng = np.random.default_rng(seed)
    A1, A2 = (W._tensors(rng, len(g), -2.0, 2.0, not iso) for g in (g1, g2))
    return SysParam.from_input_units(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.01,
                                     D=W.axial_dipolar(-0.4), kS_per_us=1.0, kT_per_us=kT)


# dims 8 (m above n), 48, 144 and 1296: Z = 2, 12, 36 and 324 rows against 32-row chunks
@pytest.mark.parametrize("g1, g2", [((2,), ()), ((2,), (2, 3)), ((3, 3), (2, 2)), ((3, 2, 2), (3, 3, 3))])
@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 24, 25, 32, 33])
@pytest.mark.parametrize("method, M, kT", [("mgs", 3, 1.0), ("mgs", 33, 0.3), ("auto", 37, 1.0)])
def test_populations(sampler, oracle, g1, g2, m, method, M, kT):
    s = pair(g1, g2, kT=kT)
    B = np.array([0.01, 0.03, 0.04])
    rp, col, val = general_csr(oracle, s, B)
    zk = W.random_phase_samples(s.Z, M, seed=m)
    t_end = (60 if m > 1 else 3) * DT
    ref = oracle.trace_sampling(rp, col, val, zk, DT, t_end, m, 1e-6)
    sampler.set_krylov(method)
    sampler.set_sample_path("off")
    try:
        sampler.build_h(s, B, "general")
        got = sampler.trace_sampling(zk, DT, t_end, m, 1e-6)
    finally:
        sampler.set_sample_path("auto")
        sampler.set_krylov("mgs")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12


@pytest.mark.parametrize("m", [8, 9, 17])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3])
def test_given_csr(sampler, oracle, m, scale):
    """A CSR from the caller (only the FP64 product, its own bound for the
    sums): the oracle's reference Hamiltonian times a scale, over a step that
    keeps scale * dt."""
    s = W.small_pair()
    rp, col, val = iso_csr(oracle, s, 0.05)
    zk = W.random_phase_samples(s.Z, 5, seed=m)
    dt = DT / scale
    ref = oracle.trace_sampling(rp, col, val * scale, zk, dt, 40 * dt, m, 1e-6)
    sampler.set_sample_path("off")
    try:
        sampler.set_h(rp, col, val * scale)
        got = sampler.trace_sampling(zk, dt, 40 * dt, m, 1e-6)
    finally:
        sampler.set_sample_path("auto")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12


def test_undefined_samples_stay_undefined(sampler):
    """A NaN in one sample vector reaches every population of the mean, as in
    FP64 arithmetic: the digits of a NaN are no number."""
    s = pair((3, 3), (2, 2))
    zk = W.random_phase_samples(s.Z, 5)
    zk[3, 7] = np.nan
    sampler.set_sample_path("off")
    try:
        sampler.build_h(s, np.array([0.0, 0.0, 0.05]), "general")
        got = sampler.trace_sampling(zk, DT, 4 * DT, 16, 1e-6)
    finally:
        sampler.set_sample_path("auto")
    for k in KEYS:
        assert np.all(np.isnan(getattr(got, k)[1:5]))


@pytest.mark.parametrize("m", [7, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("more", [0, 1])
def test_dt_loop_forms(sampler, oracle, m, more):
    """As many samples as the dt loop takes on a CTA each, and one more (packed
    into warps up to m = 16)."""
    import torch
    s = pair((2,), (2, 3))
    B = np.array([0.01, 0.03, 0.04])
    M = 7 * torch.cuda.get_device_properties(0).multi_processor_count + more
    rp, col, val = general_csr(oracle, s, B)
    zk = W.random_phase_samples(s.Z, M, seed=m)
    ref = oracle.trace_sampling(rp, col, val, zk, DT, 30 * DT, m, 1e-6)
    sampler.set_sample_path("off")
    try:
        sampler.build_h(s, B, "general")
        got = sampler.trace_sampling(zk, DT, 30 * DT, m, 1e-6)
    finally:
        sampler.set_sample_path("auto")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12


@pytest.mark.parametrize("mode", ["on", "single"])
@pytest.mark.parametrize("m, steps, scale", [(1, 2, 1.0), (2, 9, 1.0), (7, 40, 1.0), (15, 60, 1.0), (16, 60, 1.0),
                                             (17, 60, 1.0), (21, 60, 1.0), (22, 60, 1.0), (31, 60, 1.0), (32, 60, 1.0),
                                             (12, 63, 0.02), (12, 64, 0.02), (12, 65, 0.02), (12, 129, 0.02)])
def test_dt_loop_per_sample(sampler, oracle, mode, m, steps, scale):
    """The per-sample kernels' dt loops at the edges of their thread layouts
    (parts of a row, components past a warp) and of a 64-step history buffer
    (small steps: one basis carries all of them)."""
    s = pair((2,), (2, 3))
    B = np.array([0.01, 0.03, 0.04])
    rp, col, val = general_csr(oracle, s, B)
    zk = W.random_phase_samples(s.Z, 5, seed=m)
    dt = scale * DT
    t_end = (steps - 0.5) * dt
    ref = oracle.trace_sampling(rp, col, val, zk, dt, t_end, m, 1e-6)
    sampler.set_sample_path(mode)
    try:
        sampler.build_h(s, B, "general")
        got = sampler.trace_sampling(zk, dt, t_end, m, 1e-6)
        stats = sampler.stats()
    finally:
        sampler.set_sample_path("auto")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12
    assert stats["krylov_builds"] == int(ref["n_builds"].sum())
    assert stats["sample_steps"] == 5 * steps


@pytest.mark.parametrize("m", [9, 10, 17, 24])
@pytest.mark.parametrize("kT", [1.0, 1.0 + 1e-12, 1.0 + 1e-9, 1.0 + 1e-6, 1.3])
def test_small_coefficients(sampler, oracle, m, kT):
    """Projection coefficients below, around and above the size that is
    subtracted in single precision: they grow with the difference of the rates."""
    s = pair((3, 2, 2), (3, 3, 3), kT=kT)
    B = np.array([0.01, 0.03, 0.04])
    rp, col, val = general_csr(oracle, s, B)
    zk = W.random_phase_samples(s.Z, 33, seed=m)
    ref = oracle.trace_sampling(rp, col, val, zk, DT, 40 * DT, m, 1e-6)
    sampler.set_krylov("mgs")
    sampler.set_sample_path("off")
    try:
        sampler.build_h(s, B, "general")
        got = sampler.trace_sampling(zk, DT, 40 * DT, m, 1e-6)
    finally:
        sampler.set_sample_path("auto")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12


def test_least_memory(sampler):
    """The least memory limit that the call accepts is the same for the general
    builder's Hamiltonian (whose kernel wants a vector's digits beside it) as for
    the reference builder's, and at that limit the populations are the same."""
    s = pair((2, 2, 3), (3, 2), iso=True)
    zk = W.random_phase_samples(s.Z, 40, seed=2)

    def run(limit):
        sampler.set_memory_limit(limit)
        return sampler.trace_sampling(zk, DT, 6 * DT, 2, 1e-6)

    least = []
    sampler.set_sample_path("off")
    try:
        for mode, B in (("reference", 0.05), ("general", np.array([0.0, 0.0, 0.05]))):
            sampler.build_h(s, B, mode)
            whole = run(0)
            lo, hi = 1 << 18, 1 << 24
            while hi - lo > 1:
                mid = (lo + hi) // 2
                try:
                    got = run(mid)
                    hi = mid
                except SpcError:
                    lo = mid
            got = run(hi)
            least.append(hi)
            assert max(np.max(np.abs(getattr(got, k) - getattr(whole, k))) for k in KEYS) <= 1e-13
    finally:
        sampler.set_memory_limit(0)
        sampler.set_sample_path("auto")
    assert least[0] == least[1]


@pytest.mark.parametrize("method", ["mgs", "auto"])
@pytest.mark.parametrize("scale", [2.0**-90, 2.0**-45, 2.0**40, 2.0**105])
def test_extreme_units(sampler, oracle, method, scale):
    """A CSR in units far from those of the builders: scaled by a power of two,
    with dt scaled back, every number keeps its digits, past the range of single
    precision too."""
    s = W.small_pair()
    rp, col, val = iso_csr(oracle, s, 0.05)
    zk = W.random_phase_samples(s.Z, 5, seed=3)
    dt = DT / scale
    ref = oracle.trace_sampling(rp, col, val, zk, DT, 40 * DT, 17, 1e-6)
    sampler.set_krylov(method)
    sampler.set_sample_path("off")
    try:
        sampler.set_h(rp, col, val * scale)
        got = sampler.trace_sampling(zk, dt, 40 * dt, 17, 1e-6)
    finally:
        sampler.set_sample_path("auto")
        sampler.set_krylov("mgs")
    assert max(np.max(np.abs(getattr(got, k) - ref[k])) for k in KEYS) <= 1e-12


@pytest.mark.parametrize("m", [8, 12, 20])
@pytest.mark.parametrize("size", [1e-14, 1e-10, 1e-7, 1e-4])
def test_weak_couplings(sampler, m, size):
    """Hyperfine couplings so weak that a basis passes near an invariant subspace
    of the electrons' part: vectors past it lose orthogonality, and the products
    of basis vectors (single precision but for neighbours where H is Hermitian
    up to a shift) carry the projections. Against the per-sample kernel, whose
    products are all FP64; what is left of a defect reaches the populations
    through the coupling alone."""
    rng = np.random.default_rng(6)
    A1, A2 = ([a * size for a in W._tensors(rng, len(g), -2.0, 2.0, True)] for g in ((3, 2), (2, 2)))
    s = SysParam.from_input_units(Electron(g_I=[3, 2], A=A1), Electron(g_I=[2, 2], A=A2), J=0.01,
                                  D=W.axial_dipolar(-0.4), kS_per_us=1.0, kT_per_us=1.0)
    zk = W.random_phase_samples(s.Z, 5, seed=m)
    sampler.set_krylov("mgs")
    out = {}
    try:
        sampler.build_h(s, np.array([0.01, 0.03, 0.04]), "general")
        for mode in ("off", "single"):
            sampler.set_sample_path(mode)
            out[mode] = sampler.trace_sampling(zk, DT, 40 * DT, m, 1e-6)
    finally:
        sampler.set_sample_path("auto")
    assert max(np.max(np.abs(getattr(out["off"], k) - getattr(out["single"], k))) for k in KEYS) <= 1e-12
