"""The general builder's product on blocks (k_spmm_blk) against the product on
the CSR of the same Hamiltonian, given as a CSR. Both carry rounding of order
1e-16 of ||H|| a step: 1e-13 of populations of at most 1 over a few steps; a
wrong list entry or an inexact sum of digits shows at 1e-7 and above."""
import numpy as np
import pytest

from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300.spinsys import GAMMA_E, Electron, SysParam

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000
KEYS = ("P_S", "P_T0", "P_Tp", "P_Tm")


def pair(g1, g2, seed=4, kT=1.0):
    rng = np.random.default_rng(seed)
    A1, A2 = (W._tensors(rng, len(g), -2.0, 2.0, True) for g in (g1, g2))
    return SysParam.from_input_units(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.01,
                                     D=W.axial_dipolar(-0.4), kS_per_us=1.0, kT_per_us=kT)


def difference(a, b):
    return max(np.max(np.abs(getattr(a, k) - getattr(b, k))) for k in KEYS)


@pytest.mark.parametrize("g1, g2", [((3,) * 5, (3,) * 4), ((3,) * 5, (3, 3, 3, 3, 2)), ((3,) * 5, (3,) * 5)])
def test_longest_lists(sampler, g1, g2):
    """18 and 19 neighbours (the most that the blocks take) and 20 (the CSR)."""
    s = pair(g1, g2)
    zk = W.random_phase_samples(s.Z, 2, seed=1)
    sampler.build_h(s, np.array([0.01, 0.03, 0.04]), "general")
    out = {k: [] for k in ("built", "given")}
    for which in out:
        if which == "given":
            sampler.set_h(*sampler.get_h())
        for method in ("mgs", "auto"):
            sampler.set_krylov(method)
            out[which].append(sampler.trace_sampling(zk, DT, 4 * DT, 6, 1e-6))
    sampler.set_krylov("mgs")
    for a, b in zip(out["built"], out["given"]):
        assert difference(a, b) <= 1e-13


@pytest.mark.parametrize("method, kT", [("mgs", 1.0), ("auto", 1.0), ("mgs", 0.3)])
@pytest.mark.parametrize("size", [1.0, 1e4, 1e8])
def test_large_coupling_out_of_reach(sampler, method, kT, size):
    """A nucleus of spin 1 whose one coupling, along z, is large, and states with
    its m = 0 alone: no row of theirs holds the coupling, and the rest of H keeps
    its digits beside it."""
    s = pair((3, 2, 2), (3, 2), kT=kT)
    s.e1.A[0] = np.diag([0.0, 0.0, size])
    s.e1.gamma_I = [0.0] + s.e1.gammas[1:]
    zk = W.random_phase_samples(s.Z, 3, seed=2).reshape(3, 3, -1)
    zk[:, [0, 2]] = 0.0
    zk = zk.reshape(3, -1) / np.linalg.norm(zk.reshape(3, -1), axis=1, keepdims=True)
    out = []
    sampler.set_sample_path("off")
    sampler.set_krylov(method)
    try:
        sampler.build_h(s, np.array([0.01, 0.03, 0.04]), "general")
        out.append(sampler.trace_sampling(zk, DT, 40 * DT, 12, 1e-6))
        sampler.set_h(*sampler.get_h())
        out.append(sampler.trace_sampling(zk, DT, 40 * DT, 12, 1e-6))
    finally:
        sampler.set_krylov("mgs")
        sampler.set_sample_path("auto")
    assert difference(*out) <= 1e-13


def test_memory_held(oracle):
    """A call holds no more device memory than its limit allows, the blocks'
    fragments (1 KB a nuclear index) included: two jobs of a batch of 64
    systems, and a call whose limit has no room for the fragments after one
    that built them."""
    from spin_dynamics_gb300.dynamics import TraceSampler, device_memory
    s = pair((3, 3, 2, 2, 2, 2), (2, 2, 2, 2))
    zk = [W.random_phase_samples(s.Z, 32, seed=k) for k in range(2)]
    fields = [np.array([0.01, 0.03, 0.04]) * (1 + k) for k in range(64)]
    slack = 24 << 20  # the plan, tables and the allocator's granularity
    with TraceSampler(0) as sp:
        sp.set_sample_path("off")
        sp.build_h_batch([s] * 64, fields, "general")
        free0 = device_memory()[0]

        def run(limit):
            sp.set_memory_limit(limit)
            got = sp.trace_sampling_batch(zk, DT, 3 * DT, 4, 1e-6, job_sys=[5, 40])
            return got, free0 - device_memory()[0]

        limit = 64 << 20
        bounded, held = run(limit)
        assert held <= limit + slack
        whole, _ = run(0)
        need = 16 * 2 * s.Z * 4 * 32  # the states
        tight, _ = run(need + (32 << 20))
        for a, b, c in zip(bounded, whole, tight):
            assert difference(a, b) <= 1e-13 and difference(c, b) <= 1e-13


def test_small_gradients_hold_no_tiled_buffers():
    """A gradient whose bases are built a sample per CTA allocates neither block
    fragments nor the tiles' work vectors: the tiled build of the same call then
    takes that much more memory."""
    from spin_dynamics_gb300.dynamics import TraceSampler, device_memory
    s = pair((2, 3, 3), (2,))
    n, jobs = 4 * s.Z, 300
    fields = [np.array([0.01, 0.03, 0.04]) * (1 + 0.01 * k) for k in range(jobs)]
    zk = [W.random_phase_samples(s.Z, 1, seed=1)] * jobs
    held = []
    with TraceSampler(0) as sp:
        for mode in ("auto", "off"):
            sp.set_sample_path(mode)
            sp.yield_gradient_batch([s] * jobs, fields, zk, DT, 2 * DT, 4, n_quad=1, checkpoint_every=1, hyperfine=False)
            held.append(device_memory()[0])
    state = 16 * n * 32 * jobs
    fragments = 2 * jobs * s.Z * 1024
    assert held[0] - held[1] >= 0.9 * (2 * state + fragments)
