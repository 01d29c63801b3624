"""A Hamiltonian that does not fit leaves the handle without one: calls on it are
refused, and a later build works as ever."""
import numpy as np
import pytest

from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300._native import SpcError
from spin_dynamics_gb300.dynamics import TraceSampler, device_memory
from spin_dynamics_gb300.spinsys import GAMMA_E, Electron, SysParam

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000
B = np.array([0.01, 0.03, 0.04])


def pair(g1, g2):
    rng = np.random.default_rng(4)
    A1, A2 = (W._tensors(rng, len(g), -2.0, 2.0, True) for g in (g1, g2))
    return SysParam.from_input_units(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.01,
                                     D=W.axial_dipolar(-0.4), kS_per_us=1.0, kT_per_us=1.0)


@pytest.mark.parametrize("batch", [False, True])
def test_calls_after_a_failed_build(batch):
    import torch
    small, large = pair((2,), (2, 3)), pair((2,) * 10, (2,) * 9)  # the large one's entries take 4 GB
    zk = W.random_phase_samples(small.Z, 3, seed=1)
    hog = []
    with TraceSampler(0) as sp:
        def run():
            if batch:
                return sp.trace_sampling_batch([zk], DT, 5 * DT, 8, 1e-6)[0].P_S
            return sp.trace_sampling(zk, DT, 5 * DT, 8, 1e-6).P_S

        def build(s):
            return sp.build_h_batch([s], [B], "general") if batch else sp.build_h(s, B, "general")

        build(small)
        before = run()
        try:
            while device_memory()[0] > 2 << 30:  # all but two gigabytes
                hog.append(torch.empty(max(1 << 20, device_memory()[0] - (3 << 29)), dtype=torch.uint8, device="cuda"))
            with pytest.raises(SpcError):
                build(large)
        finally:
            hog.clear()
            torch.cuda.empty_cache()
        with pytest.raises(SpcError):
            run()
        build(small)
        assert np.array_equal(run(), before)
