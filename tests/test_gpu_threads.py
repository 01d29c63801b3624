"""Handles of several threads at once, each with a Krylov dimension of its own:
every call gives what it gives alone. A kernel's limit of dynamic shared memory
belongs to the process, so no call may set it below what another one needs."""
import threading

import numpy as np
import pytest

from spin_dynamics_gb300 import workloads as W
from spin_dynamics_gb300.dynamics import TraceSampler
from spin_dynamics_gb300.spinsys import GAMMA_E, Electron, SysParam

pytestmark = pytest.mark.gpu
DT = 1.0 * GAMMA_E / 1000
KEYS = ("P_S", "P_T0", "P_Tp", "P_Tm")


def pair(g1, g2, kT=1.0):
    rng = np.random.default_rng(4)
    A1, A2 = (W._tensors(rng, len(g), -2.0, 2.0, True) for g in (g1, g2))
    return SysParam.from_input_units(Electron(g_I=list(g1), A=A1), Electron(g_I=list(g2), A=A2), J=0.01,
                                     D=W.axial_dipolar(-0.4), kS_per_us=1.0, kT_per_us=kT)


def populations(mode, m):
    s = pair((2,), (2, 3))
    zk = W.random_phase_samples(s.Z, 3, seed=m)

    def call(sp):
        sp.set_sample_path(mode)
        sp.build_h(s, np.array([0.01, 0.03, 0.04]), "general")
        got = sp.trace_sampling(zk, DT, 6 * DT, m, 1e-6)
        return np.stack([getattr(got, k) for k in KEYS])
    return call


def gradient(mode, m):
    s = pair((2,), (2, 3))
    zk = W.random_phase_samples(s.Z, 3, seed=m)

    def call(sp):
        sp.set_sample_path(mode)
        return sp.yield_gradient_batch([s], [np.array([0.01, 0.03, 0.04])], [zk], DT, 2 * DT, m)[0].raw
    return call


@pytest.mark.parametrize("kind, mode, dims", [(populations, "off", (4, 18, 32, 48)), (populations, "on", (4, 14, 24, 32)),
                                              (populations, "single", (4, 14, 24, 32)), (gradient, "off", (4, 18, 32, 48)),
                                              (gradient, "auto", (4, 14, 24, 32))])
def test_krylov_dimensions_side_by_side(kind, mode, dims):
    calls = [kind(mode, m) for m in dims]
    with TraceSampler(0) as sp:
        alone = [c(sp) for c in calls]
    go = threading.Barrier(len(calls))
    wrong = []

    def work(call, ref):
        try:
            with TraceSampler(0) as sp:
                go.wait()
                for _ in range(60):
                    if not np.array_equal(call(sp), ref):
                        wrong.append("differs")
                        return
        except Exception as e:  # noqa: BLE001
            wrong.append(str(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
