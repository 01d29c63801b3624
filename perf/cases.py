"""Performance cases: the work a user has this package do, through its public entry points.

A case names its radical pairs by their nuclear multiplicities, "radical 1|radical 2" (2 = 1H, 3 = 14N, others =
total spins of symmetry groups), several pairs separated by ";". Couplings, fields and sample vectors come from the
seed. `kind` is the entry point:

  trace      TraceSampler.build_h + trace_sampling, host vectors in, populations out (what the drivers call per field)
  torch      the same on CUDA tensors (torch_ops.trace_sampling)
  batch      build_h_batch + trace_sampling_batch: every (pair, field) job in one call (field scans, orientation sets)
  grad       torch_ops.yield_objective and its backward (every parameter's derivative)
  gradbatch  yield_gradient_batch with the field set of derivatives (compass maps over symmetry blocks)

Every run builds its Hamiltonians: a program that scans fields or fits couplings does so for each call.
"""
import math

import numpy as np
import torch

from spin_dynamics_gb300 import torch_ops
from spin_dynamics_gb300.dynamics import TraceSampler
from spin_dynamics_gb300.spinsys import Electron, SysParam

GAMMA_E = 176.08596      # electron, 1/(us mT)
GAMMA_1H = 0.26752218708
GAMMA_14N = 0.0193297792
TOL = 1e-5
STATES = ("singlet", "T0", "Tp", "Tm")
# The two 14N + five 1H | one 14N + four 1H pair of the repository's benchmark, dimension 55296.
LARGE = "3,3,2,2,2,2,2|3,2,2,2,2"
# Pairs of 2-10 nuclei with dimensions 16-9216, as the repository's uneven set draws them.
UNEVEN = ("2|2;2,3|2;2,2|2,2;3,2|2,2;2,2,3|2;3,3|2,2;2,2,2|2,2,3;3,2,2|3,2,2;2,2,2,2|2,2,2;3,3,2|2,2,2;"
          "2,2,2,2|3,2,2,2;3,3,2,2|2,2,2;3,2,2,2|2,2,2,2,2;3,3,2,2,2|2,2,2,2")
# Total-spin blocks of two radicals with groups of four equivalent 1H beside a 14N.
BLOCKS = "3,5,3|3,3;3,3,3,1|3,5,3;3,5,5|3,5;3,1,3|3,3,1;3,5,3,3|3,5,1;3,1,1|3,1"


def _case(name, kind, systems, samples, m, steps, **more):
    c = dict(name=name, kind=kind, systems=systems, samples=samples, m=m, steps=steps, dt_ns=1.0, mode="general",
             method="auto", kS=1.0, kT=1.0, fields=1, state="singlet")
    c.update(more)
    return c


def listed():
    return [
        # the example input of the original program: 48 rows, half-nanosecond steps, the drivers' default method
        _case("example_48", "trace", "2|2,3", "16", 10, 500, dt_ns=0.5, mode="reference", method="mgs", kS=0.0, kT=0.0),
        # the small pair that is run on a CPU: the whole 5 us window
        _case("pair_288", "trace", "2,2,3|3,2", "64", 20, 5000, mode="reference"),
        # unequal recombination rates (no Hermitian shift), anisotropic couplings, an odd number of samples
        _case("rates_288", "trace", "2,2,3|3,2", "201", 20, 100, method="mgs", kT=0.2),
        # a field scan as the drivers run it: every field value one job, the default method
        _case("scan_2304", "batch", "3,3,2,2|2,2,2,2", "64", 16, 120, mode="reference", method="mgs", fields=6),
        # uneven pairs x orientations in one call
        _case("uneven", "batch", UNEVEN, "32;77;256;64;200;131;96;64;50;128;33;100;64;32", 16, 20, fields=3),
        # one mid-size pair on device tensors, samples that do not fill their last tile
        _case("ragged_2304", "torch", "3,3,2,2|2,2,2,2", "77", 20, 150),
        # unequal rates at 9216 rows: full orthogonalisation is the only method
        _case("rates_9216", "torch", "3,3,2,2,2,2|2,2,2,2", "64", 24, 40, method="mgs", kT=0.1),
        # the large pair in the form the original program accepts, the drivers' default method
        _case("large_iso", "trace", LARGE, "32", 30, 60, mode="reference", method="mgs"),
        # the benchmark's large pair, a slice of its 2 us window
        _case("large", "torch", LARGE, "512", 30, 54),
        # fitting the couplings of a small pair
        _case("grad_288", "grad", "2,2,3|3,2", "32", 16, 20, method="mgs"),
        # the same at a size where the states no longer fit the caches, three-term recurrence
        _case("grad_13824", "grad", "3,3,2,2,2,2|3,2,2,2", "64", 24, 6, method="lanczos"),
        # a compass map's field derivatives over symmetry blocks
        _case("blocks_grad", "gradbatch", BLOCKS, "32", 20, 6, fields=2, method="mgs"),
    ]


def _dims(c):
    return [math.prod(int(x) for x in s.replace("|", ",").split(",") if x) for s in c["systems"].split(";")]


def _samples(c):
    k = [int(x) for x in c["samples"].split(";")]
    return k * len(_dims(c)) if len(k) == 1 else k


def work(case):
    """The vectors in and the populations (gradients) out, and the arithmetic of the method: bases of m products with
    H, each carried over about 0.9 m steps of 1 ns (twice that for isotropic couplings), orthogonalised against two
    vectors where H is Hermitian but for a shift and against all otherwise, the four quadratic forms and the new state.
    A gradient needs a basis each step forward and back, and the reduced matrices of its quadrature nodes."""
    c = case
    flops = 0.0
    byts = 0.0
    T = c["steps"] + 2
    for s, Z, M in zip(c["systems"].split(";"), _dims(c), _samples(c)):
        n, m = 4 * Z, min(c["m"], 4 * Z)
        nn = len([x for x in s.replace("|", ",").split(",") if x])
        row = 2 + 2.2 * nn if c["mode"] == "general" else 2 + 0.5 * nn
        orth = 10 * m if c["kS"] == c["kT"] else 8 * m * m
        basis = n * (8 * m * row + orth)
        if c["kind"].startswith("grad"):
            nodes = 6
            per = c["steps"] * (2 * basis + n * 8 * m * (2 * nodes + 2) + n * 8 * nodes * (4 + 4 * nn))
            byts += c["fields"] * 8 * (15 + 9 * nn)
        else:
            builds = max(1.0, c["steps"] * c["dt_ns"] / (0.9 * m * (1 if c["mode"] == "general" else 2)))
            per = builds * (basis + n * 4 * m * m + n * 8 * m) + c["steps"] * 40 * m * m
            byts += c["fields"] * 32 * T
        flops += per * M * c["fields"]
        byts += 16 * Z * M * c["fields"]
    return {"bytes": byts, "flops": flops}


def draw(rng):
    """Cases between and around the listed ones: nuclei of each kind, samples, Krylov dimension, window, rates, method."""
    top = max(work(c)["flops"] for c in listed())

    def pair(zmax):
        nuc = []
        while True:
            g = rng.choice((2, 2, 3))
            if math.prod(nuc) * g > zmax:
                break
            nuc.append(g)
        rng.shuffle(nuc)
        k = rng.randint(0, len(nuc))
        return ",".join(map(str, nuc[:k])) + "|" + ",".join(map(str, nuc[k:]))

    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    while True:
        kind = rng.choice(("trace", "torch", "torch", "batch", "grad", "gradbatch"))
        c = _case("", kind, "", "", rng.randint(8, 32), 0, mode=rng.choice(("general", "general", "reference")),
                  method=rng.choice(("auto", "mgs")), kT=rng.choice((1.0, 1.0, 0.3)), state=rng.choice(STATES[:2]))
        del c["name"]
        if kind in ("trace", "torch"):
            c["systems"], c["samples"], c["steps"] = pair(log(12, 13824)), str(log(4, 512)), log(40, 400)
        elif kind == "batch":
            k = rng.randint(1, 8)
            c["systems"] = ";".join(pair(log(4, 2304)) for _ in range(k))
            c["samples"] = ";".join(str(log(16, 256)) for _ in range(k))
            c["steps"], c["fields"] = log(20, 120), rng.randint(1, 6)
        else:
            c["mode"], c["steps"] = "general", rng.randint(4, 16)
            if kind == "grad":  # yields of the singlet-born pair
                c["state"] = "singlet"
                c["systems"], c["samples"] = pair(log(12, 3456)), str(log(8, 96))
            else:
                k = rng.randint(1, 5)
                c["systems"] = ";".join(rng.choice(BLOCKS.split(";")) for _ in range(k))
                c["samples"], c["fields"] = str(log(8, 64)), rng.randint(1, 3)
            c["m"] = max(12, c["m"])
        if c["method"] == "auto" and kind == "grad" and c["kT"] == c["kS"]:
            c["method"] = "lanczos"
        if work(c)["flops"] <= 0.5 * top:
            return c


_SAMPLER = []


def _sampler():
    """One handle for the whole program, as a program keeps one."""
    if not _SAMPLER:
        _SAMPLER.append(TraceSampler(0))
    return _SAMPLER[0]


def _values(case, seed):
    """The physical values of a case: per system (nuclei of both radicals, tensors, gyromagnetic ratios), the fields,
    and the sample vectors of every job (pair-major), normalised: random phases or Gaussian amplitudes."""
    c = case
    rng = np.random.default_rng(seed)
    iso = c["mode"] == "reference"
    systems = []
    for s in c["systems"].split(";"):
        side = []
        for part in s.split("|"):
            g = [int(x) for x in part.split(",") if x]
            A = []
            for _ in g:
                if iso:
                    A.append(np.eye(3) * rng.uniform(0.1, 1.5))
                else:
                    q, r = np.linalg.qr(rng.normal(size=(3, 3)))
                    q = q * np.sign(np.diag(r))
                    A.append(q @ np.diag(rng.uniform(-2.0, 2.0, 3)) @ q.T)
            side.append((g, A, [GAMMA_14N if x == 3 else GAMMA_1H for x in g]))
        systems.append(side)
    if iso:
        fields = [0.05] if c["fields"] == 1 else list(np.linspace(0.0, 2.0, c["fields"]))
    else:
        d = rng.normal(size=(c["fields"], 3))
        fields = list(0.05 * d / np.linalg.norm(d, axis=1, keepdims=True))
    J, D = (0.0, np.zeros((3, 3))) if iso else (0.01, 2.0 / 3.0 * np.diag((-1.0, -1.0, 2.0)) * -0.4)
    dt = c["dt_ns"] * GAMMA_E / 1000.0
    return systems, fields, J, D, dt, dt * c["steps"]


def _vectors(case, seed):
    """Per job the M x Z sample vectors, a CUDA tensor for kind torch and NumPy arrays otherwise."""
    c = case
    if c["kind"] == "torch":
        g = torch.Generator(device="cuda").manual_seed(seed)
        Z, M = _dims(c)[0], _samples(c)[0]
        phi = torch.rand((M, Z), generator=g, device="cuda", dtype=torch.float64) * (2.0 * math.pi)
        return [torch.polar(torch.full_like(phi, 1.0 / math.sqrt(Z)), phi)]
    rng = np.random.default_rng(seed + 1)
    out = []
    for Z, M in zip(_dims(c), _samples(c)):
        for _ in range(c["fields"]):
            z = rng.normal(size=(M, Z)) + 1j * rng.normal(size=(M, Z))
            out.append(z / np.linalg.norm(z, axis=1, keepdims=True))
    return out


def prepare(case, seed):
    systems, fields, J, D, dt, t_end = _values(case, seed)
    sys_ = [SysParam(Electron(g_I=a[0], A=a[1], gamma_I=a[2]), Electron(g_I=b[0], A=b[1], gamma_I=b[2]), J=J, D=D,
                     kS=case["kS"] / GAMMA_E, kT=case["kT"] / GAMMA_E) for a, b in systems]
    st = dict(case=case, sampler=_sampler(), z=_vectors(case, seed), dt=dt, t_end=t_end,
              systems=[s for s in sys_ for _ in fields], fields=[f for _ in sys_ for f in fields])
    if case["kind"] == "grad":
        st["params"] = torch_ops.pack_params(sys_[0], fields[0])
    return st


def run(state):
    c, sp = state["case"], state["sampler"]
    sy, B, z, dt, t_end, m = state["systems"], state["fields"], state["z"], state["dt"], state["t_end"], c["m"]
    sp.set_krylov(c["method"])
    if c["kind"] in ("trace", "torch"):
        sp.build_h(sy[0], B[0], c["mode"])
        if c["kind"] == "torch":
            return torch_ops.trace_sampling(sp, z[0], dt, t_end, m, TOL, c["state"])
        sp.set_stream(0)
        return _rows(sp.trace_sampling(z[0], dt, t_end, m, TOL, c["state"]))
    sp.set_stream(0)
    if c["kind"] == "batch":
        sp.build_h_batch(sy, B, c["mode"])
        return np.stack([_rows(r) for r in sp.trace_sampling_batch(z, dt, t_end, m, TOL, c["state"])])
    if c["kind"] == "grad":
        p = state["params"].clone().requires_grad_()
        v = torch_ops.yield_objective(p, sp, sy[0], z[0], dt, t_end, m)
        v.backward()
        return {"yield": v.detach(), "gradient": p.grad}
    got = sp.yield_gradient_batch(sy, B, z, dt, t_end, m, hyperfine=False, init_state=c["state"])
    return {"yields": np.array([[g.Phi_S, g.Phi_T] for g in got]), "gradient": np.concatenate([g.raw[:15] for g in got])}


def _rows(o):
    return np.stack([o.P_S, o.P_T0, o.P_Tp, o.P_Tm])


# ----------------------------------------------------------------------------------------------------------------------
# The same outputs in plain torch, 64 bits: sparse products, Gram-Schmidt done twice, torch.linalg.matrix_exp, and the
# populations straight from the states.

def _spin(g):
    S = 0.5 * (g - 1)
    up = np.diag([math.sqrt(S * (S + 1) - (S - i) * (S - i + 1)) for i in range(1, g)], 1)
    return 0.5 * (up + up.T), -0.5j * (up - up.T), np.diag([S - i for i in range(g)]).astype(float)


_S1 = [np.kron(a, np.eye(2)) for a in _spin(2)]
_S2 = [np.kron(np.eye(2), a) for a in _spin(2)]
_DOT = sum(a @ b for a, b in zip(_S1, _S2))
_PS = 0.25 * np.eye(4) - _DOT


def _nuclei(system, iso):
    """(owner, multiplicity, stride, tensor, gamma ratio) of every nucleus, radical 1's first, row-major."""
    out = [(o, g, A, gam / GAMMA_E) for o, (gs, As, gams) in enumerate(system) for g, A, gam in zip(gs, As, gams)]
    Z = math.prod(x[1] for x in out)
    res, left = [], 1
    for o, g, A, gr in out:
        left *= g
        res.append((o, g, Z // left, np.eye(3) * np.trace(A) / 3.0 if iso else A, gr))
    return res, Z


def _hamiltonian(system, field, J, D, kS, kT, iso, dev):
    B = np.array([0.0, 0.0, field]) if iso else np.asarray(field)
    nuc, Z = _nuclei(system, iso)
    el = -sum(B[a] * (_S1[a] + _S2[a]) for a in range(3)) + 2.0 * J * _DOT
    el = el + sum(D[a, b] * _S1[a] @ _S2[b] for a in range(3) for b in range(3))
    el = el - 0.5j * (kS * _PS + kT * (np.eye(4) - _PS))
    n = torch.arange(Z, device=dev)
    rows, cols, vals = [], [], []

    def add(op, g, stride):  # op on (electron pair, nucleus): (e, m) <- (e', m')
        for r, c in zip(*np.nonzero(op)):
            (e, a), (f, b) = divmod(int(r), g), divmod(int(c), g)
            k = n[(n // stride) % g == a]
            rows.append(e * Z + k)
            cols.append(f * Z + k + (b - a) * stride)
            vals.append(torch.full((k.numel(),), complex(op[r, c]), dtype=torch.complex128, device=dev))

    add(el, 1, 1)
    for o, g, stride, A, gr in nuc:
        I, S = _spin(g), (_S1, _S2)[o]
        op = sum(np.kron(np.eye(4), gr * B[b] * I[b]) for b in range(3))
        add(op + sum(A[a, b] * np.kron(S[a], I[b]) for a in range(3) for b in range(3)), g, stride)
    H = torch.sparse_coo_tensor(torch.stack([torch.cat(rows), torch.cat(cols)]), torch.cat(vals), (4 * Z, 4 * Z))
    return H.coalesce().to_sparse_csr()


def _theta(state):
    h = math.sqrt(0.5)
    th = {"singlet": (0, h, -h, 0), "T0": (0, h, h, 0), "Tp": (1, 0, 0, 0), "Tm": (0, 0, 0, 1)}[state]
    return th, {"singlet": (1, 0, 0, 0), "T0": (0, 1, 0, 0), "Tp": (0, 0, 1, 0), "Tm": (0, 0, 0, 1)}[state]


def _pops(psi):
    """(samples, n) -> (samples, 4): singlet, T0, T+, T-."""
    p = psi.reshape(psi.shape[0], 4, -1)
    f = (p[:, 1] - p[:, 2], p[:, 1] + p[:, 2], p[:, 0], p[:, 3])
    return torch.stack([w * x.abs().square().sum(-1) for w, x in zip((0.5, 0.5, 1.0, 1.0), f)], 1)


def _trace(H, z, theta, pop0, dt, t_end, T, m, dev):
    """Populations summed over the samples, (4, T)."""
    M, n = z.shape[0], H.shape[0]
    m = min(m, n)
    psi = torch.cat([t * z for t in theta], 1)
    N, t = 0, 0.0
    while t < t_end:
        N, t = N + 1, t + dt
    out = torch.zeros((M, 4, T), dtype=torch.float64, device=dev)
    out[:, :, 0] = torch.tensor(pop0, dtype=torch.float64, device=dev)
    k = torch.zeros(M, dtype=torch.int64, device=dev)
    while True:
        live = torch.nonzero(k < N).flatten()
        if not live.numel():
            return out.sum(0)
        x = psi[live]
        L = live.numel()
        A = torch.zeros((L, m, m), dtype=torch.complex128, device=dev)
        Q = torch.zeros((L, m, n), dtype=torch.complex128, device=dev)
        b = torch.linalg.vector_norm(x, dim=1)
        Q[:, 0] = x / b[:, None]
        for i in range(m):
            p = (H @ Q[:, i].t().contiguous()).t().contiguous()
            for _ in range(2):
                h = torch.bmm(Q[:, :i + 1], p.conj().resolve_conj()[:, :, None]).conj()
                p = p - torch.bmm(h.resolve_conj().transpose(1, 2), Q[:, :i + 1])[:, 0]
                A[:, :i + 1, i] += h[:, :, 0]
            if i + 1 < m:
                w = torch.linalg.vector_norm(p, dim=1)
                A[:, i + 1, i] = w
                Q[:, i + 1] = p * torch.where(w > 0, 1.0 / w, 0.0)[:, None]
        E = torch.linalg.matrix_exp(-1j * dt * A)
        c = torch.zeros((L, m), dtype=torch.complex128, device=dev)
        c[:, 0] = b.to(c.dtype)
        on = torch.ones(L, dtype=torch.bool, device=dev)
        kk = k[live]
        while bool(on.any()):
            new = torch.bmm(E, c[:, :, None])[:, :, 0]
            c = torch.where(on[:, None], new, c)
            kk = kk + on
            s = torch.nonzero(on).flatten()
            out[live[s], :, kk[s]] = _pops(torch.bmm(c[:, None, :], Q)[:, 0])[s]
            on = on & (c[:, -1].abs().square() <= TOL * c.abs().square().sum(1)) & (kk < N)
        psi[live] = torch.bmm(c[:, None, :], Q)[:, 0]
        k[live] = kk


def _evolve(H, x, tau):
    """exp(-i tau H) x by Taylor steps; x (n, samples)."""
    bound = float(torch.zeros(H.shape[0], dtype=torch.float64, device=x.device).index_add_(
        0, H.col_indices(), H.values().abs()).max())
    s = max(1, math.ceil(abs(tau) * bound))
    for _ in range(s):
        term, acc = x, x.clone()
        for k in range(1, 23):
            term = (H @ term) * (-1j * tau / s / k)
            acc += term
        x = acc
    return x


def _gradient(system, field, J, D, kS, kT, z, theta, dt, T, dev):
    """Phi_S, Phi_T and d Phi_S / d (B, J, D, kS, kT, tensors) of the sample mean."""
    nuc, Z = _nuclei(system, False)
    M = z.shape[0]
    H = _hamiltonian(system, field, J, D, kS, kT, False, dev)
    Ha = _hamiltonian(system, field, J, D, -kS, -kT, False, dev)  # the adjoint
    psi = [torch.cat([t * z for t in theta], 1).t().contiguous()]
    N = 2 * (T // 2) - 2
    for _ in range(N):
        psi.append(_evolve(H, psi[-1], dt))
    w = [dt / 3.0 * (1.0 if k in (0, N) else 4.0 if k % 2 else 2.0) for k in range(N + 1)]
    ps = sum(a * float(_pops(x.t())[:, 0].sum()) for a, x in zip(w, psi)) / M
    pt = sum(a * float(_pops(x.t())[:, 1:].sum()) for a, x in zip(w, psi)) / M
    P = torch.tensor(_PS, dtype=torch.complex128, device=dev)

    def source(x):
        return kS * torch.einsum("ab,bzm->azm", P, x.reshape(4, Z, M)).reshape(4 * Z, M)

    R = torch.zeros((4, 4), dtype=torch.complex128, device=dev)
    Rn = [torch.zeros((4, g, 4, g), dtype=torch.complex128, device=dev) for _, g, _, _, _ in nuc]
    xs, ws = np.polynomial.legendre.leggauss(10)
    lam = w[N] * source(psi[N])
    for k in range(N - 1, -1, -1):
        mu, nu, at = lam, psi[k], 0.0
        for x, q in zip(0.5 * (xs + 1.0), 0.5 * ws):
            nu = _evolve(H, nu, dt * (x - at))
            mu = _evolve(Ha, lam, -dt * (1.0 - x))
            at = x
            a, b = mu.conj().resolve_conj(), nu
            R += q * dt * torch.einsum("azm,bzm->ab", a.reshape(4, Z, M), b.reshape(4, Z, M))
            for j, (_, g, stride, _, _) in enumerate(nuc):
                u, v = (y.reshape(4, Z // (g * stride), g, stride * M).permute(0, 2, 1, 3).reshape(4 * g, -1) for y in (a, b))
                Rn[j] += q * dt * (u @ v.t()).reshape(4, g, 4, g)
        lam = w[k] * source(psi[k]) + _evolve(Ha, lam, -dt)
    d = lambda op, r: 2.0 / M * float((torch.tensor(op, dtype=torch.complex128, device=dev) * r.reshape(op.shape)).sum().imag)  # noqa: E731
    gB = np.array([d(-(_S1[a] + _S2[a]), R) for a in range(3)])
    gA = []
    for (o, g, _, _, gr), r in zip(nuc, Rn):
        I, S = _spin(g), (_S1, _S2)[o]
        gB += np.array([gr * d(np.kron(np.eye(4), I[b]), r) for b in range(3)])
        gA += [d(np.kron(S[a], I[b]), r) for b in range(3) for a in range(3)]
    rest = [d(2.0 * _DOT, R)] + [d(_S1[a] @ _S2[b], R) for b in range(3) for a in range(3)]
    rest += [d(-0.5j * _PS, R) + ps, d(-0.5j * (np.eye(4) - _PS), R)]
    return kS * ps, kT * pt, np.array(list(gB) + rest + gA)


def exact(case, seed):
    c = case
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if work(c)["flops"] > (4e13 if dev == "cuda" else 1e11):
        return None
    systems, fields, J, D, dt, t_end = _values(c, seed)
    kS, kT, iso = c["kS"] / GAMMA_E, c["kT"] / GAMMA_E, c["mode"] == "reference"
    theta, pop0 = _theta(c["state"])
    T = math.ceil((t_end + dt) / dt) + 1
    z = [torch.as_tensor(v, device=dev) for v in _vectors(c, seed)]
    jobs = [(s, f) for s in systems for f in fields]
    if c["kind"].startswith("grad"):
        got = [_gradient(s, f, J, D, kS, kT, v, theta, dt, T, dev) for (s, f), v in zip(jobs, z)]
        if c["kind"] == "grad":
            return {"yield": torch.tensor(got[0][0], dtype=torch.float64), "gradient": torch.from_numpy(got[0][2])}
        return {"yields": np.array([g[:2] for g in got]), "gradient": np.concatenate([g[2][:15] for g in got])}
    res = []
    for (s, f), v in zip(jobs, z):
        H = _hamiltonian(s, f, J, D, kS, kT, iso, dev)
        total = sum(_trace(H, part, theta, pop0, dt, t_end, T, c["m"], dev) for part in v.split(64))
        res.append(total / v.shape[0])
    if c["kind"] == "torch":
        return res[0]
    return np.stack([r.cpu().numpy() for r in res]) if c["kind"] == "batch" else res[0].cpu().numpy()
