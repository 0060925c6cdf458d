"""The timed work of this framework: time evolution as its users call it.

Each case is one whole call (or one layer of it) through the public entry points:

* ``mesolve``: a master equation integrated over ``tlist`` with expectation values and the
  final state (``solver.solve_system`` with the operator a user's program keeps);
* ``apply``: one application of a Liouvillian to a density matrix (``DeviceOperator.matvec``);
* ``mcsolve``: Monte-Carlo trajectories of one system (``batched.mcsolve_batch``);
* ``served``: many small master equations of mixed sizes in one call (``batched.mesolve_batch``);
* ``sde``: fixed-step stochastic trajectories (``stochastic.SdeOperator.advance``).

The mixed form integrates complex64 stages; where its result is a state or a trajectory of
a single system, the caller here keeps it in complex64.
"""
import math

import numpy as np
import torch

from qutip_gb300 import systems
from qutip_gb300.batched import mcsolve_batch, mesolve_batch
from qutip_gb300.coefficients import coefficient
from qutip_gb300.dense import DenseLindbladOperator
from qutip_gb300.lindblad import LindbladOperator
from qutip_gb300.operator import DeviceOperator
from qutip_gb300.solver import ExpectOps, solve_system
from qutip_gb300.stochastic import SdeOperator
from qutip_gb300.superop import liouvillian_groups, sliced_padding

DEVICE = "cuda"
OMEGA = 1.3          # drive frequency of the Ising chain
RATE = {"jc": 17.0, "ising": 13.0, "bh": 30.0, "dense": 60.0}   # right-hand sides per unit time (about)


# ------------------------------------------------------------------ cases ----
def listed():
    return [
        # one small master equation: the driven Jaynes-Cummings system of the first
        # configuration, 400 rows; latency and launches are what it costs
        {"name": "jc10_double", "kind": "mesolve", "system": "jc", "size": 10, "form": "superop",
         "precision": "double", "t": 20.0, "outputs": 201},
        # an ordinary time-dependent spin chain, 65,536 rows
        {"name": "ising8_double", "kind": "mesolve", "system": "ising", "size": 8,
         "form": "superop", "precision": "double", "t": 10.0, "outputs": 101},
        # the headline: the ten-spin chain, 1,048,576 rows and 24.6 million entries
        {"name": "ising10_double", "kind": "mesolve", "system": "ising", "size": 10,
         "form": "superop", "precision": "double", "t": 10.0, "outputs": 101},
        # the same with complex64 stages
        {"name": "ising10_mixed", "kind": "mesolve", "system": "ising", "size": 10,
         "form": "superop", "precision": "mixed", "t": 10.0, "outputs": 101},
        # an odd dimension (125, 15,625 rows) with many distinct matrix elements
        {"name": "bh5_double", "kind": "mesolve", "system": "bh", "size": 5, "form": "superop",
         "precision": "double", "t": 5.0, "outputs": 51},
        # the matrix form: the generator without its superoperator
        {"name": "ising10_matrix_mixed", "kind": "mesolve", "system": "ising", "size": 10,
         "form": "matrix", "precision": "mixed", "t": 10.0, "outputs": 101},
        # a small system with dense operators, on the tensor cores
        {"name": "dense128_mixed", "kind": "mesolve", "system": "dense", "size": 128,
         "form": "dense", "precision": "mixed", "t": 2.0, "outputs": 21},
        # one right-hand side: the sparse Liouvillian matvec alone, 262,144 rows
        {"name": "apply_ising9_c64", "kind": "apply", "system": "ising", "size": 9, "dtype": "c64"},
        # trajectories of the Bose-Hubbard trimer (512 states), two per resident CTA
        {"name": "mc_bh8_mixed", "kind": "mcsolve", "system": "bh", "size": 8, "ntraj": 608,
         "precision": "mixed", "group": "cta", "t": 10.0, "outputs": 101},
        # a batch of requests of mixed sizes, as the server packs them
        {"name": "served_jc_mixed", "kind": "served", "jobs": 96, "size": 30,
         "precision": "mixed", "t": 20.0, "outputs": 101},
        # a stochastic master equation of a driven cavity, a batch of trajectories
        {"name": "sme20", "kind": "sde", "open": True, "size": 20, "ntraj": 256, "steps": 100,
         "scheme": "platen"},
        # the stochastic Schroedinger equation: short kets, many of them
        {"name": "sse40", "kind": "sde", "open": False, "size": 40, "ntraj": 1000, "steps": 100,
         "scheme": "platen"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mesolve", "mesolve", "mesolve", "apply", "mcsolve", "served", "sde"])
    if kind == "mesolve":
        system = rng.choice(["jc", "ising", "bh", "dense"])
        form = rng.choice(["superop", "superop", "matrix"]) if system != "dense" else "dense"
        size = {"jc": _log(rng, 5, 60), "ising": rng.randint(4, 10), "bh": rng.randint(3, 6),
                "dense": _log(rng, 9, 128)}[system]
        precision = rng.choice(["double", "mixed"])
        if form == "dense":
            precision = "mixed"
        t = round(rng.uniform(1.0, {"jc": 20.0, "ising": 8.0, "bh": 5.0, "dense": 2.0}[system]), 2)
        if system == "ising" and form == "matrix" and precision == "double":
            size = min(size, 9)
        return {"kind": kind, "system": system, "size": size, "form": form,
                "precision": precision, "t": t, "outputs": rng.randint(5, 101)}
    if kind == "apply":
        system = rng.choice(["ising", "bh", "jc"])
        size = {"jc": _log(rng, 5, 60), "ising": rng.randint(4, 10), "bh": rng.randint(3, 7)}[system]
        return {"kind": kind, "system": system, "size": size, "dtype": rng.choice(["c64", "c128"])}
    if kind == "mcsolve":
        system = rng.choice(["bh", "jc"])
        return {"kind": kind, "system": system,
                "size": rng.randint(3, 8) if system == "bh" else _log(rng, 5, 60),
                "ntraj": _log(rng, 16, 608), "precision": rng.choice(["double", "mixed"]),
                "group": rng.choice(["auto", "cta", "cta128"]),
                "t": round(rng.uniform(2.0, 8.0), 2), "outputs": rng.randint(5, 81)}
    if kind == "served":
        return {"kind": kind, "jobs": _log(rng, 4, 160), "size": _log(rng, 8, 40),
                "precision": rng.choice(["double", "mixed"]), "t": round(rng.uniform(2.0, 20.0), 2),
                "outputs": rng.randint(5, 101)}
    is_open = rng.random() < 0.5
    return {"kind": "sde", "open": is_open, "size": _log(rng, 4, 24) if is_open else _log(rng, 5, 200),
            "ntraj": _log(rng, 1, 512), "steps": rng.randint(10, 100),
            "scheme": rng.choice(["platen", "platen", "euler"])}


# ---------------------------------------------------------------- systems ----
def _system(case, rng, kind="me"):
    """A system of the named family with parameters drawn from ``rng``."""
    size = case["size"]
    if case["system"] == "jc":
        return systems.jaynes_cummings(size, g=float(rng.uniform(0.01, 0.1) * 2 * np.pi),
                                       kappa=float(10 ** rng.uniform(-3, -1)),
                                       gamma=float(10 ** rng.uniform(-3, -1)), kind=kind)
    if case["system"] == "ising":
        return systems.ising_chain(size, h=rng.uniform(0.5, 1.5, size), omega=OMEGA, kind=kind,
                                   build_terms=size <= 4)
    if case["system"] == "bh":
        return systems.bose_hubbard_trimer(size, U=float(rng.uniform(0.3, 0.7)),
                                           F=float(rng.uniform(0.2, 0.4)),
                                           kappa=float(rng.uniform(0.05, 0.2)), kind=kind)
    d = size

    def mat(herm=False):
        m = rng.normal(size=(d, d)) + 1j * rng.normal(size=(d, d))
        return (m + m.conj().T) / 2 if herm else m
    h_terms = [(mat(True) / np.sqrt(d), None),
               (0.3 * mat(True) / np.sqrt(d), coefficient("cos(w*t)", args={"w": OMEGA}))]
    c_ops = [0.1 * mat() / np.sqrt(d), 0.05 * mat() / np.sqrt(d)]
    psi = rng.normal(size=d) + 1j * rng.normal(size=d)
    psi /= np.linalg.norm(psi)
    return systems.OpenSystem("dense", "me", d, None, np.outer(psi, psi.conj()).reshape(-1, order="F"),
                              [mat(True)], c_ops, h_terms)


def _snap(v):
    """Values on a grid of 2^-50 of the largest: the device sums equal matrix elements in
    varying order, and a Liouvillian summed on the host has equal elements with equal bits."""
    parts = torch.view_as_real(v)
    step = 2.0 ** (math.ceil(math.log2(max(float(parts.abs().max()), 1e-300))) - 50)
    return torch.view_as_complex((parts / step).round() * step)


def _superoperator(s, dtype):
    """The device Liouvillian, laid out on the device from 1024 rows up."""
    if s.dim * s.dim >= 1024:
        groups = [(ip, ix, _snap(v), c)
                  for ip, ix, v, c in liouvillian_groups(s.h_terms, s.c_ops, DEVICE)]
        if sliced_padding(groups) <= 1.15:
            return DeviceOperator.from_device_groups(groups, dtype)
        del groups
    terms = s.terms if s.terms is not None else systems._me_terms(s.h_terms, s.c_ops)
    return DeviceOperator(terms, dtype=dtype)


def _sde(case, rng):
    """H, measured operator, and for an open system a deterministic collapse operator."""
    n = case["size"]
    a = systems.destroy(n)
    num = a.conj().T @ a
    h = num + float(rng.uniform(0.3, 0.6)) * (a + a.conj().T)
    return h, np.sqrt(float(rng.uniform(0.1, 0.3))) * a, np.sqrt(0.1) * num


# ---------------------------------------------------------------- prepare ----
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "mesolve":
        s = _system(case, rng)
        dtype = "c128" if case["precision"] == "double" else "c64"
        if case["form"] == "dense":
            op = DenseLindbladOperator.from_hamiltonian(s.h_terms, s.c_ops)
        elif case["form"] == "matrix":
            op = LindbladOperator.from_hamiltonian(s.h_terms, s.c_ops, dtype=dtype)
        else:
            op = _superoperator(s, dtype)
        st.update(system=s, op=op, ex=ExpectOps(s.e_ops),
                  tlist=np.linspace(0.0, case["t"], case["outputs"]))
    elif kind == "apply":
        s = _system(case, rng)
        op = _superoperator(s, case["dtype"])
        dt = torch.complex64 if case["dtype"] == "c64" else torch.complex128
        m = torch.from_numpy(rng.normal(size=(2, op.n_rows))).to(DEVICE)
        st.update(op=op, x=torch.complex(m[0], m[1]).to(dt), y=torch.zeros(op.n_rows, dtype=dt,
                                                                            device=DEVICE))
    elif kind == "mcsolve":
        st.update(system=_system(case, rng, "mc"),
                  seeds=np.random.SeedSequence(int(rng.integers(2 ** 62))).spawn(case["ntraj"]),
                  tlist=np.linspace(0.0, case["t"], case["outputs"]))
    elif kind == "served":
        sizes = rng.integers(5, case["size"] + 1, case["jobs"])
        sizes[0] = case["size"]
        st.update(systems=[_system({"system": "jc", "size": int(n)}, rng) for n in sizes],
                  tlist=np.linspace(0.0, case["t"], case["outputs"]))
    else:
        h, sc, c = _sde(case, rng)
        n = case["size"]
        if case["open"]:
            L = systems.liouvillian(h, [sc, c])
            op = SdeOperator(L, [systems.spre(sc) + systems.spost(sc.conj().T)], open=True, d=n)
        else:
            op = SdeOperator.sse(h, [sc])
        psi = rng.normal(size=(case["ntraj"], n)) + 1j * rng.normal(size=(case["ntraj"], n))
        psi *= np.exp(-0.5 * np.arange(n))[None, :]
        psi /= np.linalg.norm(psi, axis=1, keepdims=True)
        if case["open"]:   # column-stacked |psi><psi|
            x0 = (psi.conj()[:, :, None] * psi[:, None, :]).reshape(case["ntraj"], -1)
        else:
            x0 = psi
        dt = 1e-3
        dW = rng.normal(size=(case["ntraj"], case["steps"], 1)) * np.sqrt(dt)
        st.update(op=op, x0=torch.from_numpy(x0).to(DEVICE), dW=torch.from_numpy(dW).to(DEVICE),
                  dt=dt)
    return st


# -------------------------------------------------------------------- run ----
def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "mesolve":
        r = solve_system(state["system"], state["tlist"],
                         {"precision": case["precision"], "store_final_state": True},
                         op=state["op"], ex=state["ex"])
        out = {"expect": np.stack(r.expect), "final_state": r.final_state}
        if case["precision"] == "mixed":
            out = {k: v.astype(np.complex64) for k, v in out.items()}
        return out
    if kind == "apply":
        return state["op"].matvec(0.37, state["x"], state["y"])
    if kind == "mcsolve":
        r = mcsolve_batch(state["system"], state["tlist"], case["ntraj"], seeds=state["seeds"],
                          precision=case["precision"], group=case["group"])
        times, which = (np.zeros((case["ntraj"], 512), t) for t in (np.float64, np.int64))
        for i, (t, w) in enumerate(zip(r.col_times, r.col_which)):
            times[i, :len(t)], which[i, :len(w)] = t, w
        return {"runs_expect": r.runs_expect, "col_times": times, "col_which": which}
    if kind == "served":
        return np.stack([np.stack(e) for e in mesolve_batch(state["systems"], state["tlist"],
                                                            precision=case["precision"])[0]])
    x = state["x0"].clone()
    state["op"].advance(x, state["dW"], case["steps"], state["dt"], scheme=case["scheme"])
    return x


# ------------------------------------------------------------------- work ----
def _dim(case):
    size = case["size"]
    return {"jc": 2 * size, "ising": 2 ** size, "bh": size ** 3, "dense": size}[case["system"]]


def _entries(case):
    """Stored entries of the superoperator per row of vec(rho) (about)."""
    size = case["size"]
    return {"jc": 4.0, "ising": 2.25 * size + 1, "bh": 13.0, "dense": 0.0}[case["system"]]


def work(case):
    kind = case["kind"]
    if kind == "mesolve":
        d = _dim(case)
        es = 16 if case["precision"] == "double" else 8
        rate = RATE[case["system"]] * (case["size"] if case["system"] in ("jc", "ising") else 1)
        if case["system"] == "jc":
            rate = RATE["jc"]
        rhs = max(17.0, rate * case["t"])
        if case["form"] == "dense":
            flops = rhs * 8.0 * d ** 3 * 6
        else:
            flops = rhs * d * d * (8.0 * _entries(case) + 20.0)
        return {"bytes": rhs * d * d * es * 2.0, "flops": flops}
    if kind == "apply":
        d = _dim(case)
        es = 8 if case["dtype"] == "c64" else 16
        return {"bytes": 2.0 * d * d * es, "flops": 8.0 * d * d * _entries(case)}
    if kind == "mcsolve":
        d = _dim(case)
        rhs = case["ntraj"] * RATE[case["system"]] * case["t"]
        return {"bytes": case["ntraj"] * case["outputs"] * 64.0, "flops": rhs * d * (8.0 * 9 + 20)}
    if kind == "served":
        n = case["jobs"] * (2.0 * case["size"]) ** 2 / 3.0
        return {"bytes": case["jobs"] * case["outputs"] * 48.0,
                "flops": RATE["jc"] * case["t"] * n * (8.0 * 4 + 20)}
    n = case["size"] ** 2 if case["open"] else case["size"]
    applications = 5 if case["scheme"] == "platen" else 2
    per = n * (8.0 * (7 if case["open"] else 3) * applications + 60)
    return {"bytes": case["ntraj"] * (2.0 * 16 * n + 8.0 * case["steps"]),
            "flops": case["ntraj"] * case["steps"] * per}


# ------------------------------------------------------------------ exact ----
def _dense(m):
    return np.asarray(m.toarray() if hasattr(m, "toarray") else m, dtype=np.complex128)


def _generator(s):
    """L(t)[rho] of a Hermitian rho (d x d tensor) in complex128 torch."""
    d = s.dim

    def up(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)

    def sparse(a):
        a = a.tocsr() if hasattr(a, "tocsr") else None
        return None if a is None or a.nnz > d * d // 8 else torch.sparse_csr_tensor(
            up(a.indptr.astype(np.int64)), up(a.indices.astype(np.int64)),
            up(a.data.astype(np.complex128)), size=(d, d))

    const, driven = None, None
    for h, c in s.h_terms:
        if c is None:
            const = -1j * h if const is None else const - 1j * h
        else:
            driven = -1j * h
    for c in s.c_ops:
        const = const - 0.5 * (c.conj().T @ c)
    parts = []
    for m in (const, driven):
        if m is not None:
            sm = sparse(m)
            parts.append(sm if sm is not None else up(_dense(m)))
        else:
            parts.append(None)
    factor, moved, full = torch.zeros((d, d), dtype=torch.complex128, device=DEVICE), [], []
    for c in s.c_ops:
        a = c.tocoo() if hasattr(c, "tocoo") else None
        if a is None or np.bincount(a.row, minlength=d).max() > 1:
            full.append(up(_dense(c)))
            continue
        col, val = np.arange(d), np.zeros(d, dtype=np.complex128)
        col[a.row], val[a.row] = a.col, a.data
        w = up(val)
        w = w[:, None] * w.conj()[None, :]
        if np.array_equal(col, np.arange(d)):
            factor += w
        else:
            moved.append((up(col.astype(np.int64)), w))

    def rhs(t, rho):
        b = parts[0] @ rho
        if parts[1] is not None:
            b = b + math.cos(OMEGA * t) * (parts[1] @ rho)
        out = b + b.conj().T + factor * rho
        for idx, w in moved:
            out += w * rho[idx][:, idx]
        for c in full:
            out += c @ rho @ c.conj().T
        return out
    return rhs


def _evolve(rhs, rho, t0, t1, h_max):
    """Modified midpoint steps extrapolated over six subdivisions (Gragg, Bulirsch, Stoer)."""
    steps = max(1, math.ceil((t1 - t0) / h_max))
    h = (t1 - t0) / steps
    subs = (2, 4, 6, 8, 10, 12, 14)
    for k in range(steps):
        t = t0 + k * h
        f0 = rhs(t, rho)
        row = []
        for i, n in enumerate(subs):
            g = h / n
            a, b = rho, rho + g * f0
            for j in range(1, n):
                a, b = b, a + (2 * g) * rhs(t + j * g, b)
            new = [0.5 * (a + b + g * rhs(t + h, b))]
            for j in range(i):
                new.append(new[j] + (new[j] - row[j]) / ((n / subs[i - 1 - j]) ** 2 - 1))
            row = new
        rho = row[-1]
    return rho


def _exact_me(s, tlist, scale):
    rhs = _generator(s)
    d = s.dim
    rho = torch.from_numpy(s.state0.reshape(d, d, order="F").copy()).to(DEVICE)
    e_ops = [torch.from_numpy(_dense(e)).to(DEVICE) for e in s.e_ops]
    tr = [torch.stack([(e.T * rho).sum() for e in e_ops])]
    for t0, t1 in zip(tlist[:-1], tlist[1:]):
        rho = _evolve(rhs, rho, float(t0), float(t1), 4.0 / scale)
        rho = 0.5 * (rho + rho.conj().T)
        tr.append(torch.stack([(e.T * rho).sum() for e in e_ops]))
    return torch.stack(tr, dim=1).cpu().numpy(), rho.T.reshape(-1).cpu().numpy()


def _scale(s):
    """About the largest rate of the generator."""
    total = 0.0
    for h, _ in s.h_terms:
        a = abs(_dense(h))
        dg = np.real(np.diag(_dense(h)))
        off = a.sum(axis=1) - np.diag(a)
        total += (dg.max() - dg.min()) + 2 * off.max() if s.name != "dense" else 4.0
    return total + 1.0


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "mesolve":
        s = _system(case, rng)
        scale = _scale(s)
        outputs = case["outputs"]
        # about 60 generator calls per extrapolated step of length 4 / scale
        calls = 60 * max(outputs - 1, scale * case["t"] / 4.0)
        per = 1.5e-4 + 2e-8 * _dim(case) ** 2 / 8 * (1 + len(s.c_ops) / 4)
        if calls * per > 18.0:
            return None
        expect, final = _exact_me(s, np.linspace(0.0, case["t"], outputs), scale)
        return {"expect": expect, "final_state": final}
    if kind == "apply":
        s = _system(case, rng)
        m = torch.from_numpy(rng.normal(size=(2, s.dim * s.dim))).to(DEVICE)
        x = torch.complex(m[0], m[1])
        if case["dtype"] == "c64":
            x = x.to(torch.complex64).to(torch.complex128)
        x = x.reshape(s.dim, s.dim).T
        # any matrix is H1 + i H2 with Hermitian H1, H2, and the generator is linear
        rhs = _generator(s)
        h1, h2 = 0.5 * (x + x.conj().T), -0.5j * (x - x.conj().T)
        out = rhs(0.37, h1) + 1j * rhs(0.37, h2)
        return out.T.reshape(-1)
    if kind == "sde":
        return _exact_sde(case, rng)
    if kind == "served":
        sizes = rng.integers(5, case["size"] + 1, case["jobs"])
        sizes[0] = case["size"]
        tl = np.linspace(0.0, case["t"], case["outputs"])
        out, spent = [], 0.0
        for n in sizes:
            s = _system({"system": "jc", "size": int(n)}, rng)
            spent += 60 * max(case["outputs"] - 1, _scale(s) * case["t"] / 4.0) * 1.5e-4
            if spent > 18.0:
                return None
            out.append(_exact_me(s, tl, _scale(s))[0])
        return np.stack(out)
    return None


def _exact_sde(case, rng):
    h, sc, c = (_dense(m) for m in _sde(case, rng))
    n = case["size"]
    ntraj, steps, dt = case["ntraj"], case["steps"], 1e-3
    psi = rng.normal(size=(ntraj, n)) + 1j * rng.normal(size=(ntraj, n))
    psi *= np.exp(-0.5 * np.arange(n))[None, :]
    psi /= np.linalg.norm(psi, axis=1, keepdims=True)
    dW = torch.from_numpy(rng.normal(size=(ntraj, steps, 1)) * np.sqrt(dt)).to(DEVICE)

    def up(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)
    if case["open"]:
        x = up(psi[:, :, None] * psi.conj()[:, None, :])     # rho[r, c]
        a = up(-1j * h - 0.5 * (sc.conj().T @ sc + c.conj().T @ c))
        s, c = up(sc), up(c)

        def drift(v):
            b = a @ v
            return b + v @ a.conj().T + s @ v @ s.conj().T + c @ v @ c.conj().T

        def diffusion(v):
            b = s @ v + v @ s.conj().T
            return b - torch.einsum("bii->b", b)[:, None, None] * v
        shape = (ntraj, 1, 1)
    else:
        x = up(psi)
        a, s, m = up((-1j * h - 0.5 * sc.conj().T @ sc).T), up(sc.T), up((sc + sc.conj().T).T)

        def mean(v):
            return (v.conj() * (v @ m)).sum(dim=1, keepdim=True)

        def drift(v):
            e = mean(v)
            return v @ a - 0.125 * e * e * v + 0.5 * e * (v @ s)

        def diffusion(v):
            return v @ s - 0.5 * mean(v) * v
        shape = (ntraj, 1)
    root = math.sqrt(dt)
    for k in range(steps):
        w = dW[:, k, 0].reshape(shape)
        d1, d2 = x + dt * drift(x), diffusion(x)
        if case["scheme"] == "euler":
            x = d1 + w * d2
            continue
        vt, vp, vm = d1 + w * d2, d1 + root * d2, d1 - root * d2
        dw2 = (0.25 / root) * (w * w - dt)
        x = (0.5 * d1 + 0.5 * dt * drift(vt) + 0.5 * x + 0.5 * w * d2
             + (dw2 + 0.25 * w) * diffusion(vp) + (0.25 * w - dw2) * diffusion(vm))
    if case["open"]:
        x = x.transpose(1, 2)
    return x.reshape(ntraj, -1)
