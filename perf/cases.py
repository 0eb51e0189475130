"""The performance cases of the statevector framework.

A case is one call that a user's program makes again and again: an adjoint
gradient of a McClean or QAOA circuit (through the host API, with device
tensors, or through autograd), a forward run with its final state, a run
with basis-state shots, or a batch of small circuits in one graph replay.

  listed()             the cases that are always measured
  draw(rng)            one more case from the same ranges
  prepare(case, seed)  the circuit, its parameters and what a program keeps
  run(state)           one pass through the public entry points
  work(case)           bytes and floating-point operations of one pass
  exact(case, seed)    the same outputs from plain complex128 torch

Circuit axes are drawn uniformly from {X, Y, Z} and angles uniformly from
[0, 2 pi); QAOA graphs are 3-regular with beta, gamma uniform in [0, pi).
"""
import math

import numpy as np
import torch

X, Y, Z, ZZ = 0, 1, 2, 3
# on-chip memory that a state may stay in from one layer to the next (L2)
ON_CHIP = 100e6


# ------------------------------------------------------------------ cases

def listed():
    return [
        # the smallest whole call: host angles in, host E and gradient out (a
        # variational loop on ten qubits, where launches and latency count)
        {"name": "mcclean_n10_c128_host", "kind": "mcclean", "api": "host", "n": 10, "layers": 10,
         "dtype": "complex128", "entangler": "cnot", "placement": "before", "obs": "zz01", "grad_mode": "auto"},
        # an odd small size in single precision, one circuit at a time
        {"name": "mcclean_n15_c64", "kind": "mcclean", "api": "tensors", "n": 15, "layers": 20,
         "dtype": "complex64", "entangler": "cnot", "placement": "before", "obs": "chain", "grad_mode": "auto"},
        # an odd medium size with a transverse-field observable (X and Y terms)
        {"name": "mcclean_n17_c128_ising", "kind": "mcclean", "api": "tensors", "n": 17, "layers": 20,
         "dtype": "complex128", "entangler": "cnot", "placement": "before", "obs": "ising", "grad_mode": "auto"},
        # a training step through autograd; CZ ladder after the rotations
        {"name": "mcclean_n20_c128_cz", "kind": "mcclean", "api": "autograd", "n": 20, "layers": 50,
         "dtype": "complex128", "entangler": "cz", "placement": "after", "obs": "chain", "grad_mode": "auto"},
        # the benchmark circuit in both precisions
        {"name": "mcclean_n24_c128", "kind": "mcclean", "api": "tensors", "n": 24, "layers": 50,
         "dtype": "complex128", "entangler": "cnot", "placement": "before", "obs": "chain", "grad_mode": "auto"},
        {"name": "mcclean_n24_c64", "kind": "mcclean", "api": "tensors", "n": 24, "layers": 50,
         "dtype": "complex64", "entangler": "cnot", "placement": "before", "obs": "chain", "grad_mode": "auto"},
        # a state too large for its history: psi is uncomputed backwards
        {"name": "mcclean_n28_c128", "kind": "mcclean", "api": "tensors", "n": 28, "layers": 5,
         "dtype": "complex128", "entangler": "cnot", "placement": "before", "obs": "chain",
         "grad_mode": "uncompute"},
        # the forward direction alone, with the final state
        {"name": "mcclean_n23_c64_run", "kind": "run", "n": 23, "layers": 30, "dtype": "complex64",
         "entangler": "cnot", "placement": "before", "obs": "chain"},
        # MaxCut QAOA gradient
        {"name": "qaoa_n24_c128", "kind": "qaoa", "n": 24, "layers": 6, "dtype": "complex128"},
        # MaxCut QAOA forward run and 100 basis-state shots
        {"name": "qaoa_n20_c128_shots", "kind": "shots", "n": 20, "layers": 4, "dtype": "complex128",
         "shots": 100},
        # many parameter vectors of one small circuit in one graph replay
        {"name": "batch_n14_c64", "kind": "batch", "n": 14, "layers": 30, "jobs": 2048, "dtype": "complex64"},
        # a serving round's mix of small circuits of both kinds
        {"name": "batch_mixed_c128", "kind": "mixed", "n_min": 8, "n_max": 14, "jobs": 96, "mix": 1,
         "dtype": "complex128"},
    ]


def draw(rng):
    dtype = rng.choice(["complex128", "complex64"])
    f = 1 if dtype == "complex64" else 4
    kind = rng.choice(["mcclean", "mcclean", "mcclean", "run", "qaoa", "shots", "batch", "mixed"])
    if kind in ("mcclean", "run"):
        n = rng.randint(8, 27)
        # no dearer than the largest listed case, and a history of 50 GB at most
        most = int(2.0 ** 28 * 28 * 5 * 4 / (2.0 ** n * n * f))
        layers = rng.randint(min(5, max(1, most)), max(1, min(60, most)))
        ent = rng.choice(["cnot", "cnot", "cz", "cnot_periodic"])
        if n % 2 and ent == "cnot_periodic":
            ent = "cnot"
        case = {"kind": kind, "n": n, "layers": layers, "dtype": dtype, "entangler": ent,
                "placement": rng.choice(["before", "after"]), "obs": rng.choice(["zz01", "chain", "ising"])}
        if kind == "mcclean":
            case["api"] = rng.choice(["host", "tensors", "autograd"])
            case["grad_mode"] = "uncompute" if n >= 25 else rng.choice(["auto", "auto", "uncompute"])
        return case
    if kind in ("qaoa", "shots"):
        n = 2 * rng.randint(5, 12)
        case = {"kind": kind, "n": n, "layers": rng.randint(1, 10 if n < 24 else 6), "dtype": dtype}
        if kind == "shots":
            case["shots"] = int(round(10 ** rng.uniform(1, 3)))
        return case
    if kind == "batch":
        n = rng.randint(8, 15 if dtype == "complex64" else 14)
        layers = rng.randint(5, 40)
        most = 2.0 ** 14 * 14 * 30 * 4096 / (2.0 ** n * n * layers * f * f)
        jobs = int(round(2 ** rng.uniform(5, min(12, max(5.1, math.log2(most))))))
        return {"kind": "batch", "n": n, "layers": layers, "jobs": jobs, "dtype": dtype}
    n_min = rng.randint(8, 11)
    return {"kind": "mixed", "n_min": n_min, "n_max": rng.randint(n_min + 1, 14), "jobs": rng.randint(32, 128),
            "mix": rng.randint(2, 1 << 20), "dtype": dtype}


# ------------------------------------------------------------------ inputs

def _terms(name, n, rng):
    """Observable terms (kind, q0, q1, weight)."""
    if name == "zz01":
        return [(ZZ, 0, 1, 1.0)]
    chain = [(ZZ, i, i + 1, 1.0) for i in range(n - 1)]
    if name == "chain":
        return chain
    return ([(X, q, q, -0.7) for q in range(n)] + [(Y, q, q, 0.25) for q in range(0, n, 3)]
            + [(Z, q, q, float(w)) for q, w in enumerate(rng.choice([0.5, -0.5, 0.125], n))] + chain)


def _observable(terms, n):
    d = {}
    for key, k in (("x", X), ("y", Y), ("z", Z)):
        own = [t for t in terms if t[0] == k]
        if own:
            d[key] = np.full(n, None)
            for t in own:
                d[key][t[1]] = t[3]
    zz = [t for t in terms if t[0] == ZZ]
    if zz:
        d["zz"] = np.full((n, n), None)
        for t in zz:
            d["zz"][t[1], t[2]] = t[3]
    return d


def _graph(n, rng):
    """Edges of a 3-regular graph: a shuffled ring and a perfect matching of its non-neighbours."""
    ring = rng.permutation(n)
    while True:
        m = rng.permutation(n)
        a, b = m[: n // 2], m[n // 2:]
        d = np.abs(a - b)
        if np.all((d > 1) & (d < n - 1)):
            break
    e = [(ring[i], ring[(i + 1) % n]) for i in range(n)] + [(ring[i], ring[j]) for i, j in zip(a, b)]
    return sorted((int(min(p)), int(max(p))) for p in e)


def _inputs(case, seed):
    """What a case's outputs depend on, as host arrays."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("mcclean", "run", "batch"):
        n, L = case["n"], case["layers"]
        rows = case.get("jobs", 1)
        return {"axes": rng.integers(0, 3, (L, n)), "angles": rng.uniform(0, 2 * np.pi, (rows, L, n)),
                "terms": _terms(case.get("obs", "chain"), n, rng)}
    if kind in ("qaoa", "shots"):
        n, p = case["n"], case["layers"]
        return {"edges": _graph(n, rng), "params": rng.uniform(0, np.pi, (p, 2)),
                "shot_seed": int(rng.integers(1 << 40))}
    # which circuits a mix holds goes by the case, their axes, graphs and parameters by the seed
    mix, jobs = np.random.default_rng(case["mix"]), []
    for _ in range(case["jobs"]):
        if mix.random() < 0.6:
            n, L = int(mix.integers(case["n_min"], case["n_max"] + 1)), int(mix.integers(5, 61))
            jobs.append({"n": n, "axes": rng.integers(0, 3, (L, n)), "angles": rng.uniform(0, 2 * np.pi, (1, L, n)),
                         "terms": _terms("chain", n, rng)})
        else:
            n = 2 * int(mix.integers((case["n_min"] + 1) // 2, case["n_max"] // 2 + 1))
            p = int(mix.integers(1, 7))
            jobs.append({"n": n, "edges": _graph(n, rng), "params": rng.uniform(0, np.pi, (p, 2))})
    return {"jobs": jobs}


# ------------------------------------------------------------------ the calls

def _mcclean(n, inp, case, angles):
    from qradient_gb300 import McClean

    return McClean(n, _observable(inp["terms"], n), len(inp["axes"]), axes=inp["axes"], angles=angles,
                   dtype=case["dtype"], entangler=case.get("entangler", "cnot"),
                   placement=case.get("placement", "before"), grad_mode=case.get("grad_mode", "auto"))


def _qaoa(n, inp, case):
    from qradient_gb300 import Qaoa
    from qradient_gb300.optimization_problems import MaxCut

    return Qaoa(n, MaxCut(n, edge_set=inp["edges"]).to_observable(), len(inp["params"]), dtype=case["dtype"])


def prepare(case, seed):
    inp = _inputs(case, seed)
    kind = case["kind"]
    dev = torch.device("cuda", torch.cuda.current_device())
    if kind in ("mcclean", "run"):
        host = inp["angles"][0]
        c = _mcclean(case["n"], inp, case, host)
        st = {"kind": kind if kind == "run" else case["api"], "circuit": c}
        if st["kind"] in ("tensors", "autograd"):
            st["angles"] = torch.tensor(host, dtype=torch.float64, device=dev)
        return st
    if kind in ("qaoa", "shots"):
        st = {"kind": kind, "circuit": _qaoa(case["n"], inp, case)}
        if kind == "qaoa":
            st["params"] = torch.tensor(inp["params"], dtype=torch.float64, device=dev)
        else:
            st.update(betas=inp["params"][:, 0], gammas=inp["params"][:, 1], shots=case["shots"],
                      seed=inp["shot_seed"])
        return st
    from qradient_gb300.batched import Batch, mcclean_batch

    if kind == "batch":
        b = mcclean_batch(case["n"], case["layers"], inp["axes"], _observable(inp["terms"], case["n"]), case["jobs"],
                          dtype=case["dtype"])
        params = torch.tensor(inp["angles"].reshape(-1), dtype=torch.float64, device=dev)
    else:
        b = Batch(dtype=case["dtype"])
        flat = []
        for j in inp["jobs"]:
            if "axes" in j:
                b.add(_mcclean(j["n"], j, case, j["angles"][0]))
                flat.append(j["angles"].reshape(-1))
            else:
                b.add(_qaoa(j["n"], j, case), params=j["params"])
                flat.append(j["params"].reshape(-1))
        b.finalize()
        params = torch.tensor(np.concatenate(flat), dtype=torch.float64, device=dev)
    return {"kind": "batch", "batch": b, "params": params}


def run(state):
    kind = state["kind"]
    if kind == "host":
        E, g = state["circuit"].grad_run()
        return {"E": E, "grad": g}
    if kind == "tensors":
        E, g = state["circuit"].grad_run_tensors(angles=state["angles"])
        return {"E": E, "grad": g}
    if kind == "autograd":
        from qradient_gb300.autograd import mcclean_expectation

        a = state["angles"].detach().requires_grad_(True)
        E = mcclean_expectation(a, state["circuit"])
        E.backward()
        return {"E": E.detach(), "grad": a.grad}
    if kind == "run":
        c = state["circuit"]
        E = c.run_expec_val()
        return {"E": E, "state": c.state.tensor}
    if kind == "qaoa":
        E, g = state["circuit"].grad_run_tensors(state["params"])
        return {"E": E, "grad": g}
    if kind == "shots":
        c = state["circuit"]
        E = c.run_expec_val(state["betas"], state["gammas"])
        return {"E": E, "shots": c.sample(state["shots"], seed=state["seed"]), "state": c.state.tensor}
    b = state["batch"]
    b.params_flat[: state["params"].numel()].copy_(state["params"])
    E, _ = b.grad()
    return {"E": E, "grad": b.grads_flat}


# ------------------------------------------------------------------ work

def _circuit_work(n, layers, esize, grad, qaoa):
    """A rotation of n qubits costs 6 flops per amplitude and qubit, its
    gradient reduction 4.  A state beyond on-chip memory is read and written
    once per layer, and lambda and psi once more each on the way back."""
    N = 2.0 ** n
    flops = N * n * layers * (6 + (10 if grad else 0)) + 6 * N * (1 + (layers if qaoa else 0))
    nparam = 2 * layers if qaoa else n * layers
    io = 8 * (nparam * (2 if grad else 1) + 1)
    state = N * esize
    big = state if state > ON_CHIP else 0.0
    return big * layers * (2 + (3 if grad else 0)) + io, flops


def work(case):
    e = 16 if case["dtype"] == "complex128" else 8
    kind = case["kind"]
    if kind in ("mcclean", "qaoa"):
        b, f = _circuit_work(case["n"], case["layers"], e, True, kind == "qaoa")
    elif kind in ("run", "shots"):
        b, f = _circuit_work(case["n"], case["layers"], e, False, kind == "shots")
        b += 2.0 ** case["n"] * e  # the final state is an output
    elif kind == "batch":
        b, f = _circuit_work(case["n"], case["layers"], e, True, False)
        b, f = b * case["jobs"], f * case["jobs"]
    else:
        # mean over the mix: 60% McClean with 5..60 layers, 40% QAOA with 1..6
        ns = range(case["n_min"], case["n_max"] + 1)
        mc = [_circuit_work(n, 32.5, e, True, False) for n in ns]
        qa = [_circuit_work(n, 3.5, e, True, True) for n in ns if n % 2 == 0] or mc
        b, f = (case["jobs"] * (0.6 * sum(w[k] for w in mc) / len(mc) + 0.4 * sum(w[k] for w in qa) / len(qa))
                for k in (0, 1))
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact values

class _Sim:
    """Rows of n-qubit states in complex128 torch; qubit q is bit n-1-q."""

    def __init__(self, n, rows, dev):
        self.n, self.rows, self.dev = n, rows, dev

    def pair(self, v, q):
        w = v.view(self.rows, 2 ** q, 2, 2 ** (self.n - 1 - q))
        return w[:, :, 0], w[:, :, 1]

    def col(self, t):
        return t.view(-1, 1, 1).to(torch.complex128) if self.rows > 1 else complex(t.reshape(-1)[0].item())

    def rotate(self, v, q, axis, theta):
        """v <- exp(-i theta/2 P_q) v in place; theta: one angle per row."""
        a, b = self.pair(v, q)
        c, s = self.col(torch.cos(theta / 2)), self.col(torch.sin(theta / 2))
        if axis == Z:
            a.mul_(c - 1j * s)
            b.mul_(c + 1j * s)
            return
        sa, sb = (-1j * s, -1j * s) if axis == X else (-s, s)
        a0 = a.clone()
        a.mul_(c).add_(b * sa)
        b.mul_(c).add_(a0.mul_(sb))

    def overlap(self, lam, psi, q, axis):
        """Im <lam| P_q |psi> per row."""
        (la, lb), (a, b) = self.pair(lam, q), self.pair(psi, q)
        if axis == Z:
            return ((la.conj() * a).sum((1, 2)) - (lb.conj() * b).sum((1, 2))).imag
        u, w = (la.conj() * b).sum((1, 2)), (lb.conj() * a).sum((1, 2))
        return (u + w).imag if axis == X else (w - u).real

    def ladder(self, kind):
        """(forward gather, inverse gather) of a CNOT ladder; a sign for CZ."""
        n = self.n
        x = torch.arange(2 ** n, device=self.dev)
        if kind == "cz":
            w, par = x & (x >> 1), torch.zeros_like(x)
            for k in range(n):
                par ^= (w >> k) & 1
            return "cz", (1 - 2 * par).to(torch.float64)
        pairs = [(q, q + 1) for q in range(1, n - 1, 2)]
        if kind == "cnot_periodic":
            pairs.append((n - 1, 0))
        pairs += [(q, q + 1) for q in range(0, n - 1, 2)]

        def image(order):
            y = x.clone()
            for c, t in order:
                y ^= ((y >> (n - 1 - c)) & 1) << (n - 1 - t)
            return y

        return "cnot", (image(pairs[::-1]), image(pairs))

    def entangle(self, v, ent, inverse):
        if ent[0] == "cz":
            return v.mul_(ent[1])
        return v[:, ent[1][1 if inverse else 0]]

    def diagonal(self, terms):
        d = torch.zeros(2 ** self.n, dtype=torch.float64, device=self.dev)
        x = torch.arange(2 ** self.n, device=self.dev)
        for kind, i, j, w in terms:
            if kind in (Z, ZZ):
                s = (x >> (self.n - 1 - i)) & 1
                if kind == ZZ:
                    s = s ^ ((x >> (self.n - 1 - j)) & 1)
                d += w * (1 - 2 * s).to(torch.float64)
        return d

    def observe(self, psi, terms):
        lam = psi * self.diagonal(terms)
        for kind, i, _, w in terms:
            if kind in (X, Y):
                (la, lb), (a, b) = self.pair(lam, i), self.pair(psi, i)
                la += w * b if kind == X else (-1j * w) * b
                lb += w * a if kind == X else (1j * w) * a
        return lam

    def expec(self, psi, lam):
        return (psi.conj() * lam).sum(1).real


def _exact_mcclean(n, axes, angles, terms, entangler, placement, grad, dev):
    """E [rows], gradient [rows, L, n] (or None) and the final states."""
    rows, L = angles.shape[0], len(axes)
    S = _Sim(n, rows, dev)
    th = torch.tensor(angles, dtype=torch.float64, device=dev)
    c, s = math.cos(math.pi / 8), math.sin(math.pi / 8)
    v = torch.ones(1, dtype=torch.complex128, device=dev)
    for _ in range(n):
        v = torch.kron(v, torch.tensor([c, s], dtype=torch.complex128, device=dev))
    psi = v.repeat(rows, 1)
    ent = S.ladder(entangler) if entangler and n > 1 else None
    for i in range(L):
        if ent and placement == "before":
            psi = S.entangle(psi, ent, False)
        for q in range(n):
            S.rotate(psi, q, int(axes[i, q]), th[:, i, q])
        if ent and placement == "after":
            psi = S.entangle(psi, ent, False)
    lam = S.observe(psi, terms)
    E = S.expec(psi, lam)
    if not grad:
        return E, None, psi
    g = torch.zeros(rows, L, n, dtype=torch.float64, device=dev)
    for i in range(L - 1, -1, -1):
        if ent and placement == "after":
            psi, lam = S.entangle(psi, ent, True), S.entangle(lam, ent, True)
        for q in range(n):
            g[:, i, q] = S.overlap(lam, psi, q, int(axes[i, q]))
        for q in range(n):
            S.rotate(psi, q, int(axes[i, q]), -th[:, i, q])
            S.rotate(lam, q, int(axes[i, q]), -th[:, i, q])
        if ent and placement == "before":
            psi, lam = S.entangle(psi, ent, True), S.entangle(lam, ent, True)
    return E, g, psi


def _exact_qaoa(n, edges, params, grad, dev):
    S = _Sim(n, 1, dev)
    cost = S.diagonal([(ZZ, i, j, 1.0) for i, j in edges])
    psi = torch.full((1, 2 ** n), 2.0 ** (-n / 2), dtype=torch.complex128, device=dev)
    prm = torch.tensor(params, dtype=torch.float64, device=dev)
    for beta, gamma in prm:
        psi = psi * torch.exp(-1j * gamma * cost)
        for q in range(n):
            S.rotate(psi, q, X, beta)
    lam = psi * cost
    E = S.expec(psi, lam)
    if not grad:
        return E, None, psi
    g = torch.zeros(len(params), 2, dtype=torch.float64, device=dev)
    for i in range(len(params) - 1, -1, -1):
        beta, gamma = prm[i]
        for q in range(n):
            g[i, 0] += S.overlap(lam, psi, q, X)[0]
        for q in range(n):
            S.rotate(psi, q, X, -beta)
            S.rotate(lam, q, X, -beta)
        g[i, 1] = 2 * (lam.conj() * psi * cost).sum().imag
        back = torch.exp(1j * gamma * cost)
        psi, lam = psi * back, lam * back
    return E, g, psi


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    inp = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("mcclean", "run", "batch"):
        E, g, psi = _exact_mcclean(case["n"], inp["axes"], inp["angles"], inp["terms"], case.get("entangler", "cnot"),
                                   case.get("placement", "before"), kind != "run", dev)
        if kind == "run":
            return {"E": float(E[0]), "state": psi.reshape(-1)}
        if kind == "batch":
            return {"E": E, "grad": g.reshape(-1)}
        if case["api"] == "host":
            return {"E": float(E[0]), "grad": g[0].cpu().numpy()}
        return {"E": E, "grad": g.reshape(-1)} if case["api"] == "tensors" else {"E": E[0], "grad": g[0]}
    if kind in ("qaoa", "shots"):
        E, g, psi = _exact_qaoa(case["n"], inp["edges"], inp["params"], kind == "qaoa", dev)
        if kind == "qaoa":
            return {"E": E, "grad": g.reshape(-1)}
        return {"E": float(E[0]), "shots": None, "state": psi.reshape(-1)}
    Es, gs = [], []
    for j in inp["jobs"]:
        if "axes" in j:
            E, g, _ = _exact_mcclean(j["n"], j["axes"], j["angles"], j["terms"], "cnot", "before", True, dev)
        else:
            E, g, _ = _exact_qaoa(j["n"], j["edges"], j["params"], True, dev)
        Es.append(E)
        gs.append(g.reshape(-1))
    return {"E": torch.cat(Es), "grad": torch.cat(gs)}
