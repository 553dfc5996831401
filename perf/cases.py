"""The work that a user of this framework has it do, as cases that can be timed and checked.

Every case goes through the package's public entry points (StateVector, HEAProblem, Server) as a
program does: host gate records or parameter vectors in, expectation values, outcomes, amplitudes,
gradients or tensors out.  Handles that a program keeps (a state, a problem, a server) are made in
prepare(); a pass resets and runs them.

Kinds of cases:
  circuit  reset a state, run a circuit of gate records, read the result.  "brickwork" is a layer
           of RX, RY, RZ on every qubit and CNOTs on alternating neighbour pairs, with a ZZ layer
           every `zz` layers (0: none); "qaoa" is cost and mixer layers on a random Ising graph.
           `mode` "fused" is complex64's default (tensor cores), "tiled" the more exact one, and
           what complex128 and small states run.  `read` says what the program wants back: "shots" (<Z> of every qubit and sampled outcomes), "energy"
           (<Z> and a Pauli-sum expectation) or "amplitudes" (the whole state on the host).  QAOA's
           <Z> are zero by symmetry: its "energy" is that of an Ising chain with a transverse field,
           and "shots" reads that energy and outcomes.
  observe  reductions and sampling on a state that is already there.
  vqe      energies, and gradients if `grad`, of a batch of parameter vectors of the
           hardware-efficient ansatz.
  qgt      the quantum geometric tensor of that ansatz at one parameter vector.
  serve    a burst of requests to the continuous-batching server, waited for in order.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from moonlab_b200 import StateVector
from moonlab_b200.circuits import (GATE_CNOT, GATE_H, GATE_RX, GATE_RY, GATE_RZ, GATE_ZZ, SplitMix64,
                                   brickwork, qaoa_circuit)
from moonlab_b200.serving import Server
from moonlab_b200.vqe import HEAProblem


def listed():
    return [
        # the smallest call: a ten-qubit circuit and its state, where launches and the host are the time
        {"name": "circuit_10q", "kind": "circuit", "form": "brickwork", "n": 10, "depth": 10, "zz": 0,
         "dtype": "c128", "mode": "tiled", "read": "amplitudes", "shots": 0},
        # an everyday circuit: 20 qubits, depth 20, 1024 shots
        {"name": "circuit_20q", "kind": "circuit", "form": "brickwork", "n": 20, "depth": 20, "zz": 0,
         "dtype": "c128", "mode": "tiled", "read": "shots", "shots": 1024},
        # QAOA at an odd width: long-range CNOT . RZ . CNOT terms on a random graph
        {"name": "qaoa_23q", "kind": "circuit", "form": "qaoa", "n": 23, "depth": 4, "zz": 0,
         "dtype": "c128", "mode": "tiled", "read": "shots", "shots": 1000},
        # complex64 where the fused path's rounding is too coarse; an energy read back
        {"name": "circuit_27q_c64", "kind": "circuit", "form": "brickwork", "n": 27, "depth": 20, "zz": 0,
         "dtype": "c64", "mode": "tiled", "read": "energy", "shots": 0},
        # the benchmark's circuit: 30 qubits, depth 40, a ZZ layer every 4 layers, 1024 shots
        {"name": "circuit_30q", "kind": "circuit", "form": "brickwork", "n": 30, "depth": 40, "zz": 4,
         "dtype": "c128", "mode": "tiled", "read": "shots", "shots": 1024},
        # the same circuit on the fused complex64 path
        {"name": "circuit_30q_fused", "kind": "circuit", "form": "brickwork", "n": 30, "depth": 40, "zz": 4,
         "dtype": "c64", "mode": "fused", "read": "energy", "shots": 0},
        # measurement of a large state: norm, <Z>, a Pauli sum, 4096 shots
        {"name": "observe_29q", "kind": "observe", "n": 29, "dtype": "c128", "terms": 58, "shots": 4096},
        # an optimiser's step on a small molecule: two parameter vectors
        {"name": "vqe_12q", "kind": "vqe", "n": 12, "layers": 8, "batch": 2, "dtype": "c128", "grad": True},
        # the benchmark's batch of gradients
        {"name": "vqe_20q", "kind": "vqe", "n": 20, "layers": 8, "batch": 256, "dtype": "c128", "grad": True},
        {"name": "vqe_20q_c64", "kind": "vqe", "n": 20, "layers": 8, "batch": 256, "dtype": "c64", "grad": True},
        # a natural-gradient step's metric and curvature
        {"name": "qgt_15q", "kind": "qgt", "n": 15, "layers": 6},
        # a burst of small and medium requests to the server
        {"name": "serve_64", "kind": "serve", "requests": 64, "n_lo": 8, "n_hi": 16, "depth": 40},
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return min(hi, int(round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["circuit"] * 4 + ["observe"] + ["vqe"] * 3 + ["qgt"] + ["serve"])
    if kind == "circuit":
        dtype = rng.choice(["c128", "c128", "c64"])
        form = rng.choice(["brickwork", "brickwork", "qaoa"])
        n = rng.randint(3, 29)
        if form == "qaoa":
            depth, zz = _between(rng, 1, 6), 0
            n = min(n, 27)
        else:
            depth, zz = _between(rng, 3, 40), rng.choice([0, 0, 1, 2, 4])
        mode = rng.choice(["tiled", "fused"]) if dtype == "c64" and n >= 13 else "tiled"
        read = rng.choice(["shots", "energy", "amplitudes"])
        if dtype == "c64" and read == "shots":
            read = "energy"
        if n > 20 and read == "amplitudes":
            read = "energy"
        shots = _between(rng, 1, 4096) if read == "shots" else 0
        return {"kind": "circuit", "form": form, "n": n, "depth": depth, "zz": zz, "dtype": dtype, "mode": mode,
                "read": read, "shots": shots}
    if kind == "observe":
        n = rng.randint(8, 29)
        return {"kind": "observe", "n": n, "dtype": "c128", "terms": _between(rng, 1, 2 * n),
                "shots": _between(rng, 1, 4096)}
    if kind == "vqe":
        n = rng.randint(3, 20)
        return {"kind": "vqe", "n": n, "layers": rng.randint(1, 8), "batch": _between(rng, 1, 256),
                "dtype": rng.choice(["c128", "c64"]), "grad": rng.random() < 0.8}
    if kind == "qgt":
        return {"kind": "qgt", "n": rng.randint(4, 16), "layers": rng.randint(1, 6)}
    n_lo = rng.randint(6, 12)
    return {"kind": "serve", "requests": _between(rng, 4, 128), "n_lo": n_lo, "n_hi": rng.randint(n_lo, 16),
            "depth": _between(rng, 8, 80)}


def _pauli_terms(n, count, seed):
    """`count` one- and two-local Pauli strings on n qubits with N(0, 1) coefficients."""
    r = np.random.default_rng(seed)
    xs, zs = np.zeros(count, np.uint64), np.zeros(count, np.uint64)
    for t in range(count):
        for q in r.permutation(n)[:min(n, int(r.integers(1, 3)))]:
            p = int(r.integers(1, 4))
            if p in (1, 2):
                xs[t] |= np.uint64(1 << int(q))
            if p in (2, 3):
                zs[t] |= np.uint64(1 << int(q))
    return xs, zs, r.standard_normal(count)


def _terms(case, seed):
    n = case["n"]
    if case.get("form") == "qaoa":
        r = np.random.default_rng([seed, 3])
        zs = [3 << q for q in range(n - 1)] + [0] * n
        xs = [0] * (n - 1) + [1 << q for q in range(n)]
        return np.array(xs, np.uint64), np.array(zs, np.uint64), r.standard_normal(2 * n - 1)
    return _pauli_terms(n, case.get("terms", 2 * n), [seed, 3])


def _gates(case, seed):
    if case["form"] == "qaoa":
        return qaoa_circuit(case["n"], case["depth"], 0x0A0A + seed)
    return brickwork(case["n"], case["depth"], 0xB1C0 + seed, zz_every=case["zz"])


def _vqe_inputs(case, seed):
    n = case["n"]
    r = np.random.default_rng([seed, n, case["layers"]])
    xs, zs, c = _pauli_terms(n, 4 * n, [seed, 7])
    params = r.uniform(-math.pi, math.pi, (case.get("batch", 1), 2 * n * case["layers"]))
    return xs, zs, c, params


def _requests(case, seed):
    """(qubits, records, shots, seed, dtype) of each request; complex64 ones stay small, where outcomes are
    far enough apart that rounding does not choose between them."""
    r = np.random.default_rng([case["requests"], case["n_lo"], case["n_hi"], case["depth"]])
    out = []
    for i in range(case["requests"]):  # the sizes belong to the case, circuits and outcomes to the seed
        n = int(r.integers(case["n_lo"], case["n_hi"] + 1))
        depth = int(r.integers(max(1, case["depth"] // 4), case["depth"] + 1))
        shots = int(r.integers(1, 1025))
        dtype = "c64" if n <= 10 and r.random() < 0.5 else "c128"
        out.append((n, brickwork(n, depth, 0x5E00 + 1000 * seed + i), shots, 1 + 7919 * seed + i, dtype))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("circuit", "observe"):
        n = case["n"]
        s["state"] = StateVector(n, dtype=case["dtype"])
        s["uniforms"] = SplitMix64(0x5EED + seed).uniforms(case["shots"])
        s["terms"] = _terms(case, seed)
        if kind == "circuit":
            s["gates"] = _gates(case, seed)
            s["state"].set_exec_mode(case["mode"])
        else:  # the state that is measured: a few layers deep
            s["state"].run(brickwork(n, 3, 0x0B5 + seed))
            s["state"].synchronize()
    elif kind == "vqe":
        xs, zs, c, s["params"] = _vqe_inputs(case, seed)
        s["problem"] = HEAProblem(case["n"], case["layers"], c, xmasks=xs, zmasks=zs, dtype=case["dtype"])
    elif kind == "qgt":
        s["params"] = _vqe_inputs(case, seed)[3][0]
        s["problem"] = HEAProblem(case["n"], case["layers"], [], xmasks=[], zmasks=[])
    else:
        s["requests"] = _requests(case, seed)
        s["server"] = Server(hbm_budget=8 << 30, workers=8)
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "circuit":
        sv = s["state"]
        sv.reset()
        sv.run(s["gates"])
        if case["read"] == "amplitudes":
            return {"amplitudes": sv.amplitudes()}
        out = {} if case["form"] == "qaoa" else {"z": sv.expectation_z_all()}
        if case["read"] == "energy" or case["form"] == "qaoa":
            out["energy"] = np.float64(sv.expectation_pauli_sum(*s["terms"]))
        if case["read"] == "shots":
            out["shots"] = sv.sample(s["uniforms"]).astype(np.int64)
        return out
    if kind == "observe":
        sv = s["state"]
        return {"norm": np.float64(sv.norm_sq()), "z": sv.expectation_z_all(),
                "energy": np.float64(sv.expectation_pauli_sum(*s["terms"])),
                "shots": sv.sample(s["uniforms"]).astype(np.int64)}
    if kind == "vqe":
        e, g = s["problem"].evaluate(s["params"], want_grad=case["grad"])
        return {"energies": e, "gradients": g} if case["grad"] else {"energies": e}
    if kind == "qgt":
        metric, curvature = s["problem"].geometry(s["params"])
        return {"metric": metric, "curvature": curvature}
    server = s["server"]
    tickets = [server.submit(n, g, shots, rseed, dtype) for n, g, shots, rseed, dtype in s["requests"]]
    return {"outcomes": np.concatenate([server.wait(t)[0] for t in tickets]).astype(np.int64)}


def work(case):
    """Bytes and operations of one pass.  A run of one-qubit gates is counted as one real rotation (4
    multiply-adds an amplitude: its phases join a diagonal), the diagonals between two layers as one complex
    product, permutations as nothing; a state is written once and read once for each kind of result."""
    kind, n = case["kind"], case.get("n", 0)
    amp = 16 if case.get("dtype", "c128") == "c128" else 8
    dim = 2.0 ** n
    if kind == "circuit":
        layers = case["depth"] + (case["depth"] // case["zz"] if case["zz"] else 0)
        reads = {"shots": 2, "energy": 2, "amplitudes": 1}[case["read"]]
        return {"bytes": dim * amp * (1 + reads), "flops": dim * (8 * n * case["depth"] + 6 * layers)}
    if kind == "observe":
        return {"bytes": 2 * dim * amp, "flops": dim * (4 + n + 4 * case["terms"])}
    if kind == "vqe":
        # forward; lambda = H psi; then psi and lambda backwards with 4 operations for each gradient
        fwd = 8 * n * case["layers"] + 6 * case["layers"]
        flops = dim * case["batch"] * (fwd + 4 * 4 * n + (2 * fwd + 8 * n * case["layers"] if case["grad"] else 0))
        return {"bytes": dim * amp * case["batch"] * (4 if case["grad"] else 2), "flops": flops}
    if kind == "qgt":
        p = 2 * n * case["layers"] + 1
        return {"bytes": 2 * dim * 16 * p, "flops": dim * (p * (8 * n + 6) * case["layers"] + 4.0 * p * p)}
    mid = (case["n_lo"] + case["n_hi"]) / 2
    return {"bytes": case["requests"] * 3 * 16 * 2.0 ** mid,
            "flops": case["requests"] * 2.0 ** mid * 0.6 * case["depth"] * (8 * mid + 6)}


def tolerance(case):
    kind = case["kind"]
    c64 = case.get("dtype") == "c64"
    if kind == "circuit":  # <Z> of a deep circuit on many qubits is a small difference of large sums
        if case["mode"] == "fused":
            return {"rel": 2.6e-2}
        return {"rel": 3e-4} if c64 else {"rel": 3e-12, "differ": 0.005}
    if kind == "observe":
        return {"rel": 2e-14, "differ": 0.005}
    if kind == "vqe":
        return {"rel": 6e-5} if c64 else {"rel": 5e-14}
    if kind == "qgt":
        return {"rel": 1e-14}
    return {"rel": 0.0, "differ": 0.005}


# ---------------------------------------------------------------------------------------------
# the same results in plain torch, complex128
# ---------------------------------------------------------------------------------------------
_I2 = np.eye(2)


def _gate_matrix(t, theta):
    c, s = math.cos(theta / 2), math.sin(theta / 2)
    if t == GATE_RX:
        return np.array([[c, -1j * s], [-1j * s, c]])
    if t == GATE_RY:
        return np.array([[c, -s], [s, c]], dtype=complex)
    if t == GATE_RZ:
        return np.diag([complex(c, -s), complex(c, s)])
    return np.array([[1, 1], [1, -1]], dtype=complex) * math.sqrt(0.5)  # H


def _embed(record, qubits):
    """The record's matrix on the sorted qubit list (the first qubit is the lowest bit)."""
    k = len(qubits)
    at = {q: i for i, q in enumerate(qubits)}
    idx = np.arange(1 << k)
    t, q = int(record["type"]), int(record["target"])
    if t == GATE_CNOT:
        m = np.zeros((1 << k, 1 << k), complex)
        m[idx ^ ((idx >> at[int(record["control"])] & 1) << at[q]), idx] = 1
        return m
    if t == GATE_ZZ:
        odd = (idx >> at[q] & 1) ^ (idx >> at[int(record["control"])] & 1)
        return np.diag(np.exp(-0.5j * record["theta"] * (1 - 2 * odd)))
    m = _gate_matrix(t, float(record["theta"]))
    out = np.eye(1)
    for j in range(k):
        out = np.kron(m if qubits[j] == q else _I2, out)
    return out


def _blocks(gates, most=5):
    """The records grouped into matrices on at most `most` qubits, in order."""
    open_, done = [], []
    for g in gates:
        qs = {int(g["target"])} | ({int(g["control"])} if g["control"] >= 0 else set())
        hit = [b for b in open_ if b[0] & qs]
        if len(qs.union(*[b[0] for b in hit])) <= most:
            merged = [qs.union(*[b[0] for b in hit]), [r for b in hit for r in b[1]] + [g]]
        else:
            done += hit
            merged = [qs, [g]]
        open_ = [b for b in open_ if not any(b is h for h in hit)] + [merged]
    for qs, records in done + open_:
        qubits = sorted(qs)
        m = np.eye(1 << len(qubits), dtype=complex)
        for r in records:
            m = _embed(r, qubits) @ m
        yield qubits, m


def _simulate(n, gates):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1
    for qubits, m in _blocks(gates):
        k = len(qubits)
        dims, axes, top = [], [], n
        for q in reversed(qubits):  # axes from the highest bit down
            dims += [1 << (top - q - 1), 2]
            axes.append(len(dims) - 1)
            top = q
        dims.append(1 << top)
        rest = [a for a in range(len(dims)) if a not in axes]
        order = axes + rest
        x = psi.reshape(dims).permute(order)
        shape = x.shape
        x = x.reshape(1 << k, -1)
        del psi
        x = torch.from_numpy(m).cuda() @ x
        psi = x.reshape(shape).permute(np.argsort(order).tolist()).reshape(-1)
        del x
    return psi


def _parity_signs(dim, mask):
    v = torch.arange(dim, device="cuda") & mask
    for s in (32, 16, 8, 4, 2, 1):
        v = v ^ (v >> s)
    return (1 - 2 * (v & 1)).to(torch.float64)


def _z_all(p, n):
    return torch.stack([(lambda v: v[:, 0].sum() - v[:, 1].sum())(p.view(-1, 2, 1 << q)) for q in range(n)])


def _apply_paulis(psi, xs, zs, cs):
    """sum_k c_k P_k psi over the last axis."""
    dim = psi.shape[-1]
    out = torch.zeros_like(psi)
    idx = torch.arange(dim, device="cuda")
    for x, z, c in zip(xs.tolist(), zs.tolist(), cs.tolist()):
        # (P psi)[i ^ x] = i^ny (-1)^{|i & z|} psi[i]
        src = idx ^ x
        out += (c * 1j ** (bin(x & z).count("1") % 4)) * _parity_signs(dim, z)[src] * psi[..., src]
    return out


def _energy(psi, xs, zs, cs):
    total = 0.0
    for x, z, c in zip(xs.tolist(), zs.tolist(), cs.tolist()):
        if x:
            idx = torch.arange(psi.numel(), device="cuda") ^ x
            v = psi[idx].conj() * psi
            del idx
        else:
            v = psi.abs().square().to(torch.complex128)
        v = (v * _parity_signs(psi.numel(), z)).sum().item()
        total += c * (1j ** (bin(x & z).count("1") % 4) * v).real
    return np.float64(total)


def _hea(n, layers, theta):
    """Final states [B, 2^n] and what undoes the ansatz: per layer the rotations and the ladder's index map."""
    idx = torch.arange(1 << n, device="cuda")
    to = idx.clone()
    for q in range(n - 1):
        to = to ^ ((to >> q & 1) << (q + 1))
    psi = torch.zeros((theta.shape[0], 1 << n), dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1
    back = torch.empty_like(to)
    back[to] = idx
    for layer in range(layers):
        for q in range(n):
            psi = _rotate(psi, n, q, theta, 2 * (layer * n + q), False)
        psi = psi[:, back]
    return psi, to


def _rotate(psi, n, q, theta, p, undo):
    """RZ . RY of qubit q (parameters p, p + 1), or its inverse, on every state."""
    v = psi.view(psi.shape[0], -1, 2, 1 << q)
    y, z = theta[:, p] / 2, theta[:, p + 1] / 2
    c, s = (f(y).view(-1, 1, 1) for f in (torch.cos, torch.sin))
    ph = torch.polar(torch.ones_like(z), z).view(-1, 1, 1)
    a, b = v[:, :, 0], v[:, :, 1]
    if undo:
        a, b = a * ph, b * ph.conj()
        a, b = c * a + s * b, c * b - s * a
    else:
        a, b = c * a - s * b, s * a + c * b
        a, b = a * ph.conj(), b * ph
    return torch.stack((a, b), 2).reshape(psi.shape)


def _vqe_exact(case, seed):
    xs, zs, cs, params = _vqe_inputs(case, seed)
    n, layers = case["n"], case["layers"]
    theta = torch.from_numpy(params).cuda()
    es, gs = [], []
    step = max(1, (1 << 26) >> n)
    for th in theta.split(step):
        psi, to = _hea(n, layers, th)
        lam = _apply_paulis(psi, xs, zs, cs)
        es.append((psi.conj() * lam).sum(1).real)
        if not case["grad"]:
            continue
        g = torch.zeros_like(th)
        for layer in reversed(range(layers)):
            psi, lam = psi[:, to], lam[:, to]
            for q in range(n):
                p = 2 * (layer * n + q)
                u, w = (x.view(len(th), -1, 2, 1 << q) for x in (psi, lam))
                m = [[(w[:, :, i].conj() * u[:, :, j]).sum((1, 2)) for j in (0, 1)] for i in (0, 1)]
                g[:, p + 1] = (m[0][0] - m[1][1]).imag
                ph2 = torch.polar(torch.ones_like(th[:, p + 1]), th[:, p + 1])  # RZ undone on both sides
                g[:, p] = (-1j * m[0][1] * ph2.conj() + 1j * m[1][0] * ph2).imag
                psi, lam = (_rotate(x, n, q, th, p, True) for x in (psi, lam))
        gs.append(g)
    out = {"energies": torch.cat(es)}
    if case["grad"]:
        out["gradients"] = torch.cat(gs)
    return out


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "circuit":
        psi = _simulate(n, _gates(case, seed))
        if case["read"] == "amplitudes":
            return {"amplitudes": psi}
        out = {} if case["form"] == "qaoa" else {"z": _z_all(psi.real.square() + psi.imag.square(), n)}
        if case["read"] == "energy" or case["form"] == "qaoa":
            out["energy"] = _energy(psi, *_terms(case, seed)) if n <= 27 else None
        if case["read"] == "shots":
            out["shots"] = None
        return out
    if kind == "observe":
        psi = _simulate(n, brickwork(n, 3, 0x0B5 + seed))
        p = psi.real.square() + psi.imag.square()
        return {"norm": np.float64(p.sum().item()), "z": _z_all(p, n), "shots": None,
                "energy": _energy(psi, *_terms(case, seed)) if n <= 27 else None}
    if kind == "vqe":
        return _vqe_exact(case, seed)
    if kind == "qgt":
        theta = torch.from_numpy(_vqe_inputs(case, seed)[3][:1]).cuda()
        count = theta.shape[1]
        rows = theta.repeat(count + 1, 1)
        rows[torch.arange(1, count + 1), torch.arange(count)] += math.pi  # d_i psi = psi(theta + pi e_i) / 2
        psi = _hea(n, case["layers"], rows)[0]
        gram = psi.conj() @ psi.T
        q = gram[1:, 1:] / 4 - torch.outer(gram[0, 1:].conj(), gram[0, 1:]) / 4
        return {"metric": q.real.clone(), "curvature": -2 * (q.imag - torch.diag(torch.diag(q.imag)))}
    return None
