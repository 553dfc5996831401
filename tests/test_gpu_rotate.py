"""Rotation programs of tile passes (kernels_rotate.cu) against gate-by-gate
execution and the CPU oracle: every kind of op they take (one-qubit
unitaries, X, CNOT, SWAP, diagonals on one to three qubits) on arbitrary
qubits, at the smallest register each type runs them on, where tiles have
free qubits and where the form is chosen pass by pass; ops they do not take
(controlled rotations, two controls, matrices that are not unitary) between
them; registers that are mostly zero after a reset.  complex128 1e-12 per
amplitude (the tolerance of the other paths), complex64 2e-5."""
from __future__ import annotations

import numpy as np
import pytest

from moonlab_b200 import StateVector, _lib
from moonlab_b200.circuits import GATE_DTYPE, brickwork, qaoa_circuit
from oracle import bindings as B

pytestmark = pytest.mark.gpu
TAKEN = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 20, 21, 22, 23, 27]  # gate record types


def circuit(n, count, seed, types=TAKEN):
    rng = np.random.default_rng(seed)
    g = np.zeros(count, dtype=GATE_DTYPE)
    for i in range(count):
        t = int(rng.choice(types))
        a, b = rng.choice(n, 2, replace=False)
        two = t in (10, 11, 12, 13) or t >= 23
        # a fifth of the angles at multiples of pi / 2, where a sine or cosine vanishes
        th = rng.integers(-4, 5) * np.pi / 2 if rng.random() < 0.2 else rng.uniform(-np.pi, np.pi)
        g[i] = (t, int(a), int(b) if two else -1, 0, float(th))
    return g


def qft(n):
    recs = []
    for q in range(n - 1, -1, -1):
        recs.append((4, q, -1, 0, 0.0))
        recs += [(23, q, k, 0, np.pi / (1 << (q - k))) for k in range(q - 1, -1, -1)]
    return np.array(recs, dtype=GATE_DTYPE)


@pytest.mark.parametrize("n,count,seed", [(13, 1, 1), (13, 300, 2), (14, 500, 3), (16, 400, 4), (18, 300, 5)])
def test_matches_the_oracle(gpu, n, count, seed):
    g = circuit(n, count, seed)
    with StateVector(n) as sv:
        sv.run(g)
        got = sv.amplitudes()
        st = sv.flush_stats()
        assert st["rotation_passes"] == st["passes"]
    assert np.abs(got - B.port_run(n, g)).max() < 1e-12


@pytest.mark.parametrize("n", [21, 22])
def test_complex64_against_complex128(gpu, n):
    g = np.concatenate([circuit(n, 200, n), brickwork(n, 4, n, zz_every=2)])
    with StateVector(n) as a, StateVector(n, "c64") as b:
        a.set_dense(False)
        a.run(g)
        b.set_exec_mode("tiled")
        b.run(g)
        want, got = a.amplitudes(), b.amplitudes()
        st = b.flush_stats()
        assert a.flush_stats()["rotation_passes"] == 0 and st["rotation_passes"] == st["passes"]
    assert np.abs(got - want).max() < 2e-5


@pytest.mark.parametrize("form", ["brickwork", "random"])
def test_pass_by_pass_choice(gpu, form):
    """26 qubits: each pass runs in its cheaper form."""
    n = 26
    g = brickwork(n, 5, 77, zz_every=2) if form == "brickwork" else circuit(n, 250, 78)
    with StateVector(n) as a, StateVector(n) as b:
        a.run(g)
        b.set_dense(False)
        b.run(g)
        x, y = a.amplitudes(), b.amplitudes()
        assert a.flush_stats()["rotation_passes"] > 0 and b.flush_stats()["rotation_passes"] == 0
    assert np.abs(x - y).max() < 1e-12


def test_ops_of_both_kinds(gpu):
    """Ops that a program does not take, between ops that it takes."""
    n = 15
    rng = np.random.default_rng(9)
    parts = [circuit(n, 60, 20 + k, TAKEN + [24, 25, 26]) for k in range(2)]
    parts += [circuit(n, 600, 30 + k) for k in range(2)]
    m = rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2))  # not unitary
    with StateVector(n) as a, StateVector(n) as b:
        b.set_dense(False)
        for sv in (a, b):
            for k, g in enumerate(parts):
                sv.run(g)
                sv.mcz([1, 5, 9])
                sv.mcx([0, 7], 3 + k)
                sv.mcz([2, 4, 6, 8])
                if k == 2:
                    sv.apply_1q(4, m / np.linalg.norm(m))
        x, y = a.amplitudes(), b.amplitudes()
        st = a.flush_stats()
        assert 0 < st["rotation_passes"] < st["passes"]
    assert np.abs(x - y).max() < 1e-12


@pytest.mark.parametrize("n,dtype,mode,most", [(13, "c128", "tiled", 3), (15, "c128", "tiled", 3), (15, "c128", "tiled", 5),
                                               (21, "c64", "tiled", 3), (21, "c64", "fused", 5)])
def test_controlled_zz(gpu, n, dtype, mode, most):
    """ZZ under up to three controls, which a program takes, and up to five,
    as ops of the C ABI on any qubits, against one kernel per gate."""
    rng = np.random.default_rng(n + len(mode))
    ops = (_lib.MlbOp * 24)()
    for i, o in enumerate(ops):
        t, t2, *c = (int(q) for q in rng.permutation(n)[:2 + i % (most + 1)])
        o.kind, o.target, o.target2, o.cmask = 5, t, t2, sum(1 << q for q in c)
        for j, x in enumerate(np.exp(1j * rng.uniform(-np.pi, np.pi, 2))):
            o.m[2 * j], o.m[2 * j + 1] = x.real, x.imag
    parts = [circuit(n, 20 if mode == "fused" else 140, 60 + n + k, [4, 7, 8, 9, 10]) for k in range(5)]
    with StateVector(n, dtype) as a, StateVector(n) as b:
        a.set_exec_mode(mode)
        b.set_exec_mode("eager")
        for sv in (a, b):
            for k, g in enumerate(parts):
                sv.run(g)
                some = (_lib.MlbOp * 6)(*ops[6 * k:6 * k + 6]) if k < 4 else None
                if some:
                    _lib.check(_lib.load().mlb_apply_ops(sv.handle, some, 6), "mlb_apply_ops")
        x, y = a.amplitudes(), b.amplitudes()
        st = a.flush_stats()
    if most == 3:
        assert st["rotation_passes"] == st["passes"]
    # the whole state's error: a fidelity of 1 - 1e-6 is 1.4e-3 on the fused path
    assert np.linalg.norm(x - y) < {"c128": 1e-12, "c64": 2e-3 if mode == "fused" else 2e-5}[dtype]


@pytest.mark.parametrize("n,dtype,gates,programs", [
    # a few layers: the dense segments' matrices are cheaper than lowering
    (16, "c128", "brickwork 2", 0), (20, "c128", "brickwork 4", 0), (24, "c128", "brickwork 4", 0),
    # many, ZZ layers, QAOA: the matrices cost more
    (20, "c128", "brickwork 20", 1), (20, "c128", "zz 6", 1), (24, "c128", "qaoa 2", 1), (25, "c128", "zz 4", 1),
    # pass by pass: some of either form
    (26, "c128", "brickwork 6", None), (26, "c128", "brickwork 14", None),
    # many controlled phases: the passes that they crowd stay segments
    (16, "c128", "qft 1", None), (20, "c128", "qft 1", None),
    # registers below the programs' reach
    (12, "c128", "brickwork 20", 0), (20, "c64", "brickwork 20", 0),
    # complex64: a short circuit and a long one, and one whose last tile would hold few qubits
    (21, "c64", "qaoa 1", 0), (21, "c64", "brickwork 20", 1), (22, "c64", "brickwork 1", 1)])
def test_form_that_costs_less(gpu, n, dtype, gates, programs):
    """Which form a flush takes, and its state against that of the other
    forms' kernels (one per gate)."""
    kind, depth = gates.split()
    depth = int(depth)
    g = (qaoa_circuit(n, depth, 3) if kind == "qaoa" else qft(n) if kind == "qft" else
         brickwork(n, depth, 3, zz_every=int(kind == "zz")))
    if programs == 0 and n >= 13:  # the ops' own matrices, whatever was pushed forward on the way
        g = np.concatenate([g, circuit(n, 6, n, [4, 7])])
    with StateVector(n, dtype) as a, StateVector(n) as b:
        a.set_exec_mode("tiled")
        b.set_exec_mode("eager")
        for sv in (a, b):
            sv.run(brickwork(n, 1, 1))
            sv.flush()
            sv.run(g)
        x, y = a.amplitudes(), b.amplitudes()
        st = a.flush_stats()
    if programs is None:
        assert 0 < st["rotation_passes"] < st["passes"]
    else:
        assert st["rotation_passes"] == programs * st["passes"]
    assert np.abs(x - y).max() < (1e-12 if dtype == "c128" else 2e-5)
