"""Rotation programs (rotate_plan.h) on the host: lowered as a state lowers
them, run as the kernel runs them (rotate_plan_host.cpp), against the ops
themselves in numpy.  Every form that a program takes: controls and targets
inside and outside the tile, on as many qubits as it accepts.  Tolerance
1e-12 per amplitude of a normalised state, as for the kernels."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from moonlab_b200 import _lib
from tests.test_tile_plan import OP_1Q, OP_DIAG1, OP_PHASE, OP_SWAP, OP_X, OP_ZZ, apply_op

ROOT = Path(__file__).resolve().parent.parent
TILE = 0b1011010111  # 7 of 10 qubits
LIMIT = {OP_1Q: 0, OP_X: 1, OP_SWAP: 0, OP_DIAG1: 2, OP_ZZ: 3, OP_PHASE: 3}  # controls that a program takes


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = tmp_path_factory.mktemp("rot") / "rotate_plan_host.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    f"-I{ROOT}/include", f"-I{ROOT}/moonlab_b200/csrc", "-o", str(out),
                    str(ROOT / "tests" / "rotate_plan_host.cpp")], check=True)
    lib = C.CDLL(str(out))
    lib.host_run.argtypes = [C.c_void_p, C.c_size_t, C.c_int, C.c_uint64, C.c_int, C.c_int, C.c_void_p]
    lib.host_push_forward.argtypes = [C.c_void_p, C.c_size_t, C.c_uint32]
    lib.host_covers.argtypes = [C.c_void_p]
    return lib


def unitary(rng):
    q, r = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))
    return (q * (np.diag(r) / np.abs(np.diag(r)))).reshape(-1)


def make(kind, target, target2=-1, controls=(), m=()):
    o = _lib.MlbOp()
    o.kind, o.target, o.target2 = kind, target, target2
    o.cmask = sum(1 << int(c) for c in controls)
    for i, x in enumerate(m):
        o.m[2 * i], o.m[2 * i + 1] = x.real, x.imag
    return o


def random_op(rng, n, tile, kind, controls):
    inside = [q for q in range(n) if tile >> q & 1]
    moved = kind in (OP_1Q, OP_X, OP_SWAP)
    t = int(rng.choice(inside if moved else range(n)))
    rest = [q for q in (inside if kind == OP_SWAP else range(n)) if q != t]
    pick = [int(q) for q in rng.permutation(rest)[:1 + controls]]
    phases = np.exp(1j * rng.uniform(-np.pi, np.pi, 2))
    if kind in (OP_SWAP, OP_ZZ):
        return make(kind, t, pick[0], pick[1:], () if kind == OP_SWAP else phases)
    if kind == OP_PHASE:
        return make(kind, t, -1, [t] + pick[1:controls], phases[:1])
    return make(kind, t, -1, pick[1:], unitary(rng) if kind == OP_1Q else () if kind == OP_X else phases)


def run_both(host, n, tile, ops, dtype, seed, push=0):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    a /= np.linalg.norm(a)
    want, got = a.copy(), a.copy()
    arr = (_lib.MlbOp * len(ops))(*ops)
    for o in ops:
        apply_op(want, n, o)
    assert host.host_run(arr, len(ops), n, tile, dtype, push, got.ctypes.data) == 0
    return want, got


@pytest.mark.parametrize("dtype", [_lib.MLB_C128, _lib.MLB_C64])
@pytest.mark.parametrize("kind,controls", [(k, c) for k, most in LIMIT.items() for c in range(most + 1)
                                           if not (k == OP_PHASE and c == 0)])
def test_each_form(host, kind, controls, dtype):
    rng = np.random.default_rng(17 * kind + controls)
    for trial in range(6):  # the form between rotations, so that nothing merges it away
        ops = []
        for _ in range(8):
            ops += [random_op(rng, 10, TILE, OP_1Q, 0) for _ in range(3)]
            ops += [random_op(rng, 10, TILE, kind, controls) for _ in range(2)]
        assert host.host_covers(C.byref(ops[-1]))
        want, got = run_both(host, 10, TILE, ops, dtype, trial)
        # complex64 programs hold their tangents in 32 bits
        assert np.abs(got - want).max() < (1e-12 if dtype == _lib.MLB_C128 else 2e-6)


@pytest.mark.parametrize("kind", list(LIMIT))
def test_more_controls_are_left_to_the_other_path(host, kind):
    rng = np.random.default_rng(kind)
    for controls in range(LIMIT[kind] + 1, 6):
        o = random_op(rng, 12, (1 << 12) - 1, kind, controls)
        assert not host.host_covers(C.byref(o))


@pytest.mark.parametrize("push", [0, 1])
@pytest.mark.parametrize("seed", range(12))
def test_mixed_ops(host, seed, push):
    rng = np.random.default_rng(900 + seed)
    n = int(rng.integers(6, 12))
    tile = 3 | sum(1 << int(q) for q in rng.choice(np.arange(2, n), min(n - 2, 4), replace=False))
    ops = []
    for _ in range(int(rng.integers(1, 50))):
        kind = int(rng.choice(list(LIMIT)))
        ops.append(random_op(rng, n, tile, kind, int(rng.integers(kind == OP_PHASE, LIMIT[kind] + 1))))
    want, got = run_both(host, n, tile, ops, _lib.MLB_C128, seed, push)
    assert np.abs(got - want).max() < 1e-12


@pytest.mark.parametrize("e", [5e-324, 1e-323, 1e-320, 1e-300, 1e-160, 1e-100, 1e-17, 0.0])
def test_push_forward_keeps_tiny_entries_unitary(host, e):
    """A unitary whose off-diagonal is almost nothing, a controlled phase, then
    a Hadamard: the pushed matrices stay unitary and the product the same, to
    eight roundings of 2^-53."""
    h = np.sqrt(0.5)
    ops = [make(OP_1Q, 0, -1, (), [1, complex(-e, e), complex(e, e), 1]),
           make(OP_PHASE, 0, -1, (0, 1), [np.exp(0.7j)]), make(OP_1Q, 0, -1, (), [h, h, h, -h])]
    want = run_ops(ops)
    arr = (_lib.MlbOp * 3)(*ops)
    host.host_push_forward(arr, 3, 2)
    for o in (arr[0], arr[2]):
        u = (np.ctypeslib.as_array(o.m)[0:8:2] + 1j * np.ctypeslib.as_array(o.m)[1:8:2]).reshape(2, 2)
        assert np.abs(u.conj().T @ u - np.eye(2)).max() < 1e-15
    assert np.abs(run_ops(arr) - want).max() < 1e-15


def run_ops(ops, n=2):
    out = np.eye(1 << n, dtype=complex)
    for col in out:
        for o in ops:
            apply_op(col, n, o)
    return out


def brickwork_ops(rng, n, depth):
    """Layers of a general one-qubit unitary on every qubit, then CNOTs."""
    ops = []
    for k in range(depth):
        for q in range(n):
            x, y, z = np.exp(0.5j * rng.uniform(-np.pi, np.pi, 3))  # RZ RY RX as their product
            c, s = x.real, x.imag
            u = np.array([[c, -1j * s], [-1j * s, c]])
            u = np.array([[y.real, -y.imag], [y.imag, y.real]]) @ u
            u = np.diag([1 / z, z]) @ u
            ops.append(make(OP_1Q, q, -1, (), u.reshape(-1)))
        for q in range(k & 1, n - 1, 2):
            ops.append(make(OP_X, q + 1, -1, (q,)))
    return ops


def test_pushing_forward_costs_no_accuracy(host):
    """Programs of pushed matrices are as close to the ops, in 80-bit
    arithmetic, as programs of the ops' own matrices (1.42e-15 and 1.48e-15
    here; with products rounded to doubles 1.63e-15)."""
    n, errs = 10, []
    for seed in range(12):
        ops = brickwork_ops(np.random.default_rng(seed), n, 14)
        exact = np.zeros(1 << n, np.clongdouble)
        exact[0] = 1
        idx = np.arange(1 << n)
        for o in ops:
            if o.kind == OP_X:
                exact = exact[idx ^ ((idx & o.cmask != 0).astype(int) << o.target)]
                continue
            m = (np.ctypeslib.as_array(o.m)[0:8:2] + 1j * np.ctypeslib.as_array(o.m)[1:8:2]).astype(np.clongdouble)
            w = exact.reshape(-1, 2, 1 << o.target)
            w[:] = np.stack((m[0] * w[:, 0] + m[1] * w[:, 1], m[2] * w[:, 0] + m[3] * w[:, 1]), 1)
        arr = (_lib.MlbOp * len(ops))(*ops)
        for push in (0, 1):
            got = np.zeros(1 << n, complex)
            got[0] = 1
            assert host.host_run(arr, len(ops), n, (1 << n) - 1, _lib.MLB_C128, push, got.ctypes.data) == 0
            errs.append(float(np.linalg.norm((got - exact).astype(complex))))
    own, pushed = np.sqrt(np.mean(np.square(errs).reshape(-1, 2), 0))
    assert pushed < 1.03 * own, (pushed, own)


def test_tables_keep_the_norm(host):
    """A table of one scale for all 16 entries rounds them all alike: what its
    rounding takes from the norm is given back by the next one.  Layers of RY
    and CNOT: the norm's drift, rms of 24 circuits, is 1.4e-16, 3.4e-16
    without the correction; half as much again as the first is allowed."""
    n, drift = 10, []
    for seed in range(24):
        rng = np.random.default_rng(seed)
        ops = []
        for k in range(14):
            for q in range(n):
                t = rng.uniform(-np.pi, np.pi)
                ops.append(make(OP_1Q, q, -1, (), np.array([np.cos(t), -np.sin(t), np.sin(t), np.cos(t)]) + 0j))
            ops += [make(OP_X, q + 1, -1, (q,)) for q in range(k & 1, n - 1, 2)]
        a = np.zeros(1 << n, complex)
        a[0] = 1
        arr = (_lib.MlbOp * len(ops))(*ops)
        assert host.host_run(arr, len(ops), n, (1 << n) - 1, _lib.MLB_C128, 1, a.ctypes.data) == 0
        drift.append(float(np.linalg.norm(a.astype(np.clongdouble)) - 1))
    assert np.sqrt(np.mean(np.square(drift))) < 2.2e-16
