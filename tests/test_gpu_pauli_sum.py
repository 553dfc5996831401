"""mlb_expect_pauli_sum (kernels_pauli.cu) against numpy: registers below
three qubits (their own kernel), of exactly a tile and one qubit either side
of it, strings as wide as the register, repeated and empty X masks, more
strings than a pass holds, and few strings on small states (smaller tiles).  Tolerance: a sum of T 2^n products in another
order, 1e-15 T relative to the sum of |c_k| for a normalised state, plus
complex64's own products (exact in FP64)."""
from __future__ import annotations

import numpy as np
import pytest

from moonlab_b200 import StateVector

pytestmark = pytest.mark.gpu


def parity(v):
    v = v.copy()
    for s in (32, 16, 8, 4, 2, 1):
        v ^= v >> np.uint64(s)
    return (v & np.uint64(1)).astype(np.float64)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n,terms", [(1, 6), (2, 9), (3, 20), (5, 700), (11, 40), (12, 300), (13, 33), (14, 50), (17, 30),
                                     (7, 1), (10, 2), (13, 2), (16, 3), (18, 1), (19, 4)])
def test_pauli_sum_matches_numpy(gpu, n, terms, dtype):
    rng = np.random.default_rng(100 * n + terms)
    a = rng.standard_normal(2 << n).view(np.complex128)
    a = (a / np.linalg.norm(a)).astype(np.complex128 if dtype == "c128" else np.complex64)
    x = rng.integers(0, 1 << n, terms, dtype=np.uint64)
    z = rng.integers(0, 1 << n, terms, dtype=np.uint64)
    x[::4] = 0
    x[1::4] = np.uint64(1) << rng.integers(0, n, len(x[1::4])).astype(np.uint64)
    c = rng.standard_normal(terms)
    sv = StateVector(n, dtype=dtype)
    sv.set_amplitudes(a)
    w = a.astype(np.complex128)
    idx = np.arange(1 << n, dtype=np.uint64)
    want = 0.0
    for k in range(terms):
        ny = bin(int(x[k] & z[k])).count("1") % 4
        v = (1j ** ny) * np.vdot(w[idx ^ x[k]], (1 - 2 * parity(idx & z[k])) * w)
        want += c[k] * v.real
        if k < 3:
            assert abs(sv.expectation_pauli(int(x[k]), int(z[k])) - v.real) < 1e-15 * terms + 1e-14
    got = sv.expectation_pauli_sum(x, z, c)
    assert abs(got - want) < 1e-15 * terms * np.abs(c).sum() + 1e-14
    assert sv.expectation_pauli_sum([], [], []) == 0.0


@pytest.mark.parametrize("c", [1e308, np.inf, -np.inf, 1e-310, np.nan])
def test_extreme_coefficients(gpu, c):
    """A coefficient multiplies its string's value, whatever its size: no
    partial sum of it overflows, underflows or meets an infinity of the other
    sign."""
    n = 5
    rng = np.random.default_rng(3)
    a = rng.standard_normal(2 << n).view(np.complex128)
    a /= np.linalg.norm(a)
    with StateVector(n) as sv:
        sv.set_amplitudes(a)
        x, z = [0, 9, 21], [6, 2, 21]
        v = [sv.expectation_pauli(p, q) for p, q in zip(x, z)]
        got = sv.expectation_pauli_sum(x, z, [0.5, c, -2.0])
        want = 0.5 * v[0] + c * v[1] + -2.0 * v[2]
        tol = 16 * 2.0**-52 * (0.5 * abs(v[0]) + abs(c) * abs(v[1]) + 2 * abs(v[2]))  # sums of 32 products
        assert got == want or (np.isnan(want) and np.isnan(got)) or abs(got - want) <= tol
        assert sv.expectation_pauli_sum(x[1:2], z[1:2], [c]) == c * v[1] or np.isnan(c)
