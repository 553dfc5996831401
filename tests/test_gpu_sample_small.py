"""Sampling and measurement of states of one chunk (12 qubits) and around it,
where the phases that only several chunks need are left out and few elements
are added in order, against the oracle's sequential sums, bit for bit:
states with leading, trailing and only zeros, amplitudes of very different
size, uniforms on the running sums themselves."""
from __future__ import annotations

import numpy as np
import pytest

from moonlab_b200 import StateVector
from oracle import bindings as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 9, 10, 11, 12, 13, 14])
def test_outcomes_are_the_oracles(gpu, n, dtype):
    rng = np.random.default_rng(n)
    dim = 1 << n
    base = rng.standard_normal(2 * dim).view(np.complex128)
    states = [base, base * (np.arange(dim) >= dim // 2), base * (np.arange(dim) < dim // 2 + 1),
              base * np.exp(rng.uniform(-60, 0, dim)), np.zeros(dim, complex)]
    for a in states:
        norm = np.linalg.norm(a)
        a = (a / norm if norm else a).astype(np.complex128 if dtype == "c128" else np.complex64)
        wide = a.astype(np.complex128)
        h = np.hypot(wide.real, wide.imag)
        sums = np.cumsum(h * h)
        u = np.concatenate([rng.random(200), sums[rng.integers(0, dim, 40)], [0.0, 1.0, np.nextafter(1.0, 0)]])
        with StateVector(n, dtype) as sv:
            sv.set_amplitudes(a)
            assert np.array_equal(sv.sample(u), B.port_sample(wide, u))
