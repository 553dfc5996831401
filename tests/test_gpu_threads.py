"""Distinct states and problems used from distinct host threads at once: the
kernels whose launches differ in shared memory (Pauli sums, lambda = H psi,
rotation passes), each thread with a different number of strings, qubits or
layers.  Every result is that of the same call made alone, bit for bit (all
sums have a fixed order)."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from moonlab_b200 import StateVector
from moonlab_b200.circuits import brickwork
from moonlab_b200.vqe import HEAProblem

pytestmark = pytest.mark.gpu


def strings(n, count, seed):
    rng = np.random.default_rng(seed)
    x, z = rng.integers(0, 1 << n, (2, count), dtype=np.uint64)
    return x, z, rng.standard_normal(count)


def pauli(n, count, dtype):
    sv = StateVector(n, dtype)
    sv.run(brickwork(n, 3, n))
    args = strings(n, count, n + count)
    return lambda: (sv.expectation_pauli_sum(*args),)


def gradient(n, layers, count, dtype):
    x, z, c = strings(n, count, n + layers)
    prob = HEAProblem(n, layers, c, xmasks=x, zmasks=z, dtype=dtype)
    theta = np.random.default_rng(layers).uniform(-np.pi, np.pi, (2, 2 * n * layers))
    return lambda: prob.evaluate(theta)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_launches_of_different_sizes_at_once(gpu, dtype):
    calls = [pauli(14, 250, dtype), pauli(6, 2, dtype), pauli(13, 1, dtype), gradient(4, 1, 2, dtype),
             gradient(13, 4, 200, dtype), gradient(11, 9, 20, dtype)]
    alone = [f() for f in calls]
    failed = []
    start = threading.Barrier(len(calls))

    def work(f, want):
        start.wait()
        try:
            for _ in range(200):
                for a, b in zip(f(), want):
                    if not np.array_equal(a, b):
                        raise AssertionError("another result than alone")
        except Exception as e:  # noqa: BLE001
            failed.append(repr(e))

    threads = [threading.Thread(target=work, args=p) for p in zip(calls, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
