"""The Gram matrix behind HEAProblem.geometry (FP64 tensor-core tiles of
32 x 32 states, 16 amplitudes a step) against numpy, where the number of
states (parameters + 1) and their length meet or miss a tile.

Tolerance: the states differ from numpy's by at most a few roundings per
rotation, and a Gram entry of unit vectors by as many again and one rounding
per doubling of its sum: 16 (P + n) 2^-52 bounds both sides' products."""
from __future__ import annotations

import numpy as np
import pytest

from moonlab_b200.vqe import HEAProblem

pytestmark = pytest.mark.gpu


def states(n, layers, theta):
    """psi and the P shifted states psi(theta + pi e_i): RY, RZ on every
    qubit, then CNOT(q, q + 1), each layer."""
    out = []
    for shift in range(-1, len(theta)):
        th = theta.copy()
        if shift >= 0:
            th[shift] += np.pi
        psi = np.zeros(1 << n, dtype=complex)
        psi[0] = 1
        for layer in range(layers):
            for q in range(n):
                p = 2 * (layer * n + q)
                c, s = np.cos(th[p] / 2), np.sin(th[p] / 2)
                v = psi.reshape(-1, 2, 1 << q)
                a, b = v[:, 0] * c - v[:, 1] * s, v[:, 0] * s + v[:, 1] * c
                z = np.exp(0.5j * th[p + 1])
                psi = np.stack((a / z, b * z), 1).reshape(-1)
            x = np.arange(1 << n)
            for q in range(n - 1):
                x = x ^ ((x >> q & 1) << (q + 1))
            new = np.empty_like(psi)
            new[x] = psi
            psi = new
        out.append(psi)
    return np.array(out)


@pytest.mark.parametrize("n,layers", [(2, 1), (3, 5), (4, 4), (5, 3), (4, 8), (8, 2), (11, 3)])
def test_gram_tiles(gpu, n, layers):
    P = 2 * n * layers
    theta = np.random.default_rng(n * 100 + layers).uniform(-np.pi, np.pi, P)
    prob = HEAProblem(n, layers, [1.0], xmasks=[0], zmasks=[1], dtype="c128")
    try:
        metric, curvature = prob.geometry(theta)
    finally:
        prob.close()
    S = states(n, layers, theta)
    G = S.conj() @ S.T
    Q = G[1:, 1:] / 4 - np.outer(G[0, 1:].conj(), G[0, 1:]) / 4
    tol = 16 * (P + n) * 2.0**-52
    assert np.abs(metric - Q.real).max() <= tol
    off = -2 * (Q.imag - np.diag(np.diag(Q.imag)))
    assert np.abs(curvature - off).max() <= tol
