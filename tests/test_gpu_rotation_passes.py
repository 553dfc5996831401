"""The rotation passes of the hardware-efficient ansatz (kernels_adjoint.cu)
where they can go wrong: registers below three qubits (padded), of exactly a
tile and one qubit either side of it, angles at which a half-angle's sine or
cosine vanishes (the tangent and cotangent forms), several checkpoint
segments, and the index order restored after the tensor-core forward sweep.
Energies and gradients against the CPU oracle's adjoint, 1e-11 (sums of 2^n
products of order one in another order: 2^13 ulp is 2e-12); complex64 within
1e-4 of complex128, relative to the largest gradient."""
from __future__ import annotations

import numpy as np
import pytest

from moonlab_b200.vqe import HEAProblem
from tests.test_gpu_adjoint import port_energy_grad, random_problem

pytestmark = pytest.mark.gpu


def angles(n, layers, seed):
    """Random angles, a third of them multiples of pi / 2."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(-np.pi, np.pi, 2 * n * layers)
    special = rng.random(p.size) < 1 / 3
    p[special] = rng.integers(-4, 5, special.sum()) * (np.pi / 2)
    return p


@pytest.mark.parametrize("n,layers", [(1, 3), (2, 4), (3, 7), (4, 1), (10, 3), (11, 4), (12, 5), (13, 2)])
def test_rotation_passes_match_the_oracle(gpu, n, layers):
    paulis, coeffs, _, hf = random_problem(n, layers, 2 * n + 1, 900 + n)
    params = np.stack([angles(n, layers, 10 * n + k) for k in range(3)])
    prob = HEAProblem(n, layers, coeffs, paulis=paulis, hf_reference=hf)
    for mode in ("always", "never"):
        prob.set_checkpointing(mode)
        E, G = prob.evaluate(params)
        for k, p in enumerate(params):
            e_ref, g_ref = port_energy_grad(n, layers, hf, paulis, coeffs, p)
            assert abs(E[k] - e_ref) < 1e-11
            assert np.abs(G[k] - g_ref).max() < 1e-11


@pytest.mark.parametrize("n,layers", [(3, 2), (12, 4), (13, 5), (14, 10), (17, 3)])
@pytest.mark.parametrize("mode", ["always", "never"])
def test_complex64_rotation_passes(gpu, n, layers, mode):
    paulis, coeffs, _, hf = random_problem(n, layers, 2 * n, 700 + n)
    params = np.stack([angles(n, layers, 20 * n + k) for k in range(3)])
    E, G = HEAProblem(n, layers, coeffs, paulis=paulis, hf_reference=hf).evaluate(params)
    prob = HEAProblem(n, layers, coeffs, paulis=paulis, hf_reference=hf, dtype="c64")
    prob.set_checkpointing(mode)
    for forward in ("auto", "off"):
        prob.set_fused_forward(forward)
        e, g = prob.evaluate(params)
        assert np.abs(e - E).max() < 1e-4 * max(1.0, np.abs(E).max())
        assert np.abs(g - G).max() < 1e-4 * max(1.0, np.abs(G).max())


@pytest.mark.parametrize("n,layers", [(6, 120), (12, 60)])
def test_deep_problems_sum_gradients_in_groups(gpu, n, layers):
    """More gradient slots than are summed at once (512: 256 rotations)."""
    paulis, coeffs, _, hf = random_problem(n, layers, n, 40 + n)
    p = angles(n, layers, n)
    E, G = HEAProblem(n, layers, coeffs, paulis=paulis, hf_reference=hf).evaluate(p)
    e_ref, g_ref = port_energy_grad(n, layers, hf, paulis, coeffs, p)
    assert abs(E[0] - e_ref) < 1e-11
    assert np.abs(G[0] - g_ref).max() < 1e-11


def test_memory_of_a_deep_narrow_problem(gpu):
    """The partials stay small beside the states, whatever the depth (all
    passes' at once took 59 MB here, beside 67 MB of psi and lambda)."""
    import torch
    n, layers, batch = 18, 200, 8
    prob = HEAProblem(n, layers, [1.0, 0.5], xmasks=[0, 3], zmasks=[5, 0])
    prob.set_checkpointing("never")
    params = np.stack([angles(n, layers, k) for k in range(batch)])
    prob.evaluate(params[:1])  # modules and small tables
    free = torch.cuda.mem_get_info()[0]
    prob.evaluate(params)
    pair = 2 * 16 * batch << n
    assert free - torch.cuda.mem_get_info()[0] < pair * (1 + 1 / 16) + (8 << 20)


def test_norms_do_not_drift(gpu):
    """|psi|^2 (the energy of the identity) after 8 layers on 12 qubits.  An
    entry of a segment's table is rounded once and multiplies an eighth of the
    amplitudes: about 40 roundings of up to 2^-53 a component, at random
    2 sqrt(40) 2^-53 / sqrt(3) = 8.1e-16 rms; half as much again is allowed.
    Entries multiplied up in double gave 1.7e-15."""
    n, layers = 12, 8
    params = np.random.default_rng(1).uniform(-np.pi, np.pi, (64, 2 * n * layers))
    E = HEAProblem(n, layers, [1.0], xmasks=[0], zmasks=[0]).evaluate(params)[0]
    assert np.sqrt(np.mean((E - 1) ** 2)) < 1.2e-15
