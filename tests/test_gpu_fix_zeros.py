"""GPU: amplitudes that a circuit leaves exactly zero are exactly zero in the default arithmetic."""
import math

import numpy as np
import pytest

from helpers import apply_gates, free_state, load_state, new_state

pytestmark = pytest.mark.gpu

H, X, Y, Z, RX, RY, RZ, CNOT = range(8)


def _run(n, gates, psi):
    st = new_state(n)
    try:
        load_state(st, psi)
        apply_gates(st, gates, 1)
        return st.numpy()
    finally:
        free_state(st)


def _layers(qubits, layers, kinds, rng):
    gates = []
    for _ in range(layers):
        for q in qubits:
            gates.append((int(rng.choice(kinds)), q, -1, False, float(rng.choice([math.pi / 2, rng.uniform(0, 6)]))))
        for c, t in zip(qubits, qubits[1:]):
            gates.append((CNOT, t, c, False, 0.0))
    return [(k, t, c, o, th if k in (RX, RY, RZ) else 0.0) for k, t, c, o, th in gates]


@pytest.mark.parametrize("n", [12, 13, 15])
@pytest.mark.parametrize("untouched", [1, 2, 3, 4])
def test_qubits_in_a_basis_state(built_lib, n, untouched):
    """Rotations of the other qubits leave the amplitudes of the untouched qubits' other values zero."""
    rng = np.random.default_rng(n + untouched)
    busy = list(range(n - untouched))
    part = rng.standard_normal(1 << len(busy)) + 1j * rng.standard_normal(1 << len(busy))
    psi = np.zeros(1 << n, dtype=np.complex128)
    psi[: len(part)] = part / np.linalg.norm(part)  # the top qubits are 0
    gates = _layers(busy, 3, [RX, RY, RZ, H], rng)
    got = _run(n, gates, psi)
    assert np.count_nonzero(got[len(part):]) == 0
    assert np.count_nonzero(got[: len(part)]) == len(part)


@pytest.mark.parametrize("n", [12, 14])
def test_real_states_stay_real(built_lib, n):
    """RY, H, X, Z and CNOT on real amplitudes: every imaginary part is zero."""
    rng = np.random.default_rng(n)
    psi = rng.standard_normal(1 << n).astype(np.complex128)
    got = _run(n, _layers(list(range(n)), 3, [RY, H, X, Z], rng), psi / np.linalg.norm(psi))
    assert np.count_nonzero(got.imag) == 0
    assert np.count_nonzero(got.real) == 1 << n
