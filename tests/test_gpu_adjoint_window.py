"""GPU: the windowed adjoint sweep (runs of gates on one qubit measured once)
against the sweep gate by gate (DMV_ARITH_FP64_DIRECT keeps it).

Tolerance: a gradient is a sum of products of two states of norms 1 and at
most sum |w|, each rounded once per gate in FP64 (2^-53 of its size).
"""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H, X, Y, Z, RX, RY, RZ, CNOT = range(8)


def _gradient(n, gates, weights, arithmetic):
    from damavand_gb300 import Circuit
    from damavand_gb300.workloads import add_to_circuit
    c = Circuit(n, "gpu", arithmetic=arithmetic)
    add_to_circuit(c, gates)
    return c.adjoint_gradient(weights)


def _mixed(n, rng, layers):
    """Runs of every make: rotations next to fixed gates, lone RZ, angles whose product is
    diagonal, an exchange or the identity, CNOTs in both directions."""
    gates = []
    for _ in range(layers):
        for q in range(n):
            kinds = rng.permutation([RX, RY, RZ, H, X, Y, Z])[: int(rng.integers(1, 6))]
            for k in kinds:
                theta = float(rng.choice([0.0, math.pi, math.pi / 2, 2 * math.pi, rng.uniform(0, 6.28)]))
                gates.append((int(k), q, -1, False, theta if k in (RX, RY, RZ) else 0.0))
        for _ in range(n // 2):
            c, t = rng.permutation(n)[:2]
            gates.append((CNOT, int(t), int(c), False, 0.0))
    return gates


@pytest.mark.parametrize("arithmetic", ["fp64", "fp32x2"])
@pytest.mark.parametrize("n", [2, 3, 10, 11, 12, 13, 16])
def test_windows_equal_gate_by_gate(built_lib, n, arithmetic):
    from damavand_gb300.workloads import ring_ansatz
    rng = np.random.default_rng(70 + n)
    w = rng.standard_normal(n)
    for gates in (_mixed(n, rng, 3), ring_ansatz(n, 5, n)):
        loss, g = _gradient(n, gates, w, arithmetic)
        loss0, g0 = _gradient(n, gates, w, "fp64-direct")
        digits = 53 if arithmetic == "fp64" else 46  # FP32 pairs: 48 bits, two of them for the sums
        tol = 4 * len(gates) * 2.0 ** -digits * np.abs(w).sum()
        assert abs(loss - loss0) <= tol
        assert np.max(np.abs(g - g0)) <= tol


def test_more_measurements_than_one_launch_holds(built_lib):
    """An 11-qubit state is one window: 110 runs, in three launches."""
    from damavand_gb300.workloads import ring_ansatz
    n = 11
    gates = ring_ansatz(n, 10, 1)
    w = np.random.default_rng(1).standard_normal(n)
    _, g = _gradient(n, gates, w, "fp64")
    _, g0 = _gradient(n, gates, w, "fp64-direct")
    assert np.max(np.abs(g - g0)) <= 4 * len(gates) * 2.0 ** -53 * np.abs(w).sum()
