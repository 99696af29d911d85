"""GPU: the windowed adjoint sweep's measurement sums at the largest they can be."""
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


def test_measurement_of_a_full_tile(built_lib):
    """The sweep starts on an eighth of a tile's amplitudes, all with |re| = |im| just below a
    power of two. Three rotations spread them over the tile (the integers shrink below the
    bound under which a tile is shifted up), then the stored norm grows to twice the shifted
    one before a qubit is measured that both states hold in the same direction: 2^64 in the
    units of the sums."""
    n = 12
    a, (b0, b1, b2), (c0, c1), m, rest, g = [0, 1, 2], (3, 4, 5), (6, 7), 8, [9, 10], 11
    small = 2 * math.atan(0.02)
    large = 2 * math.atan(0.99)
    half = math.pi / 2 - 2e-5
    # what is there before the last gates: |+> (a, b2, rest), (|0> + i|1>) / sqrt 2 and its conjugate
    gates = [(RZ, g, -1, False, -math.pi / 2), (RY, g, -1, False, 2 * math.acos((1 - 0.002) / math.sqrt(2)))]
    gates += [(H, q, -1, False, 0.0) for q in a + [b2] + rest]
    gates += [(RX, q, -1, False, -math.pi / 2) for q in (b0, c0, m)]
    gates += [(RX, q, -1, False, math.pi / 2) for q in (b1, c1)]
    # exchanges that leave it, so that a qubit's gates before and after are two runs
    gates += [(CNOT, rest[0], q, False, 0.0) for q in a + [b0, b1, b2, c0, c1, m]]
    # the last gates in reverse: spread a, raise the factor over sqrt 2, bring it back up, measure m
    last = [(RY, q, -1, False, -half) for q in a]
    last += [(RY, b0, -1, False, small), (RY, b1, -1, False, small), (RY, b2, -1, False, 1e-9)]
    last += [(RY, c0, -1, False, large), (RY, c1, -1, False, large), (RY, m, -1, False, 1e-9)]
    gates += last[::-1]
    w = np.zeros(n)
    w[m] = 1.0
    loss, grads = _gradient(n, gates, w, "fp64")
    loss0, grads0 = _gradient(n, gates, w, "fp64-direct")
    tol = 4 * len(gates) * 2.0 ** -53
    assert abs(loss - loss0) <= tol
    assert np.max(np.abs(grads - grads0)) <= tol
