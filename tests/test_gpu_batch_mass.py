"""GPU: a batch's <Z> where circuits on both sides of the line between the shared mass pass and one
of their own (24 qubits) stand next to one another, in any order, and where all are on one side."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,arithmetic", [("complex128", "fp64"), ("complex128", "fp32x2"), ("complex64", "fp64")])
@pytest.mark.parametrize("sizes", [(24, 3, 23, 25, 12), (5, 24, 1), (25,), (23, 20)])
def test_every_circuit_reads_its_own_columns(built_lib, oracle_mod, precision, arithmetic, sizes):
    from damavand_gb300.batch import Batch
    RY, RX, CNOT = 5, 4, 7
    circuits = []
    for n in sizes:
        gates = [(RY, 0, -1, False, 0.3 + n), (RX, n // 2, -1, False, 0.5 + n), (RY, n - 1, -1, False, 0.7 + n)]
        circuits.append((n, gates + ([(CNOT, n // 2, n - 1, False, 0.0), (CNOT, 0, n - 1, False, 0.0)] if n > 1 else [])))
    b = Batch(circuits, precision, arithmetic)
    for _ in range(2):
        b.run()
    tol = 1e-12 if precision == "complex128" else 1e-5
    for (n, gates), z in zip(circuits, b.expect_z()):
        want = oracle_mod.expect_z(oracle_mod.measure(oracle_mod.forward(n, gates)))
        assert np.max(np.abs(z - want)) <= tol
