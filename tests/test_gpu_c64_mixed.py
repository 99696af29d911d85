"""GPU: complex64 plans that mix rewritten passes with passes of 2x2 matrices: the state's scale
between them, a last pass of either kind, passes whose rotation factors leave the range, and
passes of more ops than a kernel holds in shared memory.

Tolerance: each output is rounded to 2^-24 of itself once per gate, the rotations' and tables'
entries likewise.
"""
import numpy as np
import pytest

from helpers import apply_gates, free_state, load_state, new_state, oracle_forward_any_control, random_state
from test_fix_plan import ROT, _passes, _words

pytestmark = pytest.mark.gpu

RX, RY, CNOT = 4, 5, 7


def _check(built_lib, oracle_mod, n, gates, seed=1):
    psi = random_state(n, np.random.default_rng(seed))
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    st = new_state(n, 1)
    try:
        load_state(st, psi)
        apply_gates(st, gates, 1)
        got = st.numpy().astype(np.complex128)
    finally:
        free_state(st)
    tol = 2 * len(gates) * 2.0 ** -24
    assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))
    assert abs(np.linalg.norm(got) - 1) <= tol
    return list(_passes(_words(built_lib.lib, n, gates, 2)))


@pytest.mark.parametrize("n", [20, 21])
def test_controlled_rotations_among_the_passes(built_lib, oracle_mod, n):
    from damavand_gb300.workloads import ladder_circuit, random_circuit
    rng = np.random.default_rng(n)
    gates = ladder_circuit(n, 3, 1, False) + random_circuit(n, 6, rng, controlled_rotations=True)
    gates += ladder_circuit(n, 3, 2, False)
    passes = _check(built_lib, oracle_mod, n, gates)
    taken = [p["taken"] for p in passes]
    assert True in taken and False in taken


@pytest.mark.parametrize("n", [20, 21])
def test_last_pass_of_2x2_matrices(built_lib, oracle_mod, n):
    from damavand_gb300.workloads import ladder_circuit
    gates = ladder_circuit(n, 3, 1, False)
    for q in range(n):  # after everything else on every qubit
        gates.append((RY, (q + 1) % n, q, False, 0.3 + 0.1 * q))
    passes = _check(built_lib, oracle_mod, n, gates)
    assert any(p["taken"] for p in passes) and not passes[-1]["taken"]


def _narrow(layers, angle):
    """Gates on qubits 0 to 11: one window."""
    gates = []
    for i in range(layers):
        gates += [(RX if i % 2 else RY, q, -1, False, angle(q)) for q in range(12)]
        gates += [(CNOT, (q + 1) % 12, q, False, 0.0) for q in range(12)]
    return gates


@pytest.mark.parametrize("n,layers", [(20, 20), (20, 40), (21, 20)])
def test_factors_out_of_range(built_lib, oracle_mod, n, layers):
    """Layers of turns by 1.5 in one window: after 20 the product of the factors is far below 2^-40,
    after 40 it would pass 2^-200 and the rewrite folds it back in between."""
    from damavand_gb300.workloads import ladder_circuit
    gates = ladder_circuit(n, 2, 1, False) + _narrow(layers, lambda q: 1.5) + ladder_circuit(n, 2, 2, False)
    passes = _check(built_lib, oracle_mod, n, gates)
    scales = [p["scale"] for p in passes if p["taken"]]
    assert 2.0 ** -40 < max(scales)
    assert min(scales) < 2.0 ** -40 if layers == 20 else not all(p["taken"] for p in passes)


@pytest.mark.parametrize("n", [20, 21])
def test_more_ops_than_shared_memory_holds(built_lib, oracle_mod, n):
    gates = _narrow(30, lambda q: 0.02 + 0.001 * q)
    passes = _check(built_lib, oracle_mod, n, gates)
    assert max(len(p["fix"]) for p in passes) > 256
    assert min(p["scale"] for p in passes) > 2.0 ** -40
    assert sum(np.count_nonzero(p["fix"][:, 0] == ROT) for p in passes) == 30 * 12
