"""GPU: no device memory for the rewritten passes' tables (the library's allocation hook): the
gates run without them."""
import ctypes

import numpy as np
import pytest

from helpers import apply_gates, free_state, load_state, new_state, oracle_forward_any_control, random_state

pytestmark = pytest.mark.gpu

CNOT = 7


@pytest.mark.parametrize("precision,arith,n,eps", [(0, 0, 13, 2.0 ** -53), (0, 1, 13, 2.0 ** -47), (0, 2, 13, 2.0 ** -52),
                                                   (1, 0, 20, 2.0 ** -24)])
def test_forward_without_room_for_its_tables(built_lib, oracle_mod, precision, arith, n, eps):
    from damavand_gb300._lib import check, lib
    from damavand_gb300.workloads import ladder_circuit
    gates = ladder_circuit(n, 3, 1, False)
    psi = random_state(n, np.random.default_rng(n))
    st = new_state(n, precision)
    try:
        check(lib.dmv_state_set_arithmetic(st.handle, arith))
        apply_gates(st, [(CNOT, 1, 0, False, 0.0), (CNOT, 0, 1, False, 0.0)] * 2000, 1)  # the ops' buffer, no tables
        check(lib.dmv_state_synchronize(st.handle))
        load_state(st, psi)
        lib.dmv_debug_fail_allocations(1)
        try:
            apply_gates(st, gates, 1)
        finally:
            lib.dmv_debug_fail_allocations(0)
        got = st.numpy().astype(np.complex128)
    finally:
        free_state(st)
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    assert np.max(np.abs(got - want)) <= 2 * len(gates) * eps * np.max(np.abs(want))


@pytest.mark.parametrize("arith,digits", [(0, 53), (1, 46)])
def test_gradient_without_room_for_its_tables(built_lib, arith, digits):
    """The sweep runs gate by gate instead, from the same states."""
    from damavand_gb300._lib import check, dptr, lib
    from damavand_gb300.workloads import gate_array, ring_ansatz
    n = 12
    gates = ring_ansatz(n, 3, 5)
    w = np.random.default_rng(2).standard_normal(n)

    def gradient(st, gates):
        arr, count = gate_array(gates)
        loss, g = ctypes.c_double(), np.zeros(sum(k in (4, 5, 6) for k, *_ in gates))
        check(lib.dmv_adjoint_gradient(st.handle, arr, count, dptr(w), ctypes.byref(loss), dptr(g)))
        return loss.value, g

    want = new_state(n)
    st = new_state(n)
    try:
        check(lib.dmv_state_set_arithmetic(want.handle, 4))
        loss0, g0 = gradient(want, gates)
        check(lib.dmv_state_set_arithmetic(st.handle, arith))
        apply_gates(st, gates, 1)  # the forward's buffers
        gradient(st, [(5, 0, -1, False, 0.3)])  # the scratch states, and little else
        lib.dmv_debug_fail_allocations(1)
        try:
            loss, g = gradient(st, gates)
        finally:
            lib.dmv_debug_fail_allocations(0)
        again, g2 = gradient(st, gates)
    finally:
        free_state(st)
        free_state(want)
    tol = 4 * len(gates) * 2.0 ** -digits * np.abs(w).sum()
    assert abs(loss - loss0) <= tol and np.max(np.abs(g - g0)) <= tol
    assert abs(again - loss0) <= tol and np.max(np.abs(g2 - g0)) <= tol
