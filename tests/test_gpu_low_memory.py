"""GPU: no device memory for the rewritten passes' tables (the library's allocation hook): the
gates run without them."""
import math

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
