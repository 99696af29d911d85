"""GPU: dmv_last_upload_bytes counts the ops of the register-phase passes."""
import ctypes

import pytest

from helpers import apply_gates, free_state, new_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,layers", [(20, 3), (21, 8)])
def test_a_rewritten_complex64_plan_reports_its_ops(built_lib, n, layers):
    """Such a plan uploads nothing but its tables' terms and 48 bytes for every rotation, table and phase."""
    from damavand_gb300._lib import check, lib
    from damavand_gb300.workloads import ladder_circuit
    st = new_state(n, 1)
    try:
        apply_gates(st, ladder_circuit(n, layers, 1), 1)
        total, terms = ctypes.c_int64(), ctypes.c_int64()
        check(lib.dmv_last_upload_bytes(st.handle, ctypes.byref(total), ctypes.byref(terms)))
        check(lib.dmv_state_synchronize(st.handle))
    finally:
        free_state(st)
    assert terms.value > 0
    assert total.value - terms.value >= layers * n * 48  # a rotation per qubit and layer
