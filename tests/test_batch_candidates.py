"""CPU: what the batch autotuner times. It starts with the configuration that there is, so that
it cannot leave a batch slower than it found it, and a batch whose passes are rewritten tries
its own number of low qubits and no tiles that have no fixed-point pass."""
import ctypes

import pytest


def _candidates(lib, precision, arithmetic, max_qubits):
    out, count = (ctypes.c_int32 * 192)(), ctypes.c_int32()
    assert lib.dmv_debug_batch_candidates(precision, arithmetic, max_qubits, 64, out, ctypes.byref(count)) == 0
    return [tuple(out[3 * i:3 * i + 3]) for i in range(count.value)]


@pytest.mark.parametrize("precision,arithmetic,max_qubits", [(0, 0, 20), (0, 0, 12), (0, 0, 11), (0, 1, 20), (0, 2, 8),
                                                             (0, 4, 20), (1, 0, 20)])
def test_candidates(built_lib, precision, arithmetic, max_qubits):
    rewritten = precision == 0 and arithmetic == 0
    c = _candidates(built_lib.lib, precision, arithmetic, max_qubits)
    assert len(set(c)) == len(c)
    assert c[0][:2] == ((12, 4) if rewritten else (12, 6))  # a new batch's own
    assert max(k for k, _, _ in c) == (13 if precision else 12)
    if rewritten:
        assert {low for _, low, _ in c} == {4, 5, 6}
        assert (min(k for k, _, _ in c) == 12) == (max_qubits >= 12)
    else:
        assert {(k, low) for k, low, _ in c} >= {(k, low) for k in (10, 11, 12) for low in (5, 6)}
