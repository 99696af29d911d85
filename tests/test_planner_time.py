"""CPU: the window search's time on a long gate list does not depend on qubits that no gate touches."""
import ctypes
import time

import numpy as np


def _plan_seconds(lib, n, gates):
    from damavand_gb300.workloads import gate_array
    arr, count = gate_array(gates)
    best = float("inf")
    for _ in range(5):
        start = time.perf_counter()
        assert lib.dmv_plan_describe(n, 0, arr, count, 1, 0, None, None, None, None) == 0
        best = min(best, time.perf_counter() - start)
    return best


def test_idle_qubits_do_not_lengthen_the_search(built_lib):
    """80,000 gates on 16 of 30 qubits against the same on 16 of 16, where 5 windows are to choose
    from instead of 19: 2.6 times as long. Scans that a qubit without gates keeps from ending
    early walk the whole list for every window, 9.5 times as long and more with the list."""
    from damavand_gb300.workloads import random_circuit
    gates = random_circuit(16, 4000, np.random.default_rng(3))
    idle, full = (_plan_seconds(built_lib.lib, n, gates) for n in (30, 16))
    assert idle <= 5 * full
