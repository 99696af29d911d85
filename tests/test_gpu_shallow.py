"""GPU: passes of so few ops that the FP64 window kernel is the faster one (shallow_pass), on both
sides of the line, on dense states, from |0...0> and with a tile that is not finite.

Tolerance: an output is rounded to 2^-53 of the largest amplitude, or less, once per op; the
gates' own matrices are rounded the same way.
"""
import ctypes
import math

import numpy as np
import pytest

from helpers import apply_gates, free_state, load_state, new_state, oracle_forward_any_control, random_state

pytestmark = pytest.mark.gpu

H, X, Y, Z, RX, RY, RZ, CNOT = range(8)
OP = 224  # bytes of an op; a fixed-point one has 48


def _gates(kind, count, n):
    q = [n - 1, n - 2, 0, n - 3, 1, 2, 3, n - 4, n - 5, n - 6]
    if kind == "cnot":
        return [(CNOT, q[(i + 1) % 10], q[i], False, 0.0) for i in range(count)]
    if kind == "mixed":  # a rotation, a table, then exchanges
        return [(RY, q[0], -1, False, 0.4), (RZ, q[1], -1, False, 0.7)] + _gates("cnot", count, n)
    return [({"ry": RY, "rz": RZ}[kind], q[i], -1, False, 0.3 + 0.1 * i) for i in range(count)]


def _run(st, gates):
    from damavand_gb300._lib import check, lib
    apply_gates(st, gates, 1)
    total, terms = ctypes.c_int64(), ctypes.c_int64()
    check(lib.dmv_last_upload_bytes(st.handle, ctypes.byref(total), ctypes.byref(terms)))
    return st.numpy(), (total.value - terms.value) % OP == 0


@pytest.mark.parametrize("kind,count,shallow", [("ry", 2, True), ("ry", 3, False), ("rz", 2, True), ("rz", 10, True),
                                                ("cnot", 2, True), ("cnot", 8, True), ("cnot", 9, False),
                                                ("mixed", 1, True), ("mixed", 2, False)])
@pytest.mark.parametrize("n", [12, 13, 20])
def test_either_side_of_the_line(built_lib, oracle_mod, n, kind, count, shallow):
    gates = _gates(kind, count, n)
    dense = random_state(n, np.random.default_rng(n))
    zero = np.eye(1, 1 << n, dtype=np.complex128)[0]
    for psi in (dense, zero):
        st = new_state(n)
        try:
            load_state(st, psi)
            got, fp64 = _run(st, gates)
        finally:
            free_state(st)
        assert fp64 == shallow
        want = oracle_forward_any_control(oracle_mod, n, gates, psi)
        assert np.max(np.abs(got - want)) <= 2 * len(gates) * 2.0 ** -53 * np.max(np.abs(want))


def test_non_finite_tile_stays_apart(built_lib, oracle_mod):
    n = 14
    psi = random_state(n, np.random.default_rng(4))
    gates = [(RY, 3, -1, False, 0.4), (RY, 9, -1, False, 0.5)]
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    bad = psi.copy()
    bad[5] = complex(math.inf, 0.0)
    bad[1 << 12:2 << 12] = 0.0  # and a tile of zeros beside it
    st = new_state(n)
    try:
        load_state(st, bad)
        got, fp64 = _run(st, gates)
    finally:
        free_state(st)
    part = 1 << 12  # a window of qubits 0-11
    assert fp64 and not np.all(np.isfinite(got[:part]))
    assert np.count_nonzero(got[part:2 * part]) == 0
    assert np.max(np.abs(got[2 * part:] - want[2 * part:])) <= 4 * 2.0 ** -53 * np.max(np.abs(want))


@pytest.mark.parametrize("n,count,as_is", [(20, 4, True), (20, 8, True), (20, 9, False), (21, 8, True), (22, 4, True),
                                           (22, 5, False), (24, 4, True)])
@pytest.mark.parametrize("kind", ["h", "rz"])
def test_complex64_lists_of_few_gates(built_lib, oracle_mod, n, count, as_is, kind):
    """On both sides of the line between a rewritten pass (it has tables) and the gates as they are."""
    q = [n - 1, 0, n - 2, 7, n - 3, 1, n // 2, 2, 3]
    gates = [(H if kind == "h" else RZ, q[i], -1, False, 0.0 if kind == "h" else 0.3 + 0.1 * i) for i in range(count)]
    if count > 4:
        gates = gates[:-1] + [(CNOT, q[1], q[0], False, 0.0)]
    psi = random_state(n, np.random.default_rng(n))
    st = new_state(n, 1)
    try:
        load_state(st, psi)
        from damavand_gb300._lib import check, lib
        apply_gates(st, gates, 1)
        total, terms = ctypes.c_int64(), ctypes.c_int64()
        check(lib.dmv_last_upload_bytes(st.handle, ctypes.byref(total), ctypes.byref(terms)))
        got = st.numpy().astype(np.complex128)
    finally:
        free_state(st)
    assert (terms.value == 0) == as_is
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    assert np.max(np.abs(got - want)) <= 2 * len(gates) * 2.0 ** -24 * np.max(np.abs(want))
