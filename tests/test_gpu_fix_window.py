"""GPU: the fixed-point window passes (the default complex128 arithmetic on
tiles whose amplitudes are of one size) and the tiles that leave them: wide
ranges, zeros, non-finite values, amplitudes that outgrow the integers.

Tolerance: an output is rounded to 2^-57 of its tile's largest component, in
FP64 to 2^-53 of itself, so `count` roundings stay below count * 2^-53 of the
largest amplitude; the gates' own matrices are rounded the same way.
"""
import math

import numpy as np
import pytest

from helpers import apply_gates, free_state, load_state, new_state, oracle_forward_any_control, random_state

pytestmark = pytest.mark.gpu


def _run(n, gates, psi, arith=0):
    from damavand_gb300._lib import check, lib
    st = new_state(n)
    try:
        check(lib.dmv_state_set_arithmetic(st.handle, arith))
        load_state(st, psi)
        apply_gates(st, gates, 1)
        return st.numpy()
    finally:
        free_state(st)


def _tol(gates):
    return 2 * len(gates) * 2.0 ** -53


@pytest.mark.parametrize("shape", ["ladder", "ring", "random"])
@pytest.mark.parametrize("n", [12, 13, 14, 18])
def test_shapes_from_a_dense_state(built_lib, oracle_mod, n, shape):
    from damavand_gb300 import workloads as wl
    rng = np.random.default_rng(n)
    gates = {"ladder": lambda: wl.ladder_circuit(n, 4, 1, False), "ring": lambda: wl.ring_ansatz(n, 4, 2),
             "random": lambda: wl.random_circuit(n, 12, rng, controlled_rotations=True)}[shape]()
    psi = random_state(n, rng)
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    got = _run(n, gates, psi)
    assert np.max(np.abs(got - want)) <= _tol(gates) * np.max(np.abs(want))


@pytest.mark.parametrize("angle", [0.0, 1e-9, 2 * math.atan(0.5), 2 * math.atan(0.5) + 1e-9, math.pi / 2,
                                   math.pi / 2 + 1e-12, math.pi, 3.0, 2 * math.pi])
def test_rotation_multiplier_edges(built_lib, oracle_mod, angle):
    """tan(angle / 2) at 0, next to 0, at 1/2 (the two multiplier forms), at 1 and beyond (the exchange)."""
    n = 13
    gates = [(5, q, -1, False, angle) for q in range(n)] + [(4, q, -1, False, -angle) for q in range(n)]
    psi = random_state(n, np.random.default_rng(3))
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    got = _run(n, gates, psi)
    assert np.max(np.abs(got - want)) <= _tol(gates) * np.max(np.abs(want))


def test_concentrating_state_outgrows_the_integers(built_lib):
    """Hadamards on the uniform state gather a whole tile in one amplitude, 64 times the largest before."""
    n = 14
    psi = np.full(1 << n, 2.0 ** (-n / 2), dtype=np.complex128)
    gates = [(0, q, -1, False, 0.0) for q in range(n)]
    got = _run(n, gates, psi)
    want = np.zeros(1 << n, dtype=np.complex128)
    want[0] = 1.0
    assert np.max(np.abs(got - want)) <= _tol(gates) * 4


def test_product_state_keeps_its_small_amplitudes(built_lib):
    """Amplitudes of a product state far below the largest keep their relative accuracy (FP64 tiles)."""
    n = 15
    angles = np.random.default_rng(8).uniform(0.05, 0.4, n)
    gates = [(5, q, -1, False, float(a)) for q, a in enumerate(angles)]
    psi = np.zeros(1 << n, dtype=np.complex128)
    psi[0] = 1.0
    want = np.ones(1)
    for a in angles:  # qubit 0 is the fastest index
        want = np.concatenate([want * math.cos(a / 2), want * math.sin(a / 2)])
    got = _run(n, gates, psi)
    assert np.max(np.abs(got - want) / want) <= 8 * n * 2.0 ** -53


def test_non_finite_tile_stays_apart(built_lib, oracle_mod):
    """An infinity spoils its own tile only; the others come out as without it."""
    n = 14
    rng = np.random.default_rng(4)
    gates = [(5, q, -1, False, float(rng.uniform(0, 6))) for q in range(12)]
    psi = random_state(n, rng)
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    bad = psi.copy()
    bad[5] = complex(math.inf, 0.0)
    got = _run(n, gates, bad)
    part = 1 << 12  # the gates act on qubits 0-11
    assert not np.all(np.isfinite(got[:part]))
    assert np.max(np.abs(got[part:] - want[part:])) <= _tol(gates) * np.max(np.abs(want))


@pytest.mark.parametrize("start", ["uniform", "zero", "dense"])
def test_pair_states_off_the_integers(built_lib, oracle_mod, start):
    """FP32-pair states: tiles that leave the fixed point run in pairs (48 bits), next to ones that
    do not, over enough passes that the factors left out are multiplied back in between."""
    from damavand_gb300._lib import ARITH_FP32X2
    from damavand_gb300.workloads import ladder_circuit
    n = 15
    rng = np.random.default_rng(6)
    psi = {"uniform": np.full(1 << n, 2.0 ** (-n / 2), dtype=np.complex128),
           "zero": np.eye(1, 1 << n, dtype=np.complex128)[0], "dense": random_state(n, rng)}[start]
    gates = ladder_circuit(n, 25, 3, False)
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    got = _run(n, gates, psi, ARITH_FP32X2)
    assert np.max(np.abs(got - want)) <= 2 * len(gates) * 2.0 ** -47 * np.max(np.abs(want))


@pytest.mark.parametrize("shape", ["ladder", "ring", "random"])
@pytest.mark.parametrize("n", [12, 13, 17, 20, 21])
def test_complex64_shapes(built_lib, oracle_mod, n, shape):
    """The complex64 passes on the same shapes; each output is rounded to 2^-24 of itself, the
    rotations' and tables' entries likewise."""
    from damavand_gb300 import workloads as wl
    rng = np.random.default_rng(40 + n)
    gates = {"ladder": lambda: wl.ladder_circuit(n, 6, 1, False), "ring": lambda: wl.ring_ansatz(n, 6, 2),
             "random": lambda: wl.random_circuit(n, 12, rng)}[shape]()
    psi = random_state(n, rng)
    want = oracle_forward_any_control(oracle_mod, n, gates, psi)
    st = new_state(n, 1)
    try:
        load_state(st, psi)
        apply_gates(st, gates, 1)
        got = st.numpy().astype(np.complex128)
    finally:
        free_state(st)
    assert np.max(np.abs(got - want)) <= 2 * len(gates) * 2.0 ** -24 * np.max(np.abs(want))
