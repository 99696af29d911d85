"""GPU: tiles in which one amplitude outweighs the others by far keep FP64's accuracy.

Tolerance: an FP64 rotation rounds each component x of its tile once, by at most 2^-54 |x|'s
power of two, so with independent roundings the state's error after `count` rotations has a
norm of about sqrt(count / 3) 2^-54; four times that is allowed. Rounding every component by
2^-58 of the tile's largest one would leave sqrt(8192 count / 3) 2^-58, six times as much as
the first figure. A factor common to all amplitudes is left out of the comparison: the
rotations' scale factors, rounded once each, are all alike here and scale the state by
360 * 3.7e-17.
"""
import numpy as np
import pytest

from helpers import apply_gates, free_state, load_state, new_state

pytestmark = pytest.mark.gpu

RY, CNOT = 5, 7


def _apply(v, gates):
    """The gates on a real state, in the widest type numpy has."""
    for kind, t, c, _, theta in gates:
        if kind == CNOT:
            i = np.arange(v.size)
            v = v[np.where((i >> c) & 1, i ^ (1 << t), i)]
        else:
            w = v.reshape(-1, 2, 1 << t)
            cs, sn = np.cos(np.longdouble(theta) / 2), np.sin(np.longdouble(theta) / 2)
            a, b = w[:, 0].copy(), w[:, 1].copy()
            w[:, 0] = cs * a - sn * b
            w[:, 1] = sn * a + cs * b
    return v


@pytest.mark.parametrize("n", [12, 13])
@pytest.mark.parametrize("arith", [0, 1])
def test_small_rotations_of_a_dominated_state(built_lib, n, arith):
    from damavand_gb300._lib import check, lib
    rng = np.random.default_rng(n)
    gates = []
    for _ in range(30):  # exchanges leave |0...0> where it is
        gates += [(RY, q, -1, False, float(rng.choice([-1, 1]) * 2.0 ** -9)) for q in range(n)]
        gates += [(CNOT, (q + 1) % n, q, False, 0.0) for q in range(n)]
    psi = rng.uniform(1.0, 2.0, 1 << n) * rng.choice([-1, 1], 1 << n) * 2.0 ** -10
    psi[0] = 0.99
    want = _apply(psi.astype(np.longdouble), gates)
    st = new_state(n)
    try:
        check(lib.dmv_state_set_arithmetic(st.handle, arith))
        load_state(st, psi.astype(np.complex128))
        apply_gates(st, gates, 1)
        got = st.numpy()
    finally:
        free_state(st)
    assert np.count_nonzero(got.imag) == 0
    diff = got.real - want
    diff -= want * (np.sum(diff * want) / np.sum(want * want))
    err = float(np.sqrt(np.sum(diff * diff)))
    unit = 2.0 ** -54 if arith == 0 else 2.0 ** -48
    assert err <= 4 * np.sqrt(len(gates) / 2 / 3) * unit
