"""CPU: the register-phase form of the window passes (build_fix_pass), run here the way the kernels
run it (slots, register and thread bits, tables in their phase's order, exchanges as changes of the
slot map), gives on random tiles what the ops it was made from give, for every pass of the plans
that the kernels get. No GPU.

Tolerance: the arithmetic here is FP64 on both sides, one rounding of 2^-53 per op and component
on either (complex64 plans hold multipliers rounded to 2^-25).
"""
import ctypes

import numpy as np
import pytest

PHASE, XOR, ROT, TABLE, FETCH, GRAD, END = range(7)
COMPLEMENT, SHIFT = 4, 8
GLOBAL_BIT = 20


def _words(lib, n, gates, form):
    from damavand_gb300.workloads import gate_array
    arr, count = gate_array(gates)
    used = ctypes.c_int64()
    words = np.zeros(1 << 21, dtype=np.int64)
    rc = lib.dmv_debug_fix_plan(ctypes.cast(arr, ctypes.c_void_p), count, n, form, words.size,
                                words.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), ctypes.byref(used))
    assert rc == 0, lib.dmv_last_error_string()
    return words[:used.value]


def _passes(words):
    pos = 0

    def take(n):
        nonlocal pos
        pos += n
        return words[pos - n:pos]

    while pos < len(words):
        low, nh = take(2)
        high = take(nh)
        nops, taken, nfix, ntab, nterm, shifts = take(6)
        scale = take(1).view(np.float64)[0]
        ops = take(13 * nops).reshape(-1, 13)
        grads = take(2 * take(1)[0]).reshape(-1, 2)
        yield {"low": int(low), "high": high, "taken": bool(taken), "shifts": int(shifts), "scale": scale, "ops": ops,
               "grads": grads, "fix": take(12 * nfix).reshape(-1, 12), "tables": take(6 * ntab).reshape(-1, 6),
               "terms": take(2 * nterm).reshape(-1, 2)}


def _pauli_sums(psi, lam, t):
    """Im <lam| P |psi> for X, Y, Z on bit t."""
    p, q = psi.reshape(-1, 2, 1 << t), lam.reshape(-1, 2, 1 << t).conj()
    x = (q[:, 0] * p[:, 1] + q[:, 1] * p[:, 0]).sum()
    y = (-1j * q[:, 0] * p[:, 1] + 1j * q[:, 1] * p[:, 0]).sum()
    z = (q[:, 0] * p[:, 0] - q[:, 1] * p[:, 1]).sum()
    return np.array([x.imag, y.imag, z.imag])


def _plain(states, ops, base, sums):
    """The pass's own ops; sums[run]: the measurements before a run's op."""
    l = np.arange(states.shape[1])
    for op in ops:
        t, ctrl, kind, run, generator = (int(v) for v in op[:5])
        m = op[5:].view(np.float64).view(np.complex128).reshape(2, 2)
        if generator:
            sums[run] = _pauli_sums(states[0], states[1], t)
        if kind == 2 and not (base >> ctrl) & 1:
            continue
        zero = (l >> t) & 1 == 0
        if kind == 1:
            zero &= (l >> ctrl) & 1 == 1
        i0 = l[zero]
        a, b = states[:, i0], states[:, i0 | 1 << t]
        states[:, i0], states[:, i0 | 1 << t] = m[0, 0] * a + m[0, 1] * b, m[1, 0] * a + m[1, 1] * b
    return states


def _slot(l, single):
    return l ^ ((l >> 4 ^ l >> 8) & 15) if single else l ^ ((l >> 3 ^ l >> 6 ^ l >> 9) & 7)


def _phases(ps, table, gsel, ph):
    """Entries of a table's slice in the order of a phase: [thread, register]."""
    _, c, first, num, k, _ = (int(v) for v in table)
    tpos, rpos = int(ph[7]) & 0xFFFFFFFF, int(ph[8]) & 0xFFFFFFFF
    i = np.arange(1 << k)
    l = np.zeros_like(i)
    for b in range(8):
        l |= (i >> b & 1) << (tpos >> 4 * b & 15)
    for b in range(k - 8):
        l |= (i >> (8 + b) & 1) << (rpos >> 4 * b & 15)
    at = l | gsel << GLOBAL_BIT
    turn = np.full(1 << k, c, dtype=np.int64)
    for mask, t in ps["terms"][first:first + num]:
        parity = at & mask
        for s in (16, 8, 4, 2, 1):
            parity = parity ^ parity >> s
        turn = turn + np.where(parity & 1, t, 0)  # wraps modulo a turn
    return np.exp(1j * turn.astype(np.float64) * (np.pi * 2.0 ** -63)).reshape(k_regs(k), 256).T


def k_regs(k):
    return 1 << (k - 8)


def _register_phases(states, ps, base, k, single, sums):
    """What the kernels do with the pass's register-phase ops."""
    regs = k_regs(k)
    mem = np.empty_like(states)
    mem[:, _slot(np.arange(1 << k), single)] = states
    cx, at, r, ph, fetched = 0, None, None, None, None
    tid, reg = np.arange(256)[:, None], np.arange(regs)[None, :]
    for f in ps["fix"]:
        kind, a = int(f[0]), [int(v) for v in f[1:]]
        if kind == FETCH:
            fetched = a[:5]
        elif kind == XOR:
            if (base >> a[0]) & 1:
                cx ^= a[1]
        elif kind == TABLE:
            assert single or fetched == a[:5]
            fetched = None
            table = next(t for t in ps["tables"] if t[0] == a[0])
            assert a[1] == table[5]
            gsel = sum(((base >> a[2 + j]) & 1) << j for j in range(a[1]))
            r = r * _phases(ps, table, gsel, ph)
        elif kind == ROT:
            bit = 1 << (a[0] & 3)
            if single:
                w = float(np.array([a[1]], dtype=np.int64).astype(np.int32).view(np.float32)[0])
            else:
                w = a[1] * 2.0 ** -32 + a[2] * 2.0 ** -64
                w = 1 - w if a[0] & COMPLEMENT else w
            j0 = np.flatnonzero(np.arange(regs) & bit == 0)
            x, y = r[..., j0], r[..., j0 | bit]
            r[..., j0], r[..., j0 | bit] = x - w * y, y + w * x
            if a[0] & SHIFT and not single:
                r = r / 2
        elif kind == GRAD:
            bit = a[0] & 3
            flat = [v.reshape(-1) for v in r]  # [thread, register]: the register's bits are the low ones
            square = np.array([a[3] & 0xFFFFFFFF | a[4] << 32], dtype=np.int64).view(np.float64)[0]
            sums.append((a[1], _pauli_sums(flat[0], flat[1], bit), square))
        else:
            if r is not None:
                mem[:, at] = r
            images = [v >> s & 0xFFFF for v in a[:6] for s in (0, 16)]
            cx ^= a[8]
            at = np.full((256, regs), cx)
            for b in range(k - 8):
                at ^= np.where(reg >> b & 1, images[b], 0)
            for b in range(8):
                at ^= np.where(tid >> b & 1, images[4 + b], 0)
            assert len(np.unique(at)) == at.size and at.max() < 1 << k
            r = mem[:, at]
            ph = f
    return r.transpose(0, 2, 1).reshape(states.shape)  # amplitude tid + 256 j


def _check(lib, n, gates, form, seed):
    rng = np.random.default_rng(seed)
    k, single = (11 if form == 1 else 12), form == 2
    seen = taken = 0
    for ps in _passes(_words(lib, n, gates, form)):
        seen += 1
        if not ps["taken"]:
            continue
        taken += 1
        local = (1 << ps["low"]) - 1 | sum(1 << int(q) for q in ps["high"])
        base = int(rng.integers(0, 1 << n)) & ~local
        states = rng.standard_normal((2, 1 << k)) + 1j * rng.standard_normal((2, 1 << k))
        states /= np.linalg.norm(states, axis=1)[:, None]
        want_sums, got_sums = {}, []
        want = _plain(states.copy(), ps["ops"], base, want_sums)
        got = _register_phases(states, ps, base, k, single, got_sums)
        factor = ps["scale"] * (1 if single else 2.0 ** ps["shifts"])
        eps = 2.0 ** -25 if single else 2.0 ** -53
        tol = 4 * len(ps["fix"]) * eps
        assert np.linalg.norm(got * factor - want) <= tol
        assert len(got_sums) == len(ps["grads"]) == sum(1 for op in ps["ops"] if op[4])
        halved = 0
        order = [f for f in ps["fix"] if f[0] in (ROT, GRAD)]
        shifts = {}
        for f in order:  # halvings of both states before each measurement
            if f[0] == GRAD:
                shifts[int(f[2])] = halved
            elif f[1] & SHIFT:
                halved += 1
        frames = {int(run): int(frame) for run, frame in ps["grads"]}
        for run, (x, y, z), square in got_sums:
            s = square * 4.0 ** shifts[run]
            ang = frames[run] * np.pi * 2.0 ** -63
            v = s * np.array([np.cos(ang) * x + np.sin(ang) * y, -np.sin(ang) * x + np.cos(ang) * y, z])
            assert np.max(np.abs(v - want_sums[run])) <= tol
    return seen, taken


def _circuit(shape, n, layers, seed, **more):
    from damavand_gb300 import workloads as wl
    if shape == "random":
        return wl.random_circuit(n, layers, np.random.default_rng(seed), **more)
    return {"ladder": wl.ladder_circuit, "ring": wl.ring_ansatz}[shape](n, layers, seed)


@pytest.mark.parametrize("shape,layers", [("ladder", 6), ("ring", 5), ("random", 25)])
@pytest.mark.parametrize("form,n", [(0, 12), (0, 13), (0, 16), (0, 24), (0, 30), (1, 11), (1, 12), (1, 15), (1, 22),
                                    (2, 20), (2, 21), (2, 27)])
def test_register_phases(built_lib, form, n, shape, layers):
    seen, taken = _check(built_lib.lib, n, _circuit(shape, n, layers, n), form, n)
    assert seen == taken > 0


@pytest.mark.parametrize("form,n", [(0, 14), (1, 13), (2, 20)])
def test_passes_with_other_ops_are_left_out(built_lib, form, n):
    """Controlled rotations in some windows: those passes are declined, the others are right."""
    gates = _circuit("ladder", n, 4, 1)
    c, t = n - 1, n - 2
    gates += [(5, t, c, False, 0.7)] + _circuit("ring", n, 3, 2)
    seen, taken = _check(built_lib.lib, n, gates, form, 5)
    assert 0 < taken < seen
