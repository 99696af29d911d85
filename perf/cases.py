"""The work this framework is timed on, and what it has to come out as.

Every case goes through the package's public entry points (``Circuit``,
``circuit_loss``, ``Batch``), on the circuit shapes of
``damavand_gb300.workloads``. A case is a dict of plain values:

  kind        what a user's program does in one pass
    vqe       set the angles, run from |0...0>, read <Z_q>: the inner call of a variational loop
    train     the same through torch.autograd, loss and gradient: one small training step
    forward   run a circuit from |0...0> and leave the state on the GPU
    pipeline  run, probabilities to the host, samples, +-1 observable values: the whole simulator call
    adjoint   loss and the gradient of every angle of a deep ansatz
    readout   <Z_q>, samples and sampled means of a state that is already there
    batch     many small circuits of uneven size in one launch
  n, layers   qubits, circuit layers (batch: the largest qubit count and depth)
  shape       ladder, ring or random (damavand_gb300.workloads)
  precision, arithmetic   the storage type and the complex128 arithmetic

The arithmetics are the default (fp64), the two faster complex128 ones
(fp32x2, tc) and complex64 storage; int64 and fp64-direct are left out: the
default is faster than both and as accurate, so nobody picks them.
"""
import numpy as np
import torch

from damavand_gb300 import workloads as wl
from damavand_gb300.autograd import circuit_loss
from damavand_gb300.batch import Batch
from damavand_gb300.circuit import Circuit


def _case(kind, n, layers=0, shape="ladder", precision="complex128", arithmetic="fp64", **more):
    return {"kind": kind, "n": n, "layers": layers, "shape": shape, "precision": precision,
            "arithmetic": arithmetic, **more}


def listed():
    return [
        # The smallest call: a toy variational loop, all latency and host work.
        {"name": "vqe_4q", **_case("vqe", 4, 2, "ring")},
        # A small training step (forward, loss, backward) of a variational model.
        {"name": "train_10q", **_case("train", 10, 3, "ring")},
        # The simulator's plain use: 20 qubits, 810 gates, probabilities, 1000 samples, observables.
        {"name": "pipeline_20q", **_case("pipeline", 20, 10, samples=1000)},
        # A mid-size circuit without structure, an odd qubit count: few tiles for the chip.
        {"name": "forward_17q_random", **_case("forward", 17, 30, "random")},
        # An ordinary deep circuit in the default arithmetic.
        {"name": "forward_24q", **_case("forward", 24, 10)},
        # The largest: the benchmark's 20-layer circuit, at the most qubits that fit two seconds with room.
        {"name": "forward_28q", **_case("forward", 28, 20)},
        # The same in single precision, where half the memory is wanted.
        {"name": "forward_27q_c64", **_case("forward", 27, 20, precision="complex64")},
        # The two faster complex128 arithmetics.
        {"name": "forward_26q_fp32x2", **_case("forward", 26, 20, arithmetic="fp32x2")},
        {"name": "forward_25q_tc", **_case("forward", 25, 20, arithmetic="tc")},
        # Gradient of a deep hardware-efficient ansatz (1056 angles).
        {"name": "adjoint_22q", **_case("adjoint", 22, 16, "ring")},
        # Reading a large state that is resident.
        {"name": "readout_28q", **_case("readout", 28, samples=1000)},
        # Many uneven circuits, as a parameter study or a data set runs them.
        {"name": "batch_64", **_case("batch", 20, 40, "random", count=64, min_n=10)},
    ]


def draw(rng):
    kind = rng.choice(["vqe", "train", "pipeline", "forward", "forward", "forward", "adjoint", "readout", "batch"])
    shape = rng.choice(["ladder", "ring", "random"])
    if kind == "vqe":
        return _case(kind, rng.randint(2, 14), rng.randint(1, 8), rng.choice(["ladder", "ring"]))
    if kind == "train":
        return _case(kind, rng.randint(3, 14), rng.randint(1, 5), rng.choice(["ladder", "ring"]),
                     arithmetic=rng.choice(["fp64", "fp64", "fp32x2"]))
    if kind == "pipeline":
        return _case(kind, rng.randint(11, 22), rng.randint(2, 12), shape, samples=rng.randint(100, 2000))
    if kind == "forward":
        precision, arithmetic = rng.choice([("complex128", "fp64"), ("complex128", "fp64"), ("complex64", "fp64"),
                                            ("complex128", "fp32x2"), ("complex128", "tc")])
        return _case(kind, rng.randint(13, 28), rng.randint(2, 19), shape, precision, arithmetic)
    if kind == "adjoint":
        return _case(kind, rng.randint(13, 23), rng.randint(2, 16), rng.choice(["ladder", "ring"]),
                     arithmetic=rng.choice(["fp64", "fp64", "fp32x2"]))
    if kind == "readout":
        return _case(kind, rng.randint(10, 28), samples=rng.randint(100, 4000))
    precision, arithmetic = rng.choice([("complex128", "fp64"), ("complex128", "fp64"), ("complex128", "fp32x2"),
                                        ("complex64", "fp64")])
    return _case(kind, rng.randint(12, 20), rng.randint(5, 40), "random", precision, arithmetic,
                 count=rng.randint(8, 64), min_n=rng.randint(4, 11))


# ------------------------------------------------------------------ inputs
def _gates(case, seed):
    n, layers = case["n"], case["layers"]
    if case["shape"] == "ladder":
        return wl.ladder_circuit(n, layers, seed)
    if case["shape"] == "ring":
        return wl.ring_ansatz(n, layers, seed)
    gates = wl.random_circuit(n, layers, np.random.default_rng(seed))
    return gates + [(wl.Z, q, -1, True, 0.0) for q in range(n)]


def _batch_circuits(case, seed):
    # the sizes belong to the case, the gates and angles to the seed
    sizes = np.random.default_rng([case["count"], case["min_n"], case["n"], case["layers"]])
    circuits = []
    for i in range(case["count"]):
        n = int(sizes.integers(case["min_n"], case["n"] + 1))
        depth = int(sizes.integers(max(1, case["layers"] // 8), case["layers"] + 1))
        circuits.append((n, wl.random_circuit(n, depth, np.random.default_rng([seed, i]))))
    return circuits


def _random_state(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    v = torch.randn(2 << n, generator=g, device="cuda", dtype=torch.float64)
    v /= torch.linalg.vector_norm(v)
    return torch.view_as_complex(v.view(-1, 2))


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    if s.kind == "batch":
        s.batch = Batch(_batch_circuits(case, seed), precision=case["precision"], arithmetic=case["arithmetic"])
        s.single = case["precision"] == "complex64"
        return s
    n = case["n"]
    s.circuit = Circuit(n, "gpu", precision=case["precision"], arithmetic=case["arithmetic"])
    if s.kind == "readout":
        for q in range(n):
            s.circuit.add_pauli_z_gate(q, True)
        s.circuit.state().torch().copy_(_random_state(n, seed))
        torch.cuda.synchronize()
    else:
        gates = _gates(case, seed)
        wl.add_to_circuit(s.circuit, gates)
        s.params = wl.parameters(gates)
    s.weights = wl.loss_weights(n, seed + 1)
    if s.kind == "train":
        s.weights = torch.from_numpy(s.weights).cuda()
        s.params = torch.from_numpy(s.params).cuda().requires_grad_()
    if s.kind in ("forward", "adjoint"):
        # a view of the circuit's own memory: whoever holds it has to hold the circuit
        s.amplitudes = s.circuit.state().torch()
        s.amplitudes.circuit = s.circuit
    if s.kind in ("pipeline", "readout"):
        s.samples = case["samples"]
        s.uniforms = np.random.default_rng(seed + 2).random(s.samples)
        s.seed = seed
    return s


def run(s):
    if s.kind == "batch":
        s.batch.run()
        z = np.concatenate(s.batch.expect_z())
        # complex64 circuits: the values are accurate to single precision
        return z.astype(np.float32) if s.single else z
    c = s.circuit
    if s.kind == "vqe":
        c.set_parameters(s.params)
        c.reset_amplitudes()
        c.forward()
        return c.expectation_z()
    if s.kind == "train":
        s.params.grad = None
        loss = circuit_loss(c, s.params, s.weights)
        loss.backward()
        return loss.detach(), s.params.grad
    if s.kind == "forward":
        c.reset_amplitudes()
        c.forward()
        return s.amplitudes
    if s.kind == "pipeline":
        c.reset_amplitudes()
        c.forward()
        p = c.probabilities()
        samples = c.sample_array(s.samples, uniforms=s.uniforms)
        return p, samples.astype(np.int64), np.asarray(c.extract_expectation_values(samples))
    if s.kind == "adjoint":
        return *c.adjoint_gradient(s.weights), s.amplitudes  # the circuit keeps the forward state
    z = c.expectation_z()
    samples = c.sample_array(s.samples, uniforms=s.uniforms)
    return z, samples.astype(np.int64), c.sample_expectation_values(1 << 17, seed=s.seed)


# ------------------------------------------------------------------ the least it takes
def _count_runs(gates):
    """Single-qubit unitaries after joining neighbours on one qubit (X and CNOT only move amplitudes)."""
    runs, open_on = 0, set()
    for kind, target, control, obs, _ in gates:
        if obs:
            continue
        if kind == wl.CNOT:
            open_on -= {target, control}
        elif kind != wl.X and target not in open_on:
            open_on.add(target)
            runs += 1
    return runs


def work(case):
    """Bytes: the state written once (read once by a readout), results to the host. Flops: 14 per
    amplitude and joined 2x2 unitary; a gradient applies each twice more (the state and its adjoint)
    and takes 4 per amplitude and angle."""
    n, kind = case["n"], case["kind"]
    amps, size = 1 << n, 8 if case["precision"] == "complex64" else 16
    if kind == "readout":
        return {"bytes": amps * size, "flops": 3 * amps}
    if kind == "batch":
        circuits = _batch_circuits(case, 1)
        return {"bytes": sum(size << m for m, _ in circuits),
                "flops": sum((14 * _count_runs(g)) << m for m, g in circuits)}
    gates = _gates(case, 1)
    flops, angles = 14 * _count_runs(gates) * amps, len(wl.parameters(gates))
    if kind == "pipeline":
        return {"bytes": amps * (size + 8), "flops": flops}
    if kind in ("train", "adjoint"):
        return {"bytes": amps * size, "flops": 3 * flops + 4 * angles * amps}
    return {"bytes": amps * size, "flops": flops}


# ------------------------------------------------------------------ plain 64-bit values
def _matrix(kind, theta):
    """The 2x2 of a gate, in the widest type numpy has here."""
    t = np.longdouble(theta) / 2
    c, s = np.cos(t), np.sin(t)
    h = 1 / np.sqrt(np.longdouble(2))
    m = {wl.H: [[h, h], [h, -h]], wl.X: [[0, 1], [1, 0]], wl.Y: [[0, -1j], [1j, 0]], wl.Z: [[1, 0], [0, -1]],
         wl.RX: [[c, -1j * s], [-1j * s, c]], wl.RY: [[c, -s], [s, c]],
         wl.RZ: [[c - 1j * s, 0], [0, c + 1j * s]]}[kind]
    return np.array(m, dtype=np.clongdouble)


def _apply(v, q, m):
    w = v.view(-1, 2, 1 << q)
    m = m.astype(np.complex128)
    a, b = w[:, 0], w[:, 1]
    new = complex(m[0, 0]) * a
    new.add_(b, alpha=complex(m[0, 1]))
    b.mul_(complex(m[1, 1])).add_(a, alpha=complex(m[1, 0]))
    a.copy_(new)


def _cnot(v, control, target):
    lo, hi = min(control, target), max(control, target)
    w = v.view(-1, 2, 1 << (hi - lo - 1), 2, 1 << lo)
    a, b = (w[:, 1, :, 0], w[:, 1, :, 1]) if control == hi else (w[:, 0, :, 1], w[:, 1, :, 1])
    t = a.clone()
    a.copy_(b)
    b.copy_(t)


def _exact_state(n, gates):
    v = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    v[0] = 1
    open_on = {}
    for kind, target, control, obs, theta in gates:
        if obs:
            continue
        if kind != wl.CNOT:
            m = _matrix(kind, theta)
            open_on[target] = m @ open_on[target] if target in open_on else m
            continue
        for q in (control, target):
            if q in open_on:
                _apply(v, q, open_on.pop(q))
        _cnot(v, control, target)
    for q, m in open_on.items():
        _apply(v, q, m)
    return v


def _exact_z(v, n):
    p = v.real.square() + v.imag.square()
    # the qubit axis kept and the others summed, from the top down: the rest of p only halves
    z = []
    for q in range(n - 1, -1, -1):
        half = p.view(2, 1 << q)
        z.append(half[0].sum() - half[1].sum())
        p = half[0] + half[1]
    return torch.stack(z[::-1])


def _exact_gradient(n, gates, weights):
    """The reverse sweep gate by gate: dL/dtheta = Im <lambda| P |psi> for exp(-i theta P / 2)."""
    psi = _exact_state(n, gates)
    z = _exact_z(psi, n).cpu().numpy()
    diag = torch.zeros(1, dtype=torch.float64, device="cuda")
    for w in weights:  # qubit 0 is the fastest index
        diag = torch.cat([diag + float(w), diag - float(w)])
    lam = psi * diag
    grads = []
    for kind, target, control, obs, theta in reversed(gates):
        if obs:
            continue
        if kind == wl.CNOT:
            _cnot(psi, control, target)
            _cnot(lam, control, target)
            continue
        if kind in wl.PARAMETRISED:
            a, b = psi.view(-1, 2, 1 << target), lam.view(-1, 2, 1 << target)
            ar, br = torch.view_as_real(a), torch.view_as_real(b)
            if kind == wl.RX:  # Im(conj(l0) a1 + conj(l1) a0)
                g = (br[:, 0, :, 0] * ar[:, 1, :, 1] - br[:, 0, :, 1] * ar[:, 1, :, 0]
                     + br[:, 1, :, 0] * ar[:, 0, :, 1] - br[:, 1, :, 1] * ar[:, 0, :, 0]).sum()
            elif kind == wl.RY:  # Re(conj(l1) a0 - conj(l0) a1)
                g = ((br[:, 1] * ar[:, 0]).sum() - (br[:, 0] * ar[:, 1]).sum())
            else:  # Im(conj(l0) a0 - conj(l1) a1)
                g = (br[:, 0, :, 0] * ar[:, 0, :, 1] - br[:, 0, :, 1] * ar[:, 0, :, 0]
                     - br[:, 1, :, 0] * ar[:, 1, :, 1] + br[:, 1, :, 1] * ar[:, 1, :, 0]).sum()
            grads.append(g)
        m = _matrix(kind, theta).conj().T
        _apply(psi, target, m)
        _apply(lam, target, m)
    g = torch.stack(grads[::-1]).cpu().numpy() if grads else np.zeros(0)
    return float(np.dot(np.asarray(weights), z)), g


def exact(case, seed):
    n, kind = case["n"], case["kind"]
    if kind == "batch":
        return np.concatenate([_exact_z(_exact_state(m, g), m).cpu().numpy() for m, g in _batch_circuits(case, seed)])
    if kind == "readout":
        return _exact_z(_random_state(n, seed), n), None, None
    gates = _gates(case, seed)
    weights = wl.loss_weights(n, seed + 1)
    if kind in ("train", "adjoint"):
        loss, grads = _exact_gradient(n, gates, weights)
        if kind == "train":
            return torch.tensor(loss, dtype=torch.float64), grads
        return loss, grads, _exact_state(n, gates)
    v = _exact_state(n, gates)
    if kind == "vqe":
        return _exact_z(v, n).cpu().numpy()
    if kind == "pipeline":
        return v.real.square().add_(v.imag.square()).cpu().numpy(), None, None
    return v
