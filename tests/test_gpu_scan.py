"""GPU: the sampler's chunk prefixes where they cross from one CTA (4096 chunks of 4096
amplitudes) to several, and the batch's reductions over uneven circuits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12, 13, 23, 24, 25, 26])
def test_uniform_state_samples_exactly(built_lib, n):
    """Dyadic probabilities: every prefix is exact, so sample u is the least i with u <= (i + 1) / 2^n."""
    from damavand_gb300 import Circuit
    c = Circuit(n, "gpu")
    st = c.state().torch()
    st.fill_(2.0 ** (-(n // 2)) if n % 2 == 0 else 2.0 ** (-(n + 1) // 2) * (1 + 1j))  # |amplitude|^2 = 2^-n
    edge = np.array([1, 2, 4095, 4096, 4097, (1 << n) // 2, (1 << n) - 1]) / 2.0 ** n
    u = np.concatenate([edge, np.random.default_rng(n).random(2000)])
    u = u[u < 1.0]
    got = c.sample_array(len(u), uniforms=u)
    want = np.ceil(u * 2.0 ** n).astype(np.int64) - 1
    assert np.array_equal(got.astype(np.int64), want)


@pytest.mark.parametrize("precision", ["complex128", "complex64"])
def test_batch_reductions(built_lib, oracle_mod, precision):
    """Circuits of 1 to 16 qubits, among them ones of no gates: every <Z_q> from its own columns."""
    from damavand_gb300.batch import Batch
    from damavand_gb300.workloads import random_circuit
    rng = np.random.default_rng(12)
    circuits = [(n, random_circuit(n, d, rng)) for n, d in [(1, 3), (16, 5), (2, 0), (12, 4), (11, 6), (13, 2), (5, 9)]]
    b = Batch(circuits, precision)
    b.run()
    tol = 1e-12 if precision == "complex128" else 1e-4
    for (n, gates), z in zip(circuits, b.expect_z()):
        want = oracle_mod.expect_z(oracle_mod.measure(oracle_mod.forward(n, gates)))
        assert np.max(np.abs(z - want)) <= tol
