"""One run queues every kernel of a circuit: a complex64 pass that splits into
two launches, run once while nothing is compiled, runs as generated kernels
only as soon as the compiler is done (asynchronous mode); both runs match the
FP64 oracle (1e-5, as every state-vector run)."""
import numpy as np
import pytest

import generated
from oracle import sv as osv

N_QUBITS = 11


def _circuit():
    """128 two-qubit unitaries on neighbours, round and round: a stage of four
    register bits runs three of them, so one launch does not take them all."""
    from quict_b200.core import Circuit, Unitary
    from quict_b200.workloads import haar_unitary
    rng = np.random.default_rng(20)
    c = Circuit(N_QUBITS)
    for a in range(128):
        Unitary(haar_unitary(rng, 4)) | c([a % N_QUBITS, (a + 1) % N_QUBITS])
    return c


def test_the_pass_splits():
    assert len(generated.sources(_circuit(), N_QUBITS, 8, (11, 5, 0))) == 2


@pytest.mark.gpu
def test_one_run_queues_every_launch():
    from quict_b200 import _native as N
    from quict_b200.simulation import StateVectorSimulator
    c = _circuit()
    want = osv.run([(np.asarray(g.matrix, dtype=np.complex128), list(g.cargs) + list(g.targs)) for g in c.gates], N_QUBITS)
    old = N.jit_set_mode(N.QS_JIT_ASYNC)
    try:
        N.jit_wait(900)
        before = N.jit_stats()
        sim = StateVectorSimulator("GPU", "single", tile_bits=11, low_bits=5, merge_bits=0)
        assert np.abs(sim.run(c).get() - want).max() <= 1e-5
        N.jit_wait(900)
        first = N.jit_stats()
        assert first["compiled"] + first["failed"] - before["compiled"] - before["failed"] == 2
        assert np.abs(sim.run(c).get() - want).max() <= 1e-5
        second = N.jit_stats()
        assert second["compiled_launches"] - first["compiled_launches"] == 2
        assert second["generic_launches_while_pending"] == first["generic_launches_while_pending"]
    finally:
        N.jit_set_mode(old)
