"""Plans and parameter blocks that the library keeps between launches of a
pass: more parameter sets of one circuit than a plan keeps, in turn and again,
in both precisions, from one thread and from several on streams of their own,
match the FP64 oracle (1e-12 / 1e-5, as every state-vector run)."""
import threading

import numpy as np
import pytest
import torch

from oracle import sv as osv

N_QUBITS = 12


def _circuit(values):
    from quict_b200.core import CX, H, Circuit, Rx, Ry, Rz, Rzz, U3
    rng, val = np.random.default_rng(3), np.random.default_rng(values)
    c = Circuit(N_QUBITS)
    for q in range(N_QUBITS):
        H | c(q)
    for _ in range(40):
        a, b = (int(q) for q in rng.choice(N_QUBITS, 2, replace=False))
        t = [float(x) for x in val.uniform(0, 2 * np.pi, 4)]
        Rx(t[0]) | c(a)
        U3(t[1], t[2], t[3]) | c(b)
        CX | c([a, b])
        Rzz(t[0]) | c([b, a])
        Ry(t[1]) | c(a)
        Rz(t[2]) | c(b)
    return c


def _want(c):
    return osv.run([(np.asarray(g.matrix, dtype=np.complex128), list(g.cargs) + list(g.targs)) for g in c.gates],
                   N_QUBITS)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["double", "single"])
def test_many_parameter_sets_in_turn(precision):
    from quict_b200.simulation import StateVectorSimulator
    tol = 1e-12 if precision == "double" else 1e-5
    circuits = [_circuit(v) for v in range(11)]
    want = [_want(c) for c in circuits]
    sims = [StateVectorSimulator("GPU", precision) for _ in circuits]
    for _ in range(3):
        for sim, c, w in zip(sims, circuits, want):
            assert np.abs(sim.run(c).get() - w).max() <= tol


@pytest.mark.gpu
def test_threads_on_their_own_streams():
    from quict_b200.simulation import StateVectorSimulator
    circuits = [_circuit(v) for v in range(4)]
    want = [_want(c) for c in circuits]
    worst = [0.0] * 4

    def work(i):
        sim = StateVectorSimulator("GPU", "double")
        with torch.cuda.stream(torch.cuda.Stream()):
            for r in range(6):
                j = (i + r) % 4
                worst[i] = max(worst[i], float(np.abs(sim.run(circuits[j]).get() - want[j]).max()))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert max(worst) <= 1e-12
