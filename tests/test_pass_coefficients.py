"""Coefficients of generated passes whose matrices had factors taken out
(csrc/passgen.cu), on the CPU (generated.py): with phases next to an axis (2 pi,
4 pi, 8 pi, 1e-15) and general ones, repeated a hundred times, the passes are
as accurate as applying the gates one by one in complex128, against the same
matrices in 64 significand bits.

Bound: the passes round each coefficient once and each product and sum once, as
the gates do, in another order: twice the gates' error, measured on the same
circuit, plus two units in the last place of an amplitude."""
import numpy as np
import pytest

import generated
from oracle import sv as osv

N_QUBITS = 12


def _circuit(seed, phases):
    from quict_b200.core import CX, Circuit, H, U3
    rng = np.random.default_rng(seed)
    c = Circuit(N_QUBITS)
    for q in range(N_QUBITS):
        H | c(q)
    for _ in range(100):
        U3(float(rng.uniform(0, 6)), float(rng.choice(phases)), float(rng.choice(phases))) | c(int(rng.integers(N_QUBITS)))
        if rng.random() < 0.3:
            CX | c([int(q) for q in rng.choice(N_QUBITS, 2, replace=False)])
    return c


def _extended(gates):
    v = np.zeros(1 << N_QUBITS, dtype=np.clongdouble)
    v[0] = 1
    for m, qs in gates:
        x = np.moveaxis(v.reshape([2] * N_QUBITS), qs, range(len(qs)))
        x = (m.astype(np.clongdouble) @ x.reshape(1 << len(qs), -1)).reshape(x.shape)
        v = np.moveaxis(x, range(len(qs)), qs).reshape(-1)
    return v


@pytest.mark.parametrize("merge", [0, 2])
@pytest.mark.parametrize("phases", [[8 * np.pi, 1e-15, 0.0], [2 * np.pi, 4 * np.pi, 0.0], [3e-16, 2e-16, np.pi / 4],
                                    [0.3, 1.2, 2.9, 5.1]], ids=["8pi", "2pi", "tiny", "general"])
def test_as_accurate_as_the_gates(phases, merge):
    plain, passes = 0.0, 0.0
    for seed in range(4):
        c = _circuit(seed, phases)
        gates = [(np.asarray(g.matrix, dtype=np.complex128), list(g.cargs) + list(g.targs)) for g in c.gates]
        exact = _extended(gates)
        plain = max(plain, float(np.abs(osv.run(gates, N_QUBITS) - exact).max()))
        passes = max(passes, float(np.abs(generated.run(c, N_QUBITS, 16, (11, 5, merge)) - exact).max()))
    assert passes <= 2 * plain + 2 * 2.0 ** -53
