"""The range of generated passes whose matrices had factors taken out
(csrc/passgen.cu): two-qubit unitaries whose diagonal entries differ in size,
with their factors sent across X gates, many times in one launch.  On the CPU
the launches run as numpy statements (generated.py): the state stays within
the limits between the stages, and the result matches the FP64 oracle; on the
GPU the compiled passes match it.  Limits: 2^60 up and 2^-48 down in complex64
(24 bits each for scalars and for factors under way), 2^+-600 in complex128.
Tolerances: 1e-12 (complex128), 1e-5 (complex64), as every state-vector run."""
import numpy as np
import pytest

import generated
from oracle import sv as osv

LIMITS = {16: (2.0 ** -600, 2.0 ** 600), 8: (2.0 ** -48, 2.0 ** 60)}
TOL = {16: 1e-12, 8: 1e-5}


def _want(c, n):
    return osv.run([(np.asarray(g.matrix, dtype=np.complex128), list(g.cargs) + list(g.targs)) for g in c.gates], n)


def _phases(rng):
    return np.diag(np.exp(1j * rng.uniform(0, 6, 4)))


def _exchanged(n, blocks, c=1e-3):
    """A near-controlled unitary (a rotation with cosine c where bit 0 is set)
    whose factor on bit 0 crosses an X that CZs on the top bit keep apart."""
    from quict_b200.core import CX, CZ, Circuit, H, U3, Unitary, X
    rng = np.random.default_rng(2)
    circ = Circuit(n)
    q0, q1, top = n - 1, n - 2, 0
    H | circ(q0)
    H | circ(q1)
    m = np.eye(4, dtype=complex)
    m[1, 1] = m[3, 3] = c
    m[3, 1] = np.sqrt(1 - c * c)
    m[1, 3] = -m[3, 1]
    m = _phases(rng) @ m @ _phases(rng)
    for _ in range(blocks):
        Unitary(m) | circ([q1, q0])
        CZ | circ([q0, top])
        X | circ(q0)
        CZ | circ([q0, top])
        U3(0.7, 0.3, 0.2) | circ(q0)
        CX | circ([1, q0])
    return circ


def _partial_swaps(n, blocks, t=1.57):
    """Phases times a partial swap, then X on both qubits."""
    from quict_b200.core import Circuit, H, Unitary, X
    rng = np.random.default_rng(1)
    circ = Circuit(n)
    for q in range(n):
        H | circ(q)
    swap = np.eye(4, dtype=complex)
    swap[1, 1] = swap[2, 2] = np.cos(t)
    swap[1, 2] = swap[2, 1] = -1j * np.sin(t)
    for _ in range(blocks):
        Unitary(_phases(rng) @ swap) | circ([0, 1])
        X | circ(0)
        X | circ(1)
    return circ


def _haar_mix(n, blocks):
    """Two-qubit Haar and near-controlled unitaries among X, CX, SWAP and U3."""
    from quict_b200.core import CX, Circuit, H, Swap, U3, Unitary, X
    from quict_b200.workloads import haar_unitary
    rng = np.random.default_rng(blocks)
    circ = Circuit(n)
    for q in range(n):
        H | circ(q)
    for _ in range(5 * blocks):
        a, b = (int(q) for q in rng.choice(n, 2, replace=False))
        kind = rng.integers(6)
        if kind == 0:
            Unitary(haar_unitary(rng, 4)) | circ([a, b])
        elif kind == 1:
            t = rng.choice([1e-3, 1e-5, 0.3])
            m = np.eye(4, dtype=complex)
            m[1, 1] = m[3, 3] = t
            m[3, 1] = np.sqrt(1 - t * t)
            m[1, 3] = -m[3, 1]
            Unitary(_phases(rng) @ m @ _phases(rng)) | circ([a, b])
        elif kind == 2:
            X | circ(a)
        elif kind == 3:
            CX | circ([a, b])
        elif kind == 4:
            Swap | circ([a, b])
        else:
            U3(*(float(x) for x in rng.uniform(0.1, 6, 3))) | circ(a)
    return circ


CIRCUITS = [(_exchanged, 14, 2), (_partial_swaps, 12, 0), (_haar_mix, 12, 0), (_haar_mix, 13, 2)]
IDS = ["exchanged", "partial-swaps", "haar", "haar-merged"]


@pytest.mark.parametrize("blocks", [8, 16, 25, 40])
@pytest.mark.parametrize("esize", [16, 8])
@pytest.mark.parametrize("make,n,merge", CIRCUITS, ids=IDS)
def test_range_between_load_and_store(make, n, merge, esize, blocks):
    c = make(n, blocks)
    norms = []
    got = generated.run(c, n, esize, (11 if esize == 16 or n > 13 else 12, 5, merge), norms)
    assert min(norms) >= LIMITS[esize][0] and max(norms) <= LIMITS[esize][1]
    assert np.abs(got - _want(c, n)).max() <= TOL[esize]


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [16, 40])
@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("make,n,merge", CIRCUITS, ids=IDS)
def test_compiled_passes(make, n, merge, precision, blocks):
    from quict_b200 import _native as N
    from quict_b200.simulation import StateVectorSimulator
    c = make(n, blocks)
    old = N.jit_set_mode(N.QS_JIT_SYNC)
    try:
        before = N.jit_stats()["compiled_launches"]
        got = StateVectorSimulator("GPU", precision, merge_bits=merge).run(c).get()
        assert N.jit_stats()["compiled_launches"] > before
    finally:
        N.jit_set_mode(old)
    assert np.abs(got - _want(c, n)).max() <= TOL[16 if precision == "double" else 8]
