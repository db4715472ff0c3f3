"""Matrices of generated passes with factors taken out (csrc/passgen.cu).

CPU: the generated source of a circuit does not depend on its parameters'
values.  GPU: circuits whose factors are at their limits -- angles at and
next to 0, pi and 2 pi (a diagonal entry that vanishes or nearly does), long
runs of them (the bound on the factors), factors that cross X, SWAP, CX and
diagonals -- match the FP64 oracle.  Tolerances: 1e-12 (complex128), 1e-5
(complex64), as for every state-vector run."""
import ctypes as C

import numpy as np
import pytest

from oracle import sv as osv

ONE = ["h", "rx", "ry", "rz", "u3"]


def _gates(n, size, seed, values, angles=None):
    """[(name, params, qubits)]: structure from `seed`, angles from `values`."""
    rng, val = np.random.default_rng(seed), np.random.default_rng(values)
    out = []
    for _ in range(size):
        name = ["h", "x", "rx", "ry", "rz", "u3", "cx", "cz", "rzz", "swap"][rng.integers(10)]
        k = 2 if name in ("cx", "cz", "rzz", "swap") else 1
        qs = [int(q) for q in rng.choice(n, k, replace=False)]
        np_ = {"rx": 1, "ry": 1, "rz": 1, "rzz": 1, "u3": 3}.get(name, 0)
        if angles is None:
            p = [float(x) for x in val.uniform(0.1, 6.1, np_)]
        else:
            p = [float(angles[val.integers(len(angles))]) for _ in range(np_)]
        out.append((name, p, qs))
    return out


def _circuit(n, gates):
    from quict_b200.core import GATE_BY_NAME, Circuit
    c = Circuit(n)
    for name, p, qs in gates:
        g = GATE_BY_NAME[name]
        (g(*p) if p else g) | c(qs)
    return c


def _sources(n, circuit, esize, knobs):
    from quict_b200 import _native as N
    from quict_b200.simulation.fusion import MatrixTable, Pass, emit, iter_plan, relabel_swaps
    from quict_b200.simulation.lowering import lower_circuit
    ops = relabel_swaps(lower_circuit(circuit.gates, n), n)
    passes = [s for s in iter_plan(ops, n, *knobs[:2], merge_bits=knobs[2]) if isinstance(s, Pass) and s.ops]
    table = MatrixTable()
    cps, npass, cops, nops = emit(passes, table)
    host = table.array().astype(np.complex128 if esize == 16 else np.complex64)
    out = []
    for i in range(npass):
        ln, buf = C.c_int64(0), C.create_string_buffer(1 << 21)
        rc = N.load().qs_jit_pass_source(n, N.QS_C128 if esize == 16 else N.QS_C64, C.byref(cps[i]), cops, nops,
                                         C.c_void_p(host.ctypes.data), host.size, 0, buf, 1 << 21, C.byref(ln))
        assert rc == 0
        out.append(buf.value.decode())
    return out


@pytest.mark.parametrize("merge", [0, 2])
@pytest.mark.parametrize("esize", [16, 8])
def test_sources_do_not_depend_on_the_values(esize, merge):
    n = 14
    knobs = (11 if esize == 16 else 12, 5, merge)
    ref = _sources(n, _circuit(n, _gates(n, 150, 3, 0)), esize, knobs)
    for values in (1, 2, 3):
        assert _sources(n, _circuit(n, _gates(n, 150, 3, values)), esize, knobs) == ref


@pytest.mark.gpu
@pytest.mark.parametrize("angles", [[0.0, np.pi, 2 * np.pi], [np.pi - 1e-7, np.pi + 1e-3, 1e-7, np.pi / 2],
                                    [3.14, 3.1416, 0.3], None], ids=["exact", "near", "long", "general"])
@pytest.mark.parametrize("precision,knobs", [("double", (10, 5, 0)), ("double", (11, 5, 2)), ("single", (11, 5, 0)),
                                             ("single", (12, 5, 2))])
def test_compiled_passes_match_the_oracle(precision, knobs, angles):
    from quict_b200 import _native as N
    from quict_b200.simulation import StateVectorSimulator
    n = 13
    gates = _gates(n, 160, 5, 7, angles)
    c = _circuit(n, gates)
    sim = StateVectorSimulator("GPU", precision, tile_bits=knobs[0], low_bits=knobs[1], merge_bits=knobs[2])
    old = N.jit_set_mode(N.QS_JIT_SYNC)
    try:
        got = sim.run(c).get()
    finally:
        N.jit_set_mode(old)
    want = osv.run([(np.asarray(g.matrix, dtype=np.complex128), list(g.cargs) + list(g.targs)) for g in c.gates], n)
    assert np.abs(got - want).max() <= (1e-12 if precision == "double" else 1e-5)
