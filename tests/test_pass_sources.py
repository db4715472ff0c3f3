"""Generated sources of deep circuits, on the CPU: twelve parameter sets of one
circuit give one source per launch, in both precisions, merged and not, also
with one angle for a whole layer (whose scalars all have one size); a circuit
whose scalars leave the range of complex64 keeps its own matrices: one source
for that, and results that match the FP64 oracle (1e-5, as every state-vector
run)."""
import numpy as np
import pytest

import generated
from oracle import sv as osv


def _layers(kind, n, depth, values):
    from quict_b200.core import CX, Circuit, H, Rx, Ry, Rz, Rzz, U3
    val = np.random.default_rng(values)
    c = Circuit(n)

    def angle():
        return float(val.uniform(0, 2 * np.pi))

    if kind == "qaoa":
        edges = [[int(q) for q in np.random.default_rng(e).choice(n, 2, replace=False)] for e in range(2 * n)]
        for q in range(n):
            H | c(q)
    for _ in range(depth):
        if kind == "qaoa":
            g, b = angle(), angle()
            for e in edges:
                Rzz(g) | c(e)
            for q in range(n):
                Rx(b) | c(q)
            continue
        for q in range(n):
            if kind == "rx-rzz":
                Rx(angle()) | c(q)
            elif kind == "u3-cx":
                U3(angle(), angle(), angle()) | c(q)
            else:
                Ry(angle()) | c(q)
                Rz(angle()) | c(q)
        for q in range(n if kind == "rx-rzz" else n - 1):
            if kind == "rx-rzz":
                Rzz(angle()) | c([q, (q + 1) % n])
            else:
                CX | c([q, q + 1])
    return c


@pytest.mark.parametrize("merge", [0, 2])
@pytest.mark.parametrize("esize", [16, 8])
@pytest.mark.parametrize("kind,n,depth", [("rx-rzz", 14, 8), ("rx-rzz", 16, 12), ("u3-cx", 14, 8), ("ry-rz-cx", 14, 8),
                                          ("qaoa", 14, 8)])
def test_one_source_per_launch(kind, n, depth, esize, merge):
    runs = [generated.sources(_layers(kind, n, depth, 100 + v), n, esize, (11, 5, merge)) for v in range(12)]
    # merging the phases of this graph gives entries exp(ig) exp(-ig), which are
    # 1 or next to it in complex128: two kinds of matrices, two sources
    kinds = 2 if (kind, esize, merge) == ("qaoa", 16, 2) else 1
    assert max(len(set(launch)) for launch in zip(*runs, strict=True)) <= kinds


@pytest.mark.parametrize("angle", [np.pi - 1e-3, np.pi - 1e-5])
def test_scalars_beyond_the_range(angle):
    from quict_b200.core import Circuit, H, Rx, Rzz
    n = 12
    c = Circuit(n)
    for q in range(n):
        H | c(q)
    for _ in range(4):
        for q in range(n):
            Rx(angle) | c(q)
        Rzz(0.7) | c([0, 1])
    norms = []
    got = generated.run(c, n, 8, (11, 5, 0), norms)
    want = osv.run([(np.asarray(g.matrix, dtype=np.complex128), list(g.cargs) + list(g.targs)) for g in c.gates], n)
    assert np.abs(got - want).max() <= 1e-5
    assert max(norms) <= 2.0 ** 60
