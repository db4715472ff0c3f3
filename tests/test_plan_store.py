"""Plans and parameter blocks kept between launches, on generated kernels
(synchronous compilation, counted): more parameter sets of one circuit than a
plan keeps, with the last ones coming back at once (found again) and the first
ones after all others (made again), match the FP64 oracle (1e-12 / 1e-5, as
every state-vector run); and the store stays below 64 MB however many parameter
sets its plans see."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import sv as osv
from test_plan_reuse import N_QUBITS, _circuit, _want

STORE = 64 << 20


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["double", "single"])
def test_generated_kernels_take_the_right_parameters(precision):
    from quict_b200 import _native as N
    from quict_b200.simulation import StateVectorSimulator
    tol = 1e-12 if precision == "double" else 1e-5
    circuits = [_circuit(v) for v in range(11)]
    want = [_want(c) for c in circuits]
    old = N.jit_set_mode(N.QS_JIT_SYNC)
    try:
        sims = [StateVectorSimulator("GPU", precision) for _ in circuits]
        sims[0].run(circuits[0])
        before = N.jit_stats()
        order = [0, 1, 2, 3, 2, 1, 0, 3] + list(range(11)) + [10, 9, 8, 7, 10] + [0, 1, 10]
        for i in order:
            assert np.abs(sims[i].run(circuits[i]).get() - want[i]).max() <= tol, i
        after = N.jit_stats()
        assert after["compiled_launches"] - before["compiled_launches"] >= 2 * len(order)
        assert after["generic_launches_while_pending"] == before["generic_launches_while_pending"]
    finally:
        N.jit_set_mode(old)


@pytest.mark.gpu
def test_the_store_is_bounded():
    from quict_b200 import _native as N
    from quict_b200.core import Circuit, Unitary
    from quict_b200.simulation.fusion import MatrixTable, Pass, emit, iter_plan
    from quict_b200.simulation.lowering import lower_circuit
    from quict_b200.workloads import haar_unitary
    n, plans, sets = 11, 1200, 8
    rng = np.random.default_rng(4)
    c = Circuit(n)
    for i in range(24):
        Unitary(haar_unitary(rng, 4)) | c([i % n, (i + 1) % n])
    steps = list(iter_plan(lower_circuit(c.gates, n), n, 11, 5, merge_bits=0))
    assert len(steps) == 1 and isinstance(steps[0], Pass)
    table = MatrixTable()
    cps, npass, cops, nops = emit(steps, table)
    base = table.array()
    # one pass at `plans` places of a table: as many plans with one kernel
    host = np.zeros(base.size + plans, dtype=np.complex128)
    vec = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    vec[0] = 1
    first = [cops[i].mat for i in range(nops)]
    mats = torch.zeros(host.size, dtype=torch.complex128, device="cuda")
    lib, most = N.load(), 0
    old = N.jit_set_mode(N.QS_JIT_ASYNC)
    try:
        for s in range(sets):
            for at in range(plans):
                host[at:at + base.size] = base * np.exp(1j * s)
                for i in range(nops):
                    cops[i].mat = first[i] + at
                N.call("qs_apply_fused_ex", C.c_void_p(vec.data_ptr()), n, N.QS_C128, cps, npass, cops, nops,
                       C.c_void_p(mats.data_ptr()), C.c_void_p(host.ctypes.data), host.size,
                       N.stream_ptr(torch.cuda.current_stream()))
                most = max(most, lib.qs_plan_store_bytes())
        torch.cuda.synchronize()
        N.jit_wait(900)
    finally:
        N.jit_set_mode(old)
    assert STORE // 2 < most <= STORE
