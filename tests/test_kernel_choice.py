"""Both sides of the sizes at which a call changes its kernel: Pauli sums with
shared and with all different X masks around 2^20 and 2^22 amplitudes, dense
gates on 6 to 10 qubits with as many groups as the SMs take at once and twice
that, collapse and reset on low and high bits around 2^23 amplitudes; against
the same rules in torch's FP64.  Tolerances: sums and matrix products as
state-vector runs (1e-12 / 1e-5), collapse and reset one rounding of each kept
component."""
import ctypes as C

import numpy as np
import pytest
import torch

TOL = {torch.complex128: 1e-12, torch.complex64: 1e-5}


def _state(n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    v = torch.view_as_complex(torch.randn((1 << n, 2), generator=g, device="cuda", dtype=torch.float64))
    return (v / torch.linalg.vector_norm(v)).to(dtype)


def _qs(dtype):
    from quict_b200 import _native as N
    return N.QS_C128 if dtype == torch.complex128 else N.QS_C64


def _parity(x):
    for s in (16, 8, 4, 2, 1):
        x = x ^ (x >> s)
    return x & 1


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("masks", ["shared", "different"])
@pytest.mark.parametrize("n", [11, 19, 20, 21, 22])
def test_pauli_sums(n, masks, dtype):
    from quict_b200 import _native as N
    rng = np.random.default_rng(n)
    nt = 12
    x = rng.choice(1 << n, nt, replace=False).astype(np.uint64)
    if masks == "shared":
        x[4:] = x[:4].repeat(2)
    z = rng.integers(0, 1 << n, nt, dtype=np.uint64)
    c = rng.normal(size=nt)
    psi = _state(n, dtype)
    out = torch.full_like(psi, float("nan"))
    cc = np.ascontiguousarray(np.stack([c, np.zeros(nt)], 1).ravel())
    N.call("qs_apply_pauli_sum", C.c_void_p(psi.data_ptr()), C.c_void_p(out.data_ptr()), n, _qs(dtype),
           x.ctypes.data_as(C.c_void_p), z.ctypes.data_as(C.c_void_p), cc.ctypes.data_as(C.c_void_p), nt, None)
    h = psi.to(torch.complex128)
    j = torch.arange(1 << n, device="cuda")
    want = torch.zeros_like(h)
    for t in range(nt):
        src = j ^ int(x[t])
        sign = 1.0 - 2.0 * _parity(src & int(z[t])).double()
        want += c[t] * (1j ** (int(x[t]) & int(z[t])).bit_count()) * sign * h[src]
    assert float((out.to(torch.complex128) - want).abs().max()) <= TOL[dtype]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("controls", [0, 1])
@pytest.mark.parametrize("k", [6, 7, 8, 9, 10])
def test_dense_gates(k, controls, dtype):
    from quict_b200.simulation.engine import Engine, require_cuda
    from quict_b200.simulation.lowering import Op
    from quict_b200.workloads import haar_unitary
    rng = np.random.default_rng(k)
    eng = Engine(require_cuda(0))
    mat = haar_unitary(rng, 1 << k)
    for groups in (0, 3, 6, 7, 8, 9, 10):
        n = k + groups + controls
        if n > 18:
            continue
        bits = [int(b) for b in rng.permutation(n)[:k + controls]]
        tbits, cbits = bits[:k], tuple(bits[k:])
        psi = _state(n, dtype)
        h = psi.to(torch.complex128)
        idx = torch.arange(1 << n, device="cuda")
        zero = torch.ones_like(idx, dtype=torch.bool)
        for b in tbits:
            zero &= ((idx >> b) & 1) == 0
        for b in cbits:
            zero &= ((idx >> b) & 1) == 1
        spread = torch.tensor([sum(((r >> (k - 1 - j)) & 1) << b for j, b in enumerate(tbits)) for r in range(1 << k)],
                              device="cuda")
        cols = idx[zero][None, :] + spread[:, None]
        want = h.clone()
        want[cols] = torch.from_numpy(mat).cuda() @ h[cols]
        eng.apply_single(psi, n, Op("mat", tuple(tbits), cbits, mat))
        assert float((psi.to(torch.complex128) - want).abs().max()) <= TOL[dtype], (groups, tbits, cbits)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("n", [3, 13, 22, 23, 24])
def test_collapse_and_reset(n, dtype):
    from quict_b200.simulation.engine import Engine, require_cuda
    eng = Engine(require_cuda(0))
    base = _state(n, dtype)
    h = base.to(torch.complex128)
    idx = torch.arange(1 << n, device="cuda")
    eps = 2.0 ** -52 if dtype == torch.complex128 else 2.0 ** -23
    for bit in sorted({0, 1, 2, n // 2, n - 1}):
        one = ((idx >> bit) & 1) == 1
        for outcome in (0, 1):
            got = base.clone()
            eng.collapse(got, n, bit, outcome, 1.25)
            want = torch.where(one == bool(outcome), h * 1.25, 0)
            assert bool(((got.to(torch.complex128) - want).abs() <= eps * want.abs()).all())
        for p in (0.37, 0.0):
            got = base.clone()
            eng.reset(got, n, bit, p)
            want = torch.zeros_like(h)
            a = float(np.sqrt(p))
            want[~one] = h[one] if p == 0.0 else torch.complex(h[~one].real / a, h[~one].imag / a)
            assert bool(((got.to(torch.complex128) - want).abs() <= eps * want.abs()).all())
