"""lam = H psi in chunks of eight amplitudes per thread: sizes below, at and
above a chunk, masks on the chunk's three bits and around them, repeated X
masks, real and complex coefficients and Y factors, both dtypes, against the
FP64 sum (rounding of the result's own precision)."""
import ctypes as C

import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
@pytest.mark.parametrize("coeffs", ["real", "complex"])
@pytest.mark.parametrize("n", [1, 4, 9, 10, 11, 12, 15, 18])
def test_pauli_sum(n, coeffs, dtype):
    from quict_b200 import _native as N
    rng = np.random.default_rng(n)
    nt = 40
    top = 1 << n
    x = rng.integers(0, top, nt, dtype=np.uint64)
    x[:12] = 0
    x[12:20] = np.uint64(0x700 % top)
    x[20:24] = np.uint64(0x100 % top)
    z = rng.integers(0, top, nt, dtype=np.uint64)
    z[:4] = np.uint64(0x500 % top)
    c = rng.normal(size=nt) + (1j * rng.normal(size=nt) if coeffs == "complex" else 0)
    if coeffs == "real":  # no Y factors: real sums throughout
        z[12:] &= ~x[12:]
    v = rng.normal(size=top) + 1j * rng.normal(size=top)
    v /= np.linalg.norm(v)
    psi = torch.from_numpy(v).to("cuda", dtype)
    out = torch.full_like(psi, float("nan"))
    cc = np.ascontiguousarray(np.stack([c.real, c.imag], 1).ravel() if coeffs == "complex" else
                              np.stack([c, np.zeros(nt)], 1).ravel())
    N.call("qs_apply_pauli_sum", C.c_void_p(psi.data_ptr()), C.c_void_p(out.data_ptr()), n,
           N.QS_C128 if dtype == torch.complex128 else N.QS_C64, x.ctypes.data_as(C.c_void_p),
           z.ctypes.data_as(C.c_void_p), cc.ctypes.data_as(C.c_void_p), nt, None)
    torch.cuda.synchronize()
    h = psi.cpu().numpy().astype(np.complex128)
    j = np.arange(top, dtype=np.uint64)
    want = np.zeros(top, dtype=np.complex128)
    for t in range(nt):
        src = j ^ x[t]
        par = np.bitwise_count(src & z[t]) & 1
        want += c[t] * (1j ** int(np.bitwise_count(x[t] & z[t]))) * np.where(par, -1.0, 1.0) * h[src]
    scale = np.abs(c).sum() * np.abs(h).max()
    eps = 1e-14 if dtype == torch.complex128 else 2.0 ** -23
    assert np.abs(out.cpu().numpy() - want).max() <= eps * scale
